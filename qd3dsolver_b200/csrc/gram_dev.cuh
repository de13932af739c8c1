// Gram products A^H B of tall-skinny blocks with FP64 accumulation: one pass over the rows of every
// block that enters, on the FP64 tensor cores (mma.sync.m8n8k4.f64; the tcgen05 family has no f64
// kind).
//
// The complex product is one real GEMM over the interleaved (re, im) view: with A' (n x 2P) and
// B' (n x 2Q) the real views, C' = A'^T B' and
//   Re G_ij = C'_{2i,2j} + C'_{2i+1,2j+1},   Im G_ij = C'_{2i,2j+1} - C'_{2i+1,2j}.
//
// What bounds it: the FP64 rate (64 FMA a clock and SM) from about 24 columns on, HBM below.
// Design:
//   * A task lists its blocks once; A and B are ranges of the concatenated columns, so a block that
//     enters on both sides is read once. All products of a Rayleigh-Ritz step are one task.
//   * Rows stream through shared memory in chunks: one producer warp fills a ring of them, the other
//     warps consume it, with a full and an empty mbarrier per chunk and no CTA-wide barrier. A
//     block's rows of a chunk are four runs of memory, one bulk copy each (blocks whose rows are not
//     contiguous whole 16-byte words: element-wise cp.async by the producer). With every thread copying
//     behind a barrier the MMAs waited for the copy loop (91 us for 663,552 x 12 x 12, its bytes take
//     20); a bulk copy per row costs about 70 clocks of the copy engine each (161 us).
//   * The k index of an MMA runs over the four runs, which are skewed by eight banks: fragment loads
//     are free of bank conflicts at every block width.
//   * C' is cut into rectangles of 3 x 3 tiles of 8 x 8, a warp each, the accumulators in registers
//     over the CTA's whole row range. Rectangles nothing reads (below the diagonal of a Hermitian
//     product, the blocks a pencil takes from their adjoints) are left out; on the diagonal of one
//     the three tiles below it are. Warps beyond the rectangle count split the rows.
//   * Each CTA writes its rectangles' sums; gram_reduce adds the CTAs' in order, on many CTAs.
// The split of the rows depends only on n, so a result does not depend on what else runs.
#pragma once
#include "blockops.cuh"
#include "mbar_dev.cuh"

namespace qdkp {

static __device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}

constexpr int kGramRect = 12;            // complex columns of a rectangle's side (3 tiles)
constexpr int kGramRectElems = 24 * 24;  // real entries of a rectangle
constexpr int kGramMaxBlk = 6;
constexpr int kGramMaxWarps = 16;
constexpr int kGramMaxParts = 148;       // row parts: one CTA per SM
constexpr int kGramMaxRects = 128;       // rectangles of the widest task (72 x 144 columns: 6 x 12)

// Which entries of A^H B a task needs.
enum GramKind {
  GK_FULL = 0,
  GK_HERM,      // A and B are the same columns: the upper triangle
  // the non-explicit pencil of lobpcg.py:856-861, A = [X | R | P], B = [P | AR | AP]: everything
  // in X's rows, R^H P, the upper triangle of R^H AR, R^H AP, the upper triangle of P^H AP
  GK_PENCIL,
  // explicit Gram matrices, A = [X | R | P], B = [X | R | P | AX | AR | AP]: the upper triangle of
  // W^H W; of W^H AW the diagonal blocks and those above
  GK_EXPLICIT
};

template <typename T>
struct GramTask {
  const cplx<T>* p[kGramMaxBlk];
  long long ld[kGramMaxBlk];
  int cols[kGramMaxBlk];
  int nblk, tc;             // blocks and their columns in all
  int a0, P, b0, Q;         // A and B as ranges of the concatenated columns
  int kind;
  int m, ma, mp;            // widths of X, R, P (pencil kinds)
  long long n;
  int* fault;               // device_fault_flag
};

// Where entry (i, j) of a task's product goes. GK_FULL and GK_HERM: out, row-major, both triangles;
// GK_PENCIL: the product with P to S ((m + ma) x mp), the others to T (tot x (ma + mp));
// GK_EXPLICIT: W^H W to S, W^H AW to T, both tot x tot.
template <typename T>
static __device__ __forceinline__ void gram_put(const GramTask<T>& t, int i, int j, double2 v,
                                                double2* __restrict__ out, double2* __restrict__ S) {
  if (t.kind == GK_PENCIL) {
    if (j >= t.mp) out[i * (t.ma + t.mp) + (j - t.mp)] = v;
    else if (i < t.m + t.ma) S[i * t.mp + j] = v;
  } else if (t.kind == GK_EXPLICIT) {
    if (j < t.P) S[i * t.P + j] = v;
    else out[i * t.P + (j - t.P)] = v;
  } else {
    out[i * t.Q + j] = v;
    if (t.kind == GK_HERM && i != j) out[j * t.Q + i] = make_double2(v.x, -v.y);
  }
}

// does the rectangle at (ri, ci) hold a needed entry? 2: a diagonal one, its upper triangle only
__host__ __device__ inline int gram_need(int kind, int P, int Q, int m, int ma, int mp, int ri, int ci) {
  const int r0 = ri * kGramRect, r1 = min(P, r0 + kGramRect) - 1;
  const int c0 = ci * kGramRect, c1 = min(Q, c0 + kGramRect) - 1;
  if (kind == GK_FULL) return 1;
  if (kind == GK_HERM) return ci < ri ? 0 : (ci == ri ? 2 : 1);
  // column blocks [lo, hi) of the rows and of the columns, as (start, end) pairs
  const int rb[4] = {0, m, m + ma, m + ma + mp};
  if (kind == GK_EXPLICIT) {
    const int tot = m + ma + mp;
    if (c0 < tot && r0 <= min(c1, tot - 1)) return c0 == r0 && c1 < tot ? 2 : 1;   // W^H W, upper
    if (c1 < tot) return 0;
    for (int b = 0; b < 3; ++b)                            // W^H AW: block row b, columns from it on
      if (r0 < rb[b + 1] && r1 >= rb[b] && c1 - tot >= rb[b]) return 1;
    return 0;
  }
  const int cb[4] = {0, mp, mp + ma, 2 * mp + ma};
  // upper triangle of R^H AR and P^H AP alone in the rectangle, on their diagonal
  for (int k = 1; k < 3; ++k)
    if (r0 >= rb[k] && r1 < rb[k + 1] && c0 >= cb[k] && c1 < cb[k + 1] && r0 - rb[k] == c0 - cb[k]) return 2;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      if (r0 >= rb[i + 1] || r1 < rb[i] || c0 >= cb[j + 1] || c1 < cb[j]) continue;
      if (i == 2 && j < 2) continue;
      if (i == j && i > 0) {                               // needs a row at or above the last column
        if (max(r0, rb[i]) - rb[i] <= min(c1, cb[j + 1] - 1) - cb[j]) return 1;
      } else {
        return 1;
      }
    }
  return 0;
}

// Rows of a chunk: about 62 KB, for few columns 25 KB, a multiple of 32. A block's share of a stage:
// four runs of crow / 4 rows, each followed by kGramSkew bytes.
// Few columns (the products of one or two blocks of 12): their few warps leave room for a second CTA
// on the SM, so their ring takes less than half of its shared memory. A CTA's start and its sums then
// hide behind the other's rows (complex128 with the copy of the result: 254,800 rows of 12 x 12 columns 67 to
// 60 us, of 12 with themselves 58 to 53, 663,552 rows 72 to 63; 14 complex128 slots, 8 ticks: 48.9 to 47.8 ms).
constexpr int kGramSkew = 32;
constexpr int kGramNarrow = 24;
template <typename T> __host__ __device__ inline int gram_crow(int tc) {
  const int r = (tc <= kGramNarrow ? 25 : 62) * 1024 / (tc * (int)sizeof(cplx<T>)) / 32 * 32;
  return r < 32 ? 32 : (r > 128 ? 128 : r);
}
template <typename T> __host__ __device__ inline size_t gram_stage(int tc) {
  return (size_t)gram_crow<T>(tc) * tc * sizeof(cplx<T>) + 4 * kGramSkew * kGramMaxBlk;
}
constexpr int kGramMaxSmem = 224 * 1024;
constexpr int kGramStages = 6;
constexpr size_t kGramTable = 128;               // the barriers
// shared memory of a launch for at most tc concatenated columns and `warps` consumer warps
template <typename T> __host__ __device__ inline size_t gram_smem(int tc, int warps) {
  const size_t st = gram_stage<T>(tc), ring = (tc <= kGramNarrow ? 101 : 190) * 1024;
  const size_t bytes = kGramStages * st < ring ? kGramStages * st : (2 * st > ring ? 2 * st : ring);
  const size_t red = (size_t)warps * kGramRectElems * sizeof(double);
  return kGramTable + (bytes > red ? bytes : red);
}

struct GramShape { int rects, panels, warps, slices; };   // warps: consumers; one more produces
// Rectangles needed, panels of at most kGramMaxWarps of them, warps of a CTA and the row slices they
// make: whole multiples of a panel's rectangles, so that no warp idles.
__host__ __device__ inline GramShape gram_shape(int kind, int P, int Q, int m, int ma, int mp) {
  GramShape s;
  s.rects = 0;
  for (int ri = 0; ri * kGramRect < P; ++ri)
    for (int ci = 0; ci * kGramRect < Q; ++ci) s.rects += gram_need(kind, P, Q, m, ma, mp, ri, ci) ? 1 : 0;
  s.panels = (s.rects + kGramMaxWarps - 1) / kGramMaxWarps;
  const int per = (s.rects + s.panels - 1) / s.panels;
  s.slices = per >= 8 ? kGramMaxWarps / per : (per >= 5 ? 2 : (per >= 3 ? 4 : 8 / per));
  s.warps = per * s.slices;
  return s;
}

// Row parts of a product: a thousand rows each, which amortise a CTA's start and partial sums, but up to 74
// parts of as few as 128 rows, so that a short product still fills half of the SMs, or all of them once with the
// two panels of a wide one. 74 | n / 1024 parts, complex128, 3 m x 2 m columns, with the copy of the result (us):
// m = 13, 5,000 rows 49 | 112, 20,000 60 | 100, 40,000 73 | 100; m = 24, 20,000 65 | 107, 40,000 78 | 106; m = 6,
// 2,000 39 | 60. With up to 148 short parts 80,000 rows of m = 13 take 76 us instead of 110, but the slots of a
// small sweep, whose products run side by side, 2 to 3% longer.
constexpr int kGramShortParts = kGramMaxParts / 2, kGramShortRows = 128;
__host__ __device__ inline int gram_parts(long long n) {
  long long parts = n / 1024;
  const long long least = n / kGramShortRows < kGramShortParts ? n / kGramShortRows : kGramShortParts;
  if (parts < least) parts = least;
  if (parts > kGramMaxParts) parts = kGramMaxParts;
  return parts < 1 ? 1 : (int)parts;
}
// rows of a part: even, so that 16-byte pairs of complex64 rows stay aligned
__host__ __device__ inline long long gram_part_rows(long long n, int parts) {
  return ((n + parts - 1) / parts + 3) / 4 * 4;
}

// partial doubles of one task (all parts)
__host__ __device__ inline size_t gram_partial_doubles(int rects, int parts) {
  return (size_t)rects * parts * kGramRectElems;
}

// Every thread's rectangle (threadIdx.x = ri * gc + ci): what gram_need says and its index among the
// needed ones; returns their number. At least kGramMaxRects threads; uniform barriers.
template <typename T>
static __device__ int gram_enumerate(const GramTask<T>& t, int& need, int& index) {
  __shared__ unsigned s_bal[kGramMaxRects / 32];
  const int gr = (t.P + kGramRect - 1) / kGramRect, gc = (t.Q + kGramRect - 1) / kGramRect;
  const int i = threadIdx.x;
  need = i < gr * gc ? gram_need(t.kind, t.P, t.Q, t.m, t.ma, t.mp, i / gc, i % gc) : 0;
  const unsigned bal = __ballot_sync(0xffffffffu, need != 0);
  if ((i & 31) == 0 && i < kGramMaxRects) s_bal[i >> 5] = bal;
  __syncthreads();
  int total = 0;
  index = 0;
  for (int w = 0; w < kGramMaxRects / 32; ++w) {
    if (w == (i >> 5)) index = total + __popc(bal & ((1u << (i & 31)) - 1u));
    total += __popc(s_bal[w]);
  }
  return total;
}

// A warp's rectangle over its k steps of a chunk, the next step's fragments loaded ahead. Step i
// takes row i of each of the four runs. DIAG leaves out the three tiles below the diagonal; it is a
// loop of its own, since a branch around single MMAs is compiled to predicated ones, which hold
// the pipe all the same (27 instead of 16 clocks an MMA measured). pa / pb: the lane's fragment
// elements at step 0 and da / db from step to step; rows: steps this lane's run still has data
// for (beyond it counts as zeros).
template <bool DIAG, typename T>
static __device__ __forceinline__ void gram_chunk(const T* q, const int (&oa)[3], const int (&ob)[3],
                                                  const int (&da)[3], const int (&db)[3], int i, int di,
                                                  int rows, int steps, double (&acc)[3][3][2]) {
  double a[3], b[3];
  const T *pa[3], *pb[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    pa[k] = q + oa[k]; pb[k] = q + ob[k];
    a[k] = i < rows ? (double)*pa[k] : 0.0;
    b[k] = i < rows ? (double)*pb[k] : 0.0;
  }
  for (; i < steps; i += di) {
    double an[3], bn[3];
    const bool in = i + di < rows;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      pa[k] += da[k]; pb[k] += db[k];
      an[k] = in ? (double)*pa[k] : 0.0;
      bn[k] = in ? (double)*pb[k] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = DIAG ? k : 0; j < 3; ++j) dmma(acc[k][j][0], acc[k][j][1], a[k], b[j]);
#pragma unroll
    for (int k = 0; k < 3; ++k) { a[k] = an[k]; b[k] = bn[k]; }
  }
}

// Element offset (in T) of real column `col` of the concatenated columns in a stage, at row 0 of run
// t4; step: elements from row to row.
template <typename T>
static __device__ __forceinline__ void gram_offset(const GramTask<T>& t, int crow, int col, int t4,
                                                   int& off, int& step) {
  int c = col >> 1, b = 0, base = 0;
  while (b < t.nblk - 1 && c >= t.cols[b]) {
    base += crow * 2 * t.cols[b] + 4 * kGramSkew / (int)sizeof(T);
    c -= t.cols[b];
    ++b;
  }
  if (c >= t.cols[b]) c = 0;                        // past the last column: any value, not read out
  step = 2 * t.cols[b];
  off = base + t4 * (crow / 4 * step + kGramSkew / (int)sizeof(T)) + 2 * c + (col & 1);
}

// The CTA's part of a task: sums over the rows of part `part` of the rectangles of panel `panel`,
// into partial[(part * rects + rect) * kGramRectElems + ...]. The last warp produces; at least
// kGramMaxRects threads. A wait that gives up (a copy that never lands) leaves NaN sums and raises the device's
// fault flag.
template <typename T>
static __device__ void gram_core(const GramTask<T>& t, int part, int parts, int panel,
                                 double* __restrict__ partial, unsigned char* smem) {
  typedef cplx<T> C;
  __shared__ short s_rect[kGramMaxWarps];      // ri * 64 + ci, + 8192 for a diagonal one
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = (blockDim.x >> 5) - 1;
  const int g = lane >> 2, t4 = lane & 3;
  int need, index;
  const int total = gram_enumerate(t, need, index);
  const int panels = (total + nwarps - 1) / nwarps;
  const int per = panels ? (total + panels - 1) / panels : 0;
  const int first = panel * per, count = min(per, total - first);
  if (count <= 0) return;                          // a panel this task does not fill (uniform)
  if (need && index >= first && index < first + count) {
    const int gc = (t.Q + kGramRect - 1) / kGramRect;
    s_rect[index - first] = (short)(threadIdx.x / gc * 64 + threadIdx.x % gc + (need == 2 ? 8192 : 0));
  }
  const int slices = nwarps / count;
  // contiguous rows whose runs are whole 16-byte words in every block: bulk copies. Runs start at rows
  // that are multiples of four and, where n is even, have an even number of them, which makes odd
  // complex64 widths whole too
  bool bulk = true;
  for (int b = 0; b < t.nblk; ++b)
    bulk = bulk && (t.cols[b] == 0 || t.ld[b] == t.cols[b]) &&
           (sizeof(T) == 8 || (t.cols[b] & 1) == 0 || (t.n & 1) == 0) &&
           (reinterpret_cast<uintptr_t>(t.p[b]) & 15) == 0;
  const int crow = gram_crow<T>(t.tc), c4 = crow / 4;
  const unsigned stage = (unsigned)gram_stage<T>(t.tc);
  unsigned avail;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(avail));
  const int NS = min(kGramStages, (int)((avail - kGramTable) / stage));      // >= 2 by the launch's size
  unsigned char* st0 = smem + kGramTable;
  const unsigned full = smem_addr(smem), empty = full + 8 * kGramStages, st0a = full + (unsigned)kGramTable;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(full + 8 * i, bulk ? 1 : 32);
      mbar_init(empty + 8 * i, slices * count);
    }
    mbar_init_fence();
  }
  __syncthreads();
  const long long rpp = gram_part_rows(t.n, parts);
  const long long r0 = (long long)part * rpp, r1 = min(t.n, r0 + rpp);
  const int nchunks = r1 > r0 ? (int)((r1 - r0 + crow - 1) / crow) : 0;
  double acc[3][3][2];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  bool ok = true;
  if (warp == nwarps) {
    // ---- producer: a lane a row ------------------------------------------------------------
    int s = 0;
    unsigned ph = 1;                                 // parity of the empty phase waited for
    int c = 0;
    for (; c < nchunks; ++c) {
      if (!__all_sync(0xffffffffu, c < NS || mbar_wait(empty + 8 * s, ph))) break;
      const long long rn = r0 + (long long)c * crow;
      const int left = (int)min((long long)crow, r1 - rn);
      const unsigned bar = full + 8 * s;
      if (bulk) {
        if (lane == 0) mbar_expect_tx(bar, (unsigned)(left * t.tc * (int)sizeof(C)));
        __syncwarp();
      }
      unsigned d = st0a + s * stage;
      for (int b = 0; b < t.nblk; ++b) {
        const int cols = t.cols[b];
        const unsigned run = (unsigned)(c4 * cols * (int)sizeof(C)) + kGramSkew;
        if (bulk) {
          // run `lane` of the block: rows [lane c4, (lane + 1) c4) of the chunk that exist
          const int rows = min(c4, left - lane * c4);
          if (lane < 4 && rows > 0 && cols > 0)
            bulk_load(d + lane * run, t.p[b] + (rn + lane * c4) * cols, (unsigned)(rows * cols * (int)sizeof(C)), bar);
        } else {
          const int units = left * cols;
          for (int u = lane; u < units; u += 32) {
            const int r = u / cols, c2 = u - r * cols, q = r / c4;
            const C* src = t.p[b] + (rn + r) * t.ld[b] + c2;
            const unsigned e = d + q * run + (unsigned)(((r - q * c4) * cols + c2) * (int)sizeof(C));
            if constexpr (sizeof(T) == 8)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(e), "l"(src) : "memory");
            else
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" :: "r"(e), "l"(src) : "memory");
          }
        }
        d += 4 * run;
      }
      if (!bulk)      // arrives once this lane's copies have landed
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(bar) : "memory");
      if (++s == NS) { s = 0; if (c >= NS) ph ^= 1u; else ph = 0; }
    }
    // keep the CTA's shared memory until the copies issued have landed (or given up)
    for (int q = max(0, c - NS); q < c; ++q) mbar_wait(full + 8 * (q % NS), (unsigned)(q / NS) & 1u);
  } else if (warp < slices * count) {
    // ---- consumers -------------------------------------------------------------------------
    const int rect = warp % count, slice = warp / count;
    const int rc = s_rect[rect];
    const bool diag = rc & 8192;
    const int ri = (rc & 8191) >> 6, ci = rc & 63;
    int oa[3], ob[3], da[3], db[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      gram_offset(t, crow, 2 * (t.a0 + ri * kGramRect) + 8 * k + g, t4, oa[k], da[k]);
      gram_offset(t, crow, 2 * (t.b0 + ci * kGramRect) + 8 * k + g, t4, ob[k], db[k]);
      oa[k] += slice * da[k]; ob[k] += slice * db[k];
      da[k] *= slices; db[k] *= slices;
    }
    int s = 0;
    unsigned ph = 0;
    for (int c = 0; c < nchunks; ++c) {
      ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, ph));
      if (!ok) break;
      const int left = (int)min((long long)crow, r1 - (r0 + (long long)c * crow));
      const int steps = min(c4, left);               // run 0 has the most rows
      const int rows = min(c4, left - t4 * c4);      // of this lane's run
      const T* q = reinterpret_cast<const T*>(st0 + s * stage);
      if (slice < steps) {
        if (diag) gram_chunk<true>(q, oa, ob, da, db, slice, slices, rows, steps, acc);
        else gram_chunk<false>(q, oa, ob, da, db, slice, slices, rows, steps, acc);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + 8 * s);
      if (++s == NS) { s = 0; ph ^= 1u; }
    }
  }
  ok = __syncthreads_and(ok) != 0;
  if (!ok && threadIdx.x == 0) raise_device_fault(t.fault);
  // the row slices of a rectangle, summed in order
  double* red = reinterpret_cast<double*>(st0);
  if (warp < slices * count) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double* d = red + (size_t)warp * kGramRectElems + (8 * i + g) * 24 + 8 * j + 2 * t4;
        d[0] = acc[i][j][0]; d[1] = acc[i][j][1];
      }
  }
  __syncthreads();
  double* out = partial + ((long long)part * total + first) * kGramRectElems;
  for (int e = threadIdx.x; e < count * kGramRectElems; e += blockDim.x) {
    double v = ok ? 0.0 : __longlong_as_double(0x7ff8000000000000LL);
    for (int sl = 0; sl < slices; ++sl) v += red[(size_t)sl * count * kGramRectElems + e];
    out[e] = v;
  }
}

// the entry whose real view's upper left word stands at c (rows `row` apart), summed over parts [b0, b1) in
// order: eight parts' loads in flight, the last ones too (a remainder loop would wait for each)
static __device__ __forceinline__ double2 gram_add_parts(const double* __restrict__ c, long long pstride,
                                                         int b0, int b1, int row = 24) {
  double2 s = make_double2(0.0, 0.0);
  for (int b = b0; b < b1; b += 8) {
    double2 u[8], v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const double* cq = c + min(b + q, b1 - 1) * pstride;
      u[q] = __ldcg(reinterpret_cast<const double2*>(cq));
      v[q] = __ldcg(reinterpret_cast<const double2*>(cq + row));
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (b + q < b1) {
        s.x += u[q].x + v[q].y;
        s.y += u[q].y - v[q].x;
      }
  }
  return s;
}

// The parts of a GK_HERM task of one block added by one CTA into the upper triangle of G (ld t.P): the
// threads are dealt to (entry, share of the parts), so that 12 columns' 78 entries keep 468 threads'
// loads in flight at once.
template <typename T>
static __device__ void gram_reduce_herm(const GramTask<T>& t, int parts, const double* __restrict__ partial,
                                        double2* __restrict__ G) {
  __shared__ short s_map[kGramMaxRects];
  __shared__ double2 s_sum[512];
  int need, index;
  const int total = gram_enumerate(t, need, index);
  if (threadIdx.x < kGramMaxRects) s_map[threadIdx.x] = need ? (short)index : (short)-1;
  __syncthreads();
  const int m = t.P, gc = (m + kGramRect - 1) / kGramRect, nout = m * (m + 1) / 2;
  const int shares = min(parts, 512 / nout), ps = (parts + shares - 1) / shares;
  const int sh = threadIdx.x / nout, o = threadIdx.x - sh * nout;
  int i = 0, j = o;
  while (j >= m - i) { j -= m - i; ++i; }
  j += i;
  if (sh < shares) {
    const int k = s_map[(i / kGramRect) * gc + j / kGramRect];
    s_sum[threadIdx.x] = gram_add_parts(partial + (long long)k * kGramRectElems + 48 * (i % kGramRect) + 2 * (j % kGramRect),
                                        (long long)total * kGramRectElems, sh * ps, min(parts, (sh + 1) * ps));
  }
  __syncthreads();
  if (sh == 0) {
    double2 v = s_sum[o];
    for (int w = 1; w < shares; ++w) { v.x += s_sum[w * nout + o].x; v.y += s_sum[w * nout + o].y; }
    G[i * m + j] = v;
  }
  __syncthreads();
}
static_assert(kMaxBlock * (kMaxBlock + 1) / 2 <= 512, "an entry per thread");

// Adds the parts of a task. Output entry (i, j) of the P x Q product goes through put(i, j, value)
// where its rectangle was formed (GK_HERM: the upper triangle). A CTA of 8 warps takes 32 outputs a
// round: each warp adds an eighth of the parts in order, then the eighths are added in order.
constexpr int kGramRedThreads = 256;
template <typename T, class Put>
static __device__ void gram_reduce_core(const GramTask<T>& t, int parts, const double* __restrict__ partial,
                                        int cta, int ctas, Put put) {
  __shared__ short s_map[kGramMaxRects];       // rectangle (ri, ci) -> index, -1: not formed
  __shared__ double2 s_sum[8][32];
  int need, index;
  const int total = gram_enumerate(t, need, index);
  if (threadIdx.x < kGramMaxRects) s_map[threadIdx.x] = need ? (short)index : (short)-1;
  __syncthreads();
  const int gc = (t.Q + kGramRect - 1) / kGramRect;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ps = (parts + 7) / 8, b0 = warp * ps, b1 = min(parts, b0 + ps);
  const long long pstride = (long long)total * kGramRectElems;
  for (int o0 = cta * 32; o0 < t.P * t.Q; o0 += ctas * 32) {
    const int o = o0 + lane;
    const int i = o / t.Q, j = o - i * t.Q;
    int k = -1;
    if (o < t.P * t.Q && !(t.kind == GK_HERM && j < i)) k = s_map[(i / kGramRect) * gc + j / kGramRect];
    double re = 0.0, im = 0.0;
    if (k >= 0) {
      const double* c = partial + (long long)k * kGramRectElems + (2 * (i % kGramRect)) * 24 + 2 * (j % kGramRect);
      const double2 v = gram_add_parts(c, pstride, b0, b1);
      re = v.x;
      im = v.y;
    }
    s_sum[warp][lane] = make_double2(re, im);
    __syncthreads();
    if (warp == 0 && k >= 0) {
      double2 v = s_sum[0][lane];
      for (int w = 1; w < 8; ++w) { v.x += s_sum[w][lane].x; v.y += s_sum[w][lane].y; }
      put(i, j, v);
    }
    __syncthreads();
  }
}

}  // namespace qdkp
