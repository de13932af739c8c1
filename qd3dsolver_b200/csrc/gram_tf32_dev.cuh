// Gram products of complex64 blocks on split-precision TF32 MMA: what qdkp_block_gram forms where one CTA
// holds the product (up to 16 rectangles of 12 x 12 columns). Faster than the FP64 MMA on widened
// blocks (51 x 34 columns of 307k rows with its update: 422 us against 755 us), at FP32 accuracy; a
// solve's own products are formed in FP64 (gram_dev.cuh).
#pragma once
#include "dense_dev.cuh"

namespace qdkp {

constexpr int kStageBudget = 64 * 1024;    // shared memory for the row stages of one CTA

// Stages in flight: as many (2..4) as fit the budget, so that a CTA keeps several chunk loads
// outstanding while it works on one (the kernels are latency- or bandwidth-bound otherwise).
__host__ __device__ __forceinline__ int stage_count(size_t stage_bytes) {
  const int ns = (int)(kStageBudget / stage_bytes);
  return ns < 2 ? 2 : (ns > 4 ? 4 : ns);
}

// Dynamic shared memory this launch was given (the %dynamic_smem_size special register). The
// staged kernels fit their stage count and chunk size into it, so a product narrower than the
// one the launch was sized for can never over-run its allocation.
__device__ __forceinline__ unsigned dyn_smem_bytes() {
  unsigned r;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(r));
  return r;
}

// Stages (2..4) of `stage_bytes` that fit both the budget and `avail` bytes.
__device__ __forceinline__ int stage_count_fit(size_t stage_bytes, size_t avail) {
  int ns = stage_count(stage_bytes);
  while (ns > 2 && (size_t)ns * stage_bytes > avail) --ns;
  return ns;
}

// cp.async.wait_group takes an immediate: wait until at most n (0..3) groups are pending
__device__ __forceinline__ void cp_async_wait_pending(int n) {
  if (n >= 3) asm volatile("cp.async.wait_group 3;\n" ::: "memory");
  else if (n == 2) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
  else if (n == 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

constexpr int kGramTfParts = 296;
constexpr int kGramRows = 32;       // fewest rows per shared-memory chunk (a multiple of 8)
constexpr int kGramStageTarget = 24 * 1024;   // bytes a chunk brings in per barrier

// Rows per chunk: about kGramStageTarget bytes of the two lists, a multiple of 8 in
// [kGramRows, 512], so that narrow products still move many rows per CTA barrier.
__host__ __device__ __forceinline__ int gram_chunk_rows(int P, int Q, int elem_bytes) {
  int r = kGramStageTarget / ((P + Q) * elem_bytes);
  r = r / 8 * 8;
  return r < kGramRows ? kGramRows : (r > 512 ? 512 : r);
}

__host__ __device__ __forceinline__ size_t gram_smem_bytes(int P, int Q, int elem_bytes) {
  const size_t RP = (2 * P + 7) / 8 * 8, RQ = (2 * Q + 7) / 8 * 8;
  const size_t stage = (size_t)gram_chunk_rows(P, Q, elem_bytes) * (P + Q) * elem_bytes;
  const size_t red = RP * RQ * sizeof(double);
  const size_t st = stage_count(stage) * stage;
  return st > red ? st : red;
}

__device__ __forceinline__ void gram_copy_rows(const BlockList<float>& L, long long r, int nrows,
                                               float2* dst, int crow) {
  int off = 0;
  for (int b = 0; b < L.nblk; ++b) {
    const int cols = L.cols[b];
    const int units = nrows * cols;
    const float2* src = L.p[b] + r * L.ld[b];
    float2* d = dst + (long long)off * crow;
    if (L.ld[b] == cols) {
      if ((units & 1) == 0 && ((uintptr_t)src & 15) == 0 &&
          ((uintptr_t)d & 15) == 0) {
        // complex64 run that starts and ends on 16 bytes: two values per copy
        for (int u = 2 * threadIdx.x; u < units; u += 2 * blockDim.x) {
          const unsigned sa = (unsigned)__cvta_generic_to_shared(d + u);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(sa), "l"(src + u) : "memory");
        }
      } else {
        for (int u = threadIdx.x; u < units; u += blockDim.x) {
          const unsigned sa = (unsigned)__cvta_generic_to_shared(d + u);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" :: "r"(sa), "l"(src + u) : "memory");
        }
      }
    } else {
      for (int u = threadIdx.x; u < units; u += blockDim.x) {
        const int rr = u / cols, c = u - rr * cols;
        const unsigned sa = (unsigned)__cvta_generic_to_shared(d + u);
        const float2* g = src + (long long)rr * L.ld[b] + c;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" :: "r"(sa), "l"(g) : "memory");
      }
    }
    off += cols;
  }
}

// Gram partial C' = A'^T B' over rows [r0, r1) of complex64 lists (RP x RQ real
// values to `out`). MMA tiles: 16 columns of A' (M) x 8 columns of B' (N) x 8 rows (K); a warp owns a
// rectangle of kTfMR x kTfMC tiles and a slice of the chunk's 8-row k steps.
// Fragments (m16n8k8 tf32; g = lane / 4, t = lane % 4): A_mma[m][k] = A'[k][m]:
// a0 = (k t, m g), a1 = (k t, m g + 8), a2 = (k t + 4, m g), a3 = (k t + 4, m g + 8);
// B_mma[k][n] = B'[k][n]: b0 = (k t, n g), b1 = (k t + 4, n g); D: (m g, n 2t), (m g, n 2t + 1),
// (m g + 8, n 2t), (m g + 8, n 2t + 1).
constexpr int kTfMR = 3, kTfMC = 3;

__host__ __device__ __forceinline__ int gram_tf32_rects(int P, int Q) {
  const int TR = (2 * P + 15) / 16, TC = (2 * Q + 7) / 8;
  return ((TR + kTfMR - 1) / kTfMR) * ((TC + kTfMC - 1) / kTfMC);
}

static __device__ void gram_core_tf32(const BlockList<float>& A, const BlockList<float>& B,
                                      long long r0, long long r1, double* __restrict__ out,
                                      unsigned char* smem) {
  const int P = A.total(), Q = B.total();
  const int RP = (2 * P + 7) / 8 * 8, RQ = (2 * Q + 7) / 8 * 8;   
  const int TR = (2 * P + 15) / 16, TC = (2 * Q + 7) / 8;
  const int GC = (TC + kTfMC - 1) / kTfMC;
  const int G = gram_tf32_rects(P, Q);
  const int nwarps = blockDim.x >> 5;
  const int slices = nwarps / G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int rect = warp % G, slice = warp / G;
  const bool active_warp = slice < slices;
  const int tr0 = (rect / GC) * kTfMR, tc0 = (rect % GC) * kTfMC;
  const unsigned avail = dyn_smem_bytes();
  int crow = gram_chunk_rows(P, Q, (int)sizeof(float2));
  {
    const int fit = (int)(avail / (2 * (size_t)(P + Q) * sizeof(float2))) / 8 * 8;
    if (crow > fit) crow = fit;
  }
  const size_t stage_elems = (size_t)crow * (P + Q);
  const int NS = stage_count_fit(stage_elems * sizeof(float2), avail);
  float2* stage0 = reinterpret_cast<float2*>(smem);
  // staged real offset of a real column of A' (two per M tile: m g, m g + 8) and of B' (n g)
  int ao[kTfMR][2], aw[kTfMR][2], bo[kTfMC], bw[kTfMC];
#pragma unroll
  for (int i = 0; i < kTfMR; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = (tr0 + i) * 16 + g + 8 * h;
      int c = col >> 1, blk = 0, start = 0;
      while (blk < A.nblk - 1 && c >= A.cols[blk]) { c -= A.cols[blk]; start += A.cols[blk]; ++blk; }
      const bool ok = active_warp && tr0 + i < TR && col < 2 * P;
      ao[i][h] = ok ? 2 * start * crow + 2 * c + (col & 1) : -1;
      aw[i][h] = 2 * A.cols[blk];
    }
#pragma unroll
  for (int j = 0; j < kTfMC; ++j) {
    const int col = (tc0 + j) * 8 + g;
    int c = col >> 1, blk = 0, start = 0;
    while (blk < B.nblk - 1 && c >= B.cols[blk]) { c -= B.cols[blk]; start += B.cols[blk]; ++blk; }
    const bool ok = active_warp && tc0 + j < TC && col < 2 * Q;
    bo[j] = ok ? 2 * (P + start) * crow + 2 * c + (col & 1) : -1;
    bw[j] = 2 * B.cols[blk];
  }
  float acc[kTfMR][kTfMC][4];
#pragma unroll
  for (int i = 0; i < kTfMR; ++i)
#pragma unroll
    for (int j = 0; j < kTfMC; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

  const long long nrows = r1 - r0;
  const int nchunks = (int)((nrows + crow - 1) / crow);
  auto issue = [&](int c) {
    if (c < nchunks) {
      const long long rn = r0 + (long long)c * crow;
      const int nn = (int)min((long long)crow, r1 - rn);
      float2* st = stage0 + (size_t)(c % NS) * stage_elems;
      gram_copy_rows(A, rn, nn, st, crow);
      gram_copy_rows(B, rn, nn, st + (size_t)P * crow, crow);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (int c = 0; c < NS - 1; ++c) issue(c);
  for (int ch = 0; ch < nchunks; ++ch) {
    const long long rc = r0 + (long long)ch * crow;
    const int rows = (int)min((long long)crow, r1 - rc);
    // chunk ch has landed once at most NS - 2 groups are pending; the barrier also means every
    // warp is done with chunk ch - 1, whose stage the next copy reuses
    cp_async_wait_pending(NS - 2);
    __syncthreads();
    issue(ch + NS - 1);
    const float* sr = reinterpret_cast<const float*>(stage0 + (size_t)(ch % NS) * stage_elems);
    if (active_warp) {
      for (int k0 = 8 * slice; k0 < rows; k0 += 8 * slices) {
        const int ra = k0 + t, rb = k0 + t + 4;      // the two rows of this lane's fragments
        const bool oka = ra < rows, okb = rb < rows;
        unsigned bh[kTfMC][2], bl[kTfMC][2];
#pragma unroll
        for (int j = 0; j < kTfMC; ++j) {
          const float x0 = (oka && bo[j] >= 0) ? sr[bo[j] + ra * bw[j]] : 0.f;
          const float x1 = (okb && bo[j] >= 0) ? sr[bo[j] + rb * bw[j]] : 0.f;
          tf32_split(x0, bh[j][0], bl[j][0]);
          tf32_split(x1, bh[j][1], bl[j][1]);
        }
#pragma unroll
        for (int i = 0; i < kTfMR; ++i) {
          const float v0 = (oka && ao[i][0] >= 0) ? sr[ao[i][0] + ra * aw[i][0]] : 0.f;
          const float v1 = (oka && ao[i][1] >= 0) ? sr[ao[i][1] + ra * aw[i][1]] : 0.f;
          const float v2 = (okb && ao[i][0] >= 0) ? sr[ao[i][0] + rb * aw[i][0]] : 0.f;
          const float v3 = (okb && ao[i][1] >= 0) ? sr[ao[i][1] + rb * aw[i][1]] : 0.f;
          unsigned ah[4], al[4];
          tf32_split(v0, ah[0], al[0]);
          tf32_split(v1, ah[1], al[1]);
          tf32_split(v2, ah[2], al[2]);
          tf32_split(v3, ah[3], al[3]);
#pragma unroll
          for (int j = 0; j < kTfMC; ++j) mma_tf32x3(acc[i][j], ah, al, bh[j], bl[j]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  double* gsm = reinterpret_cast<double*>(smem);
  for (int e = threadIdx.x; e < RP * RQ; e += blockDim.x) gsm[e] = 0.0;
  __syncthreads();
  for (int sl = 0; sl < slices; ++sl) {
    if (active_warp && slice == sl) {
#pragma unroll
      for (int i = 0; i < kTfMR; ++i)
#pragma unroll
        for (int j = 0; j < kTfMC; ++j) {
          const int ti = tr0 + i, tj = tc0 + j;
          if (ti < TR && tj < TC) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int rr = ti * 16 + g + 8 * h, cc = tj * 8 + 2 * t;
              if (rr < RP && cc < RQ) {
                gsm[rr * RQ + cc] += (double)acc[i][j][2 * h];
                gsm[rr * RQ + cc + 1] += (double)acc[i][j][2 * h + 1];
              }
            }
          }
        }
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < RP * RQ; e += blockDim.x) out[e] = gsm[e];
}

constexpr int kTfMaxRects = 16;     // rectangles of 12 x 12 columns, a warp each

// threads of a CTA that holds a P x Q product whole, 0 where none does
static inline int gram_tf32_threads(int P, int Q) {
  const int rects = (((2 * P + 7) / 8 + 2) / 3) * (((2 * Q + 7) / 8 + 2) / 3);
  return rects <= 8 ? 256 : (rects <= kTfMaxRects ? 512 : 0);
}

// partial doubles of a product, all parts
static inline size_t gram_tf32_doubles(int P, int Q) {
  return (size_t)kGramTfParts * ((2 * P + 7) / 8 * 8) * ((2 * Q + 7) / 8 * 8);
}

}  // namespace qdkp
