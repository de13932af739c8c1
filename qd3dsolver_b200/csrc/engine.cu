// Batched LOBPCG engine (the served form): many solves resident on the device at once, each in
// a slot, advanced together one LOBPCG iteration per tick. The iteration is scipy's
// (lobpcg.py:688-973, B = M = Y = None, largest = False) exactly as the single-solve driver in
// lobpcg.cu runs it; the difference is that every decision is taken on the device, so a tick is
// a fixed launch sequence over all slots and the host only polls between ticks.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <limits>
#include <type_traits>
#include <vector>

#include "engine_host.cuh"
#include "umma_dev.cuh"

namespace qdkp {

// Rows per CTA of the row kernels: a multiple of the update's chunk, and no more than kEMaxParts CTAs
// for a slot, whose norm partials one CTA then sums (32768 parts of a 128^3 solve would take 0.5 ms).
constexpr int kERowsPerCta = 512;
constexpr int kEMaxParts = 4096;

// GR_RZ: the products of the Rayleigh-Ritz pencil, in one pass (GK_PENCIL or GK_EXPLICIT)
enum GramWhich { GR_XR = 0, GR_RR, GR_PP, GR_RZ };
// UP_XPNEW, UP_AXPNEW: the Ritz update of complex64 slots on the tcgen05 tensor cores, P and X (AP and
// AX) from one pass over [X | R | P] ([AX | AR | AP]); otherwise e_ritz_kernel forms all four.
enum UpdWhich { UP_RPROJ = 0, UP_RNORM, UP_PNORM, UP_APNORM, UP_XPNEW, UP_AXPNEW };

// ---------------------------------------------------------------------------------------------
// residual norms of A X - X lambda: partials per CTA, reduced in the decision kernel. Only where the
// Ritz update does not leave them (complex64 slots updated by the tcgen05 kernels).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kTallThreads)
e_norm_kernel(const ESlot* __restrict__ S, int ns) {
  const ESlot& d = S[slot_of(S, ns, blockIdx.x, &ESlot::row0)];
  const EState* st = d.st;
  if (d.prec != QDKP_C64 || !st->running) return;
  const int part = blockIdx.x - d.row0;
  const float2* AX = blk<float>(d.AX);
  const float2* X = blk<float>(d.X);
  const int m = d.m;
  const long long r0 = (long long)part * d.rows_per_cta;
  const long long r1 = min(d.n, r0 + d.rows_per_cta);
  double acc[kMaxBlock];
#pragma unroll
  for (int j = 0; j < kMaxBlock; ++j) acc[j] = 0.0;
  for (long long r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
#pragma unroll
    for (int j = 0; j < kMaxBlock; ++j) {
      if (j < m) {
        const float2 a = AX[r * m + j], x = X[r * m + j];
        const double l = st->lam[j];
        const double re = (double)a.x - l * (double)x.x, im = (double)a.y - l * (double)x.y;
        acc[j] = fma(re, re, fma(im, im, acc[j]));
      }
    }
  }
  __shared__ double red[kTallThreads / 32][kMaxBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < kMaxBlock; ++j) {
    if (j < m) {
      double v = acc[j];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][j] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < m) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w][threadIdx.x];
    d.npart[(long long)part * m + threadIdx.x] = s;
  }
}

// ---------------------------------------------------------------------------------------------
// per-slot decisions at the top of an iteration (lobpcg.py:688-760)
// ---------------------------------------------------------------------------------------------
// scipy's decisions from the column norms; one thread
static __device__ void e_decide(const ESlot& d, EState* st, const double* __restrict__ nrm) {
  const int m = d.m;
  st->idle = 1; st->r_idle = 1; st->copy_best = 0; st->skip_recompute = 1; st->skip_p = 1; st->skip_pnorm = 1;
  if (!st->running) return;
  if (st->iter >= d.maxiter) { st->running = 0; st->status = QDKP_LOBPCG_MAXITER; return; }
  if (d.stall_iterations > 0 && st->iter - st->best_iter > d.stall_iterations &&
      st->best_iter <= st->iter) {
    st->running = 0; st->status = QDKP_LOBPCG_MAXITER; return;
  }
  st->iter += 1;
  double mean = 0.0, mx = 0.0;
  bool finite = true;
  for (int j = 0; j < m; ++j) {
    st->norms[j] = nrm[j];
    mean += nrm[j];
    mx = fmax(mx, nrm[j]);
    finite = finite && isfinite(nrm[j]);
  }
  mean /= m;
  if (!finite) { st->running = 0; st->status = QDKP_LOBPCG_NONFINITE; return; }
  if (mean < st->smallest) {
    st->smallest = mean;
    st->best_iter = st->iter;
    st->copy_best = 1;
  } else if (mean > ldexp(1.0, d.restart_control) * st->smallest) {
    st->forced = 1;
    st->skip_recompute = 0;
  }
  int ma = 0;
  for (int j = 0; j < m; ++j) {
    st->active[j] = st->active[j] && (nrm[j] > d.tol);
    if (st->active[j]) st->idx[ma++] = j;
  }
  st->ma = ma;
  st->skip_resid = st->resid_ready && ma == m;
  st->resid_ready = 0;
  if (ma == 0) { st->running = 0; st->status = QDKP_LOBPCG_CONVERGED; return; }
  st->explicit_gram = !(mx > d.sqrt_eps && !st->explicit_gram);
  st->idle = 0;
  st->r_idle = 0;
  st->skip_p = st->iter == 0 ? 1 : 0;
}

constexpr int kDecideThreads = 768;    // 32 per column of the widest block

__global__ void __launch_bounds__(kDecideThreads) e_decide_kernel(const ESlot* __restrict__ S) {
  const ESlot& d = S[blockIdx.x];
  EState* st = d.st;
  __shared__ double nrm[kMaxBlock];
  const int m = d.m;
  // a warp per column, parts strided over its lanes: 28 us with a thread per column, 5 us now
  // (7 slots of 860 parts)
  const int c = threadIdx.x >> 5;
  if (c < m) {
    double s = 0.0;
    for (int b = threadIdx.x & 31; b < d.nparts; b += 32) s += d.npart[(long long)b * m + c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) nrm[c] = sqrt(fabs(s));
  }
  __syncthreads();
  if (threadIdx.x == 0) e_decide(d, st, nrm);
  if (!d.snap) return;
  __syncthreads();
  const int* from = reinterpret_cast<const int*>(st);
  int* to = reinterpret_cast<int*>(d.snap);
  for (int i = threadIdx.x; i < (int)(sizeof(EState) / sizeof(int)); i += blockDim.x) to[i] = from[i];
}

// ---------------------------------------------------------------------------------------------
// row kernels: copy of the best iterate, residual gather, P gather (tcgen05 updates only)
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void e_row_body(const ESlot& d, int which, long long r0,
                                           long long r1) {
  const EState* st = d.st;
  const int m = d.m;
  const int ma = st->ma;
  const cplx<T>* X = blk<T>(d.X);
  if (which == RW_COPYBEST) {
    cplx<T>* best = blk<T>(d.best);
    for (long long e = r0 * m + threadIdx.x; e < r1 * m; e += blockDim.x) best[e] = X[e];
  } else if (which == RW_RESID) {
    const cplx<T>* AX = blk<T>(d.AX);
    cplx<T>* Ra = blk<T>(d.Ra);
    for (long long e = r0 * ma + threadIdx.x; e < r1 * ma; e += blockDim.x) {
      const long long r = e / ma;
      const int c = (int)(e - r * ma);
      const int j = st->idx[c];
      const double l = st->lam[j];
      const cplx<T> a = AX[r * m + j], x = X[r * m + j];
      Ra[e] = mk<T>((T)((double)a.x - l * (double)x.x), (T)((double)a.y - l * (double)x.y));
    }
  } else {
    const cplx<T>* P = blk<T>(d.P);
    const cplx<T>* AP = blk<T>(d.AP);
    cplx<T>* Pa = blk<T>(d.Pa);
    cplx<T>* APa = blk<T>(d.APa);
    for (long long e = r0 * ma + threadIdx.x; e < r1 * ma; e += blockDim.x) {
      const long long r = e / ma;
      const int c = (int)(e - r * ma);
      const int j = st->idx[c];
      Pa[e] = P[r * m + j];
      APa[e] = AP[r * m + j];
    }
  }
}

__global__ void __launch_bounds__(kTallThreads)
e_row_kernel(const ESlot* __restrict__ S, int ns, int which) {
  const int k = slot_of(S, ns, blockIdx.x, &ESlot::row0);
  const ESlot& d = S[k];
  const EState* st = d.st;
  if (which == RW_COPYBEST) { if (!st->copy_best) return; }
  else if (st->idle || (which == RW_RESID && st->skip_resid)) return;
  else if (which == RW_GATHERP && (st->skip_p || d.prec != QDKP_C64)) return;
  const long long r0 = (long long)(blockIdx.x - d.row0) * d.rows_per_cta;
  const long long r1 = min(d.n, r0 + d.rows_per_cta);
  if (d.prec == QDKP_C64) e_row_body<float>(d, which, r0, r1);
  else e_row_body<double>(d, which, r0, r1);
}

// ---------------------------------------------------------------------------------------------
// Gram products, multi-slot (gram_dev.cuh). complex64 slots form them in FP64 too: the Gram matrices
// of the search stay exact to FP64 (a split TF32 form loses convergence in the explicit-Gram regime
// of scipy's method).
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ bool gram_task(const ESlot& d, int which, GramTask<T>& t, double2*& out, double2*& outS) {
  const EState* st = d.st;
  if (which == GR_PP ? st->idle || st->skip_p : st->r_idle) return false;
  const int m = d.m, ma = st->ma;
  const int mp = which == GR_RZ ? st->mp : 0;          // decided beside the products on R
  t.nblk = 0; t.tc = 0;
  t.m = m; t.ma = ma; t.mp = mp; t.n = d.n;
  t.fault = d.fault;
  t.a0 = 0; t.b0 = 0;
  auto add = [&](double2* p, int ld, int cols) {
    t.p[t.nblk] = blk<T>(p); t.ld[t.nblk] = ld; t.cols[t.nblk] = cols;
    ++t.nblk;
    t.tc += cols;
  };
  outS = nullptr;
  switch (which) {
    case GR_XR:
      add(d.X, m, m); add(d.Ra, ma, ma);
      t.P = m; t.b0 = m; t.Q = ma; t.kind = GK_FULL; out = d.W;
      return true;
    case GR_RR:
      add(d.Ra, ma, ma);
      t.P = t.Q = ma; t.kind = GK_HERM; out = nullptr;      // e_chol_kernel's
      return true;
    case GR_PP:          // all columns; e_chol_kernel takes the active ones
      add(d.P, m, m);
      t.P = t.Q = m; t.kind = GK_HERM; out = nullptr;
      return true;
    default:
      add(d.X, m, m); add(d.Ra, ma, ma); add(d.Pa, ma, mp);
      t.P = m + ma + mp;
      if (st->explicit_gram) {
        add(d.AX, m, m); add(d.ARa, ma, ma); add(d.APa, ma, mp);
        t.Q = 2 * t.P; t.kind = GK_EXPLICIT;
      } else {
        add(d.ARa, ma, ma); add(d.APa, ma, mp);
        t.b0 = m + ma; t.Q = mp + ma + mp; t.kind = GK_PENCIL;
      }
      out = d.gT; outS = d.gS;
      return true;
  }
}

// Launched once per distinct block width m present: the warps of a CTA (and so the order of every
// sum) then depend only on the slot's own sizes, never on which other solves share the batch.
template <typename T>
__device__ void e_gram_body(const ESlot& d, int which, int part, unsigned char* smem) {
  __shared__ GramTask<T> t;
  __shared__ int go;
  if (threadIdx.x == 0) {
    double2 *out, *outS;
    go = gram_task<T>(d, which, t, out, outS);
  }
  __syncthreads();
  if (go) gram_core(t, part, d.gparts, (int)blockIdx.y, which == GR_PP ? d.ppart : d.gpart, smem);
}

__global__ void __launch_bounds__(32 * (kGramMaxWarps + 1), 1)
e_gram_kernel(const ESlot* __restrict__ S, int ns, int which, int m_only) {
  extern __shared__ __align__(16) unsigned char gsm_e[];
  const int k = slot_of(S, ns, blockIdx.x, &ESlot::gram0);
  const ESlot& d = S[k];
  if (d.m != m_only) return;
  const int part = blockIdx.x - d.gram0;
  if (d.prec == QDKP_C64) e_gram_body<float>(d, which, part, gsm_e);
  else e_gram_body<double>(d, which, part, gsm_e);
}

// a row of CTAs (blockIdx.y) per slot
template <typename T>
__device__ void e_gram_reduce_body(const ESlot& d, int which) {
  __shared__ GramTask<T> t;
  __shared__ double2 *out, *outS;
  __shared__ int go;
  if (threadIdx.x == 0) {
    double2 *o = nullptr, *oS = nullptr;
    go = gram_task<T>(d, which, t, o, oS);
    out = o; outS = oS;
  }
  __syncthreads();
  if (go)
    gram_reduce_core(t, d.gparts, d.gpart, (int)blockIdx.x, (int)gridDim.x,
                     [&](int i, int j, double2 v) { gram_put(t, i, j, v, out, outS); });
}

__global__ void __launch_bounds__(kGramRedThreads)
e_gram_reduce_kernel(const ESlot* __restrict__ S, int which) {
  const ESlot& d = S[blockIdx.y];
  if (d.prec == QDKP_C64) e_gram_reduce_body<float>(d, which);
  else e_gram_reduce_body<double>(d, which);
}

// ---------------------------------------------------------------------------------------------
// block updates, multi-slot (FP64 MMA, rows staged through shared memory: in-place safe)
// ---------------------------------------------------------------------------------------------
template <typename T>
struct UpdTask {
  BlockList<T> A;
  const double2* C[3];
  const double2* C2[3];      // second output (tcgen05 only)
  const int* gather;         // columns of A's block 0 (NULL: as they stand)
  int q, accumulate, neg;
  cplx<T> *Y, *Y2;
};

// packed: P's active columns have been gathered into Pa (the tcgen05 kernels read whole rows);
// otherwise the P updates read them from P itself (the gather took 152 us of a tick of seven slots)
template <typename T>
__device__ bool upd_lists(const ESlot& d, int which, bool packed, UpdTask<T>& u) {
  const EState* st = d.st;
  if (which == UP_PNORM || which == UP_APNORM ? st->idle : st->r_idle) return false;
  const int m = d.m, ma = st->ma;
  u.accumulate = 0; u.neg = 0;
  u.Y2 = nullptr; u.gather = nullptr;
  auto set = [&](int i, double2* p, int ld, int c, const double2* cf) {
    u.A.p[i] = blk<T>(p); u.A.ld[i] = ld; u.A.cols[i] = c; u.C[i] = cf; u.C2[i] = nullptr;
  };
  u.A.nblk = 1;
  switch (which) {
    case UP_RPROJ: set(0, d.X, m, m, d.W); u.q = ma; u.Y = blk<T>(d.Ra); u.accumulate = 1; u.neg = 1; return true;
    case UP_RNORM: set(0, d.Ra, ma, ma, d.U); u.q = ma; u.Y = blk<T>(d.Ra); return true;
    case UP_PNORM: case UP_APNORM: {
      if (st->skip_pnorm) return false;
      const bool ax = which == UP_APNORM;
      if (packed) {
        set(0, ax ? d.APa : d.Pa, ma, ma, d.Up);
      } else {
        set(0, ax ? d.AP : d.P, m, ma, d.Up);
        u.gather = st->idx;
      }
      u.q = ma; u.Y = blk<T>(ax ? d.APa : d.Pa);
      return true;
    }
    default: {        // UP_XPNEW / UP_AXPNEW
      const bool ax = which == UP_AXPNEW;
      const int mp = st->mp;
      u.A.nblk = mp ? 3 : 2;
      set(0, ax ? d.AX : d.X, m, m, nullptr);            // X rows do not enter P
      set(1, ax ? d.ARa : d.Ra, ma, ma, d.Cr);
      set(2, ax ? d.APa : d.Pa, ma, mp, d.Cp);
      u.C2[0] = d.Cx; u.C2[1] = d.Cr; u.C2[2] = d.Cp;
      u.q = m;
      u.Y = blk<T>(ax ? d.AP : d.P);
      u.Y2 = blk<T>(ax ? d.AX : d.X);
      return true;
    }
  }
}

// One launch per precision present; CTAs of the other precision's slots return at once. complex128: 80 registers,
// three CTAs an SM where their rings fit (up to 12 columns; a solve of 33x33x25 x 6 3.42 ms with two, 3.32 ms so).
template <typename T>
__global__ void __launch_bounds__(kUpdThreads, std::is_same<T, double>::value ? 3 : 2)
e_update_kernel(const ESlot* __restrict__ S, int ns, int first) {
  const int which = first + blockIdx.y;               // PNORM and APNORM are one launch
  extern __shared__ __align__(16) unsigned char usm_e[];
  const int k = slot_of(S, ns, blockIdx.x, &ESlot::row0);
  const ESlot& d = S[k];
  constexpr int prec = std::is_same<T, float>::value ? QDKP_C64 : QDKP_C128;
  if (d.prec != prec) return;
  const long long r0 = (long long)(blockIdx.x - d.row0) * d.rows_per_cta;
  const long long r1 = min(d.n, r0 + d.rows_per_cta);
  UpdTask<T> u;
  if (!upd_lists<T>(d, which, false, u)) return;
  if constexpr (std::is_same<T, float>::value)
    update_rows_tf32(u.A, u.C, u.q, r0, r1, u.Y, (long long)u.q, u.accumulate, u.neg, usm_e, u.gather);
  else
    update_rows(u.A, u.C, u.q, r0, r1, u.Y, (long long)u.q, u.accumulate, u.neg, usm_e, u.gather);
}

// The Ritz update of X, AX, P and AP with the residual norms (and, while every column is active, the
// residual block) of the new iterate, one pass (ritz_rows). The next tick's decision kernel reads
// the norms. One launch per precision present.
template <typename T>
__global__ void __launch_bounds__(kUpdThreads, 2)
e_ritz_kernel(const ESlot* __restrict__ S, int ns) {
  extern __shared__ __align__(16) unsigned char usm_r[];
  const int k = slot_of(S, ns, blockIdx.x, &ESlot::row0);
  const ESlot& d = S[k];
  constexpr int prec = std::is_same<T, float>::value ? QDKP_C64 : QDKP_C128;
  const EState* st = d.st;
  if (d.prec != prec || st->r_idle) return;
  const int part = blockIdx.x - d.row0;
  const long long r0 = (long long)part * d.rows_per_cta;
  RitzArgs<T> t;
  t.X = blk<T>(d.X); t.R = blk<T>(d.Ra); t.P = blk<T>(d.P);
  t.AX = blk<T>(d.AX); t.AR = blk<T>(d.ARa); t.AP = blk<T>(d.AP);
  t.Pin = blk<T>(d.Pa); t.APin = blk<T>(d.APa);
  t.m = d.m; t.ma = st->ma; t.mp = st->mp;
  t.Rout = t.ma == t.m ? t.R : nullptr;
  t.Cx = d.Cx; t.Cr = d.Cr; t.Cp = d.Cp;
  t.lam = st->lam;
  t.npart = d.npart + (long long)part * d.m;
  if constexpr (std::is_same<T, float>::value) ritz_rows_tf32(t, r0, min(d.n, r0 + d.rows_per_cta), usm_r);
  else ritz_rows(t, r0, min(d.n, r0 + d.rows_per_cta), usm_r);
}

// complex64 slots: the same updates on the tcgen05 tensor cores (umma_dev.cuh). The CTAs split
// the 128-row tiles of the group's complex64 slots (slot k's tiles start at utile0) into
// contiguous ranges, one CTA per SM; a CTA's tiles of one slot form one pipelined run. A wait
// that gives up leaves NaN in the outputs, which the slot's next residual check turns into status
// nonfinite. Every row is computed the same way whichever CTA holds it, so results do not depend
// on the mix of slots.
__global__ void __launch_bounds__(kUmmaThreads, 1)
e_update_umma_kernel(const ESlot* __restrict__ S, int ns, int which, int utiles, int m_max) {
  extern __shared__ __align__(128) unsigned char usm_u[];
  const bool fused = which == UP_XPNEW || which == UP_AXPNEW;
  const UmmaPlan pl = umma_plan((fused ? 3 : 1) * m_max, m_max, fused ? 2 : 1, m_max, m_max);
  const long long per = (utiles + gridDim.x - 1) / gridDim.x;
  long long c = (long long)blockIdx.x * per;
  const long long c1 = min((long long)utiles, c + per);
  if (c >= c1) return;
  UmmaCtx cx;
  umma_ctx_init(cx, pl);
  bool ok = true;
  while (c < c1) {
    int k = -1;
    long long nt = 0;
    for (int j = 0; j < ns && k < 0; ++j) {
      if (S[j].prec != QDKP_C64) continue;
      nt = (S[j].n + kUmmaRows - 1) / kUmmaRows;
      if (c >= S[j].utile0 && c < S[j].utile0 + nt) k = j;
    }
    if (k < 0) break;                                  // uniform; not reached
    const ESlot& d = S[k];
    const long long seg_end = min(c1, (long long)d.utile0 + nt);
    UpdTask<float> u;
    if (upd_lists<float>(d, which, true, u)) {
      const long long r0 = (c - d.utile0) * kUmmaRows;
      const long long r1 = min(d.n, (seg_end - d.utile0) * kUmmaRows);
      if (ok) {
        ok = update_rows_umma(pl, cx, u.A, u.C, u.q, r0, r1, u.Y, (long long)u.q, u.accumulate, u.neg,
                              usm_u, u.C2, u.Y2);
        if (!ok && threadIdx.x == 0) raise_device_fault(d.fault);
      } else {
        float2* const Ys[2] = {u.Y, u.Y2};
        umma_fill_nan(Ys, u.Y2 ? 2 : 1, u.q, r0, r1, (long long)u.q);
      }
    }
    c = seg_end;
  }
  umma_ctx_free(cx);
}

// ---------------------------------------------------------------------------------------------
// per-slot Cholesky steps and Rayleigh-Ritz
// ---------------------------------------------------------------------------------------------
// the sums of a Gram product's parts into the m x m matrix G (upper triangle), by this CTA alone
template <typename T>
__device__ void e_small_gram(const ESlot& d, int which, double2* __restrict__ G) {
  __shared__ GramTask<T> t;
  if (threadIdx.x == 0) {
    double2 *o, *oS;
    gram_task<T>(d, which, t, o, oS);
  }
  __syncthreads();
  gram_reduce_herm(t, d.gparts, which == GR_PP ? d.ppart : d.gpart, G);
}

// R^H R (which = GR_RR) or P^H P (GR_PP, of which the active columns are taken) summed, its Cholesky
// factor, and U^-1 in d.U (d.Up). One kernel: reduction and factorisation are a launch of latency each (13 us
// and 15 us at 12 columns).
template <int WHICH>
__global__ void __launch_bounds__(kSmallThreads) e_chol_kernel(const ESlot* __restrict__ S) {
  extern __shared__ double2 ssm_e[];
  __shared__ double rinv[kMaxSmall];
  const ESlot& d = S[blockIdx.x];
  EState* st = d.st;
  if (WHICH == GR_PP ? st->idle : st->r_idle) return;
  const int n = st->ma, m = WHICH == GR_PP ? d.m : n;
  if (WHICH == GR_PP && st->skip_p) {      // iteration 0: no P yet, restart stays as it is
    if (threadIdx.x == 0) { st->skip_pnorm = 1; st->mp = st->restart ? 0 : n; }
    return;
  }
  double2* G = ssm_e;
  double2* C = ssm_e + d.m * d.m;
  if (d.prec == QDKP_C64) e_small_gram<float>(d, WHICH, G);
  else e_small_gram<double>(d, WHICH, G);
  if (WHICH == GR_PP && n < m) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e - i * n;
      C[e] = G[st->idx[i] * m + st->idx[j]];
    }
    __syncthreads();
    double2* swap = G;
    G = C;
    C = swap;
  }
  const int fail = rr_cholesky(G, n, rinv, 0);
  if (!fail) {
    rr_upper_inverse(G, n, rinv, C);
    double2* U = WHICH == GR_PP ? d.Up : d.U;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) U[e] = C[e];
  }
  if (threadIdx.x != 0) return;
  if (WHICH == GR_RR) {
    if (fail) { st->running = 0; st->status = QDKP_LOBPCG_RCHOL_BREAKDOWN; st->r_idle = 1; }
  } else {
    st->skip_pnorm = fail ? 1 : 0;
    st->restart = fail ? 1 : st->forced;
    st->mp = st->restart ? 0 : n;
  }
}

// gramA / gramB of lobpcg.py:826-909 from S = W^H W and T = W^H AW, then the generalized eigh,
// with the fall back to the two-block pencil when the three-block one is not definite.
__device__ void e_assemble(const ESlot& d, const EState* st, int restart, int& dim) {
  const int m = d.m, ma = st->ma, mp = restart ? 0 : st->mp;
  const int tot = m + st->ma + st->mp;      // rows of gT; layout of the explicit products
  dim = m + ma + mp;
  const bool ex = st->explicit_gram;
  const int nAB = st->ma + st->mp;          // non-explicit gT = [X|R|P]^H [AR|AP]: tot x nAB
  for (int e = threadIdx.x; e < dim * dim; e += blockDim.x) {
    int i = e / dim, j = e - i * dim;
    bool lower = i > j;
    if (lower) { const int t = i; i = j; j = t; }
    const bool iX = i < m, iR = i >= m && i < m + ma, jX = j < m, jR = j >= m && j < m + ma;
    double2 Tij, Tji, Sij;
    if (ex) {
      Tij = d.gT[i * tot + j]; Tji = d.gT[j * tot + i]; Sij = d.gS[i * tot + j];
    } else {
      // column j >= m of W^H AW is column j - m of [AR | AP]; gS = [X|R]^H P (m+ma x mp)
      Tij = j >= m ? d.gT[i * nAB + (j - m)] : make_double2(0.0, 0.0);
      Tji = (i >= m && j >= m) ? d.gT[j * nAB + (i - m)] : make_double2(0.0, 0.0);
      Sij = (j >= m + ma && i < m + ma) ? d.gS[i * st->mp + (j - m - ma)] : make_double2(0.0, 0.0);
    }
    const double2 herm = make_double2(0.5 * (Tij.x + Tji.x), 0.5 * (Tij.y - Tji.y));
    double2 a, b;
    if (iX && jX) {
      if (ex) { a = herm; b = Sij; }
      else { a = make_double2(i == j ? st->lam[i] : 0.0, 0.0); b = make_double2(i == j ? 1.0 : 0.0, 0.0); }
    } else if (iX && jR) {
      a = Tij; b = ex ? Sij : make_double2(0.0, 0.0);
    } else if ((iR && jR) || (!iX && !iR && !jX && !jR)) {
      a = ex ? herm : Tij;
      b = ex ? Sij : make_double2(i == j ? 1.0 : 0.0, 0.0);
    } else {
      a = Tij; b = Sij;
    }
    if (lower) { a.y = -a.y; b.y = -b.y; }
    d.gA[e] = a;
    d.gB[e] = b;
  }
  __syncthreads();
}

// c64_ritz: the Ritz update of complex64 slots is e_ritz_kernel's too. One launch per eigensolve size
// present; a slot's is its own widest pencil's.
template <int CLASS>
__global__ void __launch_bounds__(kSmallThreads) e_rr_kernel(const ESlot* __restrict__ S, int c64_ritz) {
  const ESlot& d = S[blockIdx.x];
  EState* st = d.st;
  if (st->r_idle || rr_class(3 * d.m) != CLASS) return;
  __shared__ int use_restart, ok, dim_s;
  if (threadIdx.x == 0) { use_restart = st->mp == 0; ok = 0; }
  __syncthreads();
  for (int attempt = 0; attempt < 2; ++attempt) {
    int dim;
    e_assemble(d, st, use_restart, dim);
    // only the first m Ritz pairs are kept
    // without the explicit products gramB is the identity on X and R (all of it without P)
    const int k0 = st->explicit_gram ? 0 : d.m + st->ma;
    const int r = block_eigh<CLASS>(d.gA, d.gB, dim, d.w, d.E, d.scr, d.m, 2 * dim * dim, k0);
    if (threadIdx.x == 0) { ok = r == 0; dim_s = dim; }
    __syncthreads();
    if (ok || use_restart) break;
    if (threadIdx.x == 0) use_restart = 1;    // drop P and retry (lobpcg.py:891-909)
    __syncthreads();
  }
  if (!ok) {
    if (threadIdx.x == 0) { st->running = 0; st->status = QDKP_LOBPCG_EIGH_BREAKDOWN; st->r_idle = 1; }
    return;
  }
  const int m = d.m, ma = st->ma, dim = dim_s;
  const int mp = dim - m - ma;
  for (int e = threadIdx.x; e < dim * m; e += blockDim.x) {
    const int i = e / m, j = e - i * m;
    const double2 v = d.E[i * dim + j];
    if (i < m) d.Cx[i * m + j] = v;
    else if (i < m + ma) d.Cr[(i - m) * m + j] = v;
    else d.Cp[(i - m - ma) * m + j] = v;
  }
  if (threadIdx.x < m) st->lam[threadIdx.x] = d.w[threadIdx.x];
  if (threadIdx.x == 0) {
    st->restart = use_restart ? 1 : st->restart;
    st->mp = mp;
    st->resid_ready = ma == m && (c64_ritz || d.prec != QDKP_C64);
  }
}

}  // namespace qdkp

// =============================================================================================
// host side
// =============================================================================================
namespace qdkp {

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

SlotLayout slot_layout(int64_t n, int m, int prec, int n_blocks) {
  SlotLayout L;
  L.blk = align256((size_t)n * m * (prec == QDKP_C64 ? sizeof(float2) : sizeof(double2)));
  L.small = align256((size_t)(3 * m) * (3 * m) * sizeof(double2));
  const int64_t rows = (n + kEMaxParts - 1) / kEMaxParts;
  L.rows_per_cta = (int)std::max<int64_t>(kERowsPerCta, (rows + kUpdChunk - 1) / kUpdChunk * kUpdChunk);
  L.nparts = (int)((n + L.rows_per_cta - 1) / L.rows_per_cta);
  L.npart = align256((size_t)L.nparts * m * sizeof(double));
  L.gparts = gram_parts(n);
  // the widest task: 3 m x 6 m columns (explicit Gram matrices)
  L.gpart = align256(gram_partial_elems(3 * m, 6 * m) * sizeof(double2));
  L.ppart = align256(gram_partial_elems(m, m) * sizeof(double2));
  L.total = align256(sizeof(EState)) + n_blocks * L.blk + 13 * L.small +
            align256(3 * m * sizeof(double)) + L.npart + L.gpart + L.ppart;
  return L;
}

void slot_carve(ESlot& d, void* ws, const SlotLayout& L, int64_t n, int m, int prec, int n_blocks) {
  char* p = static_cast<char*>(ws);
  auto take = [&](size_t b) { char* r = p; p += align256(b); return r; };
  d.st = (EState*)take(sizeof(EState));
  double2** const blocks[10] = {&d.X, &d.AX, &d.P, &d.AP, &d.best, &d.Ra, &d.ARa, &d.Pa, &d.APa, &d.T};
  for (int i = 0; i < 10; ++i) *blocks[i] = i < n_blocks ? (double2*)take(L.blk) : nullptr;
  d.W = (double2*)take(L.small); d.U = (double2*)take(L.small); d.Up = (double2*)take(L.small);
  d.gS = (double2*)take(L.small); d.gT = (double2*)take(L.small); d.gA = (double2*)take(L.small);
  d.gB = (double2*)take(L.small); d.E = (double2*)take(L.small);
  d.scr = (double2*)take(2 * L.small);
  d.Cx = (double2*)take(L.small); d.Cr = (double2*)take(L.small); d.Cp = (double2*)take(L.small);
  d.w = (double*)take(3 * m * sizeof(double));
  d.npart = (double*)take(L.npart);
  d.gpart = (double*)take(L.gpart);
  d.ppart = (double*)take(L.ppart);
  d.n = n; d.m = m; d.prec = prec;
  d.nparts = L.nparts; d.gparts = L.gparts; d.rows_per_cta = L.rows_per_cta;
  d.gram0 = d.row0 = 0;
  d.utile0 = -1;
  d.snap = nullptr;
  d.fault = nullptr;
}

void slot_params(ESlot& d, EState& s, const qdkp_lobpcg_params* prm, const double* lam) {
  const double eps = d.prec == QDKP_C64 ? (double)std::numeric_limits<float>::epsilon()
                                        : std::numeric_limits<double>::epsilon();
  d.folded = prm->folded;
  d.sqrt_eps = std::sqrt(eps);
  d.tol = prm->tol > 0 ? prm->tol : std::sqrt(std::numeric_limits<double>::epsilon()) * (double)d.n;
  d.maxiter = prm->maxiter;
  d.stall_iterations = prm->stall_iterations;
  d.restart_control = prm->restart_control > 0 ? prm->restart_control : 20;
  s = EState{};
  s.running = 1;
  s.status = QDKP_LOBPCG_MAXITER;
  s.iter = -1; s.idle = 1; s.r_idle = 1;
  s.ma = d.m; s.mp = 0; s.restart = 1; s.forced = 0; s.explicit_gram = 0;
  s.best_iter = prm->maxiter; s.skip_recompute = 1; s.skip_p = 1; s.skip_pnorm = 1;
  s.smallest = std::numeric_limits<double>::max();
  for (int j = 0; j < d.m; ++j) { s.active[j] = 1; s.lam[j] = lam[j]; }
}

static int launch_gram_multi(const EGroup& G, int which, cudaStream_t st) {
  int mmax = 0;
  for (int m : G.widths) {
    // the warps for the product at full width; panels for the most rectangles any active width and
    // either pencil can form (the CTAs of panels that stay empty return at once)
    const int P = which == GR_RZ ? 3 * m : m, Q = P, tc = which == GR_RZ ? 6 * m : 2 * m;
    const int kind = which == GR_XR ? GK_FULL : (which == GR_RZ ? GK_PENCIL : GK_HERM);
    const GramShape sh = gram_shape(kind, P, Q, m, m, m);
    const int most = (P + kGramRect - 1) / kGramRect * (((which == GR_RZ ? 6 * m : m) + kGramRect - 1) / kGramRect);
    const size_t smem = std::max(gram_smem<double>(tc, sh.warps), gram_smem<float>(tc, sh.warps));
    e_gram_kernel<<<dim3(G.gram_ctas, (most + sh.warps - 1) / sh.warps), 32 * (sh.warps + 1), smem, st>>>(
        G.d_slots, G.ns, which, m);
    count_launch();
    mmax = std::max(mmax, m);
  }
  QDKP_CUDA_TRY(cudaGetLastError());
  if (which == GR_RR || which == GR_PP) return QDKP_OK;      // e_chol_kernel adds the parts
  const int outs = (which == GR_RZ ? 3 * mmax * 6 * mmax : mmax * mmax);
  e_gram_reduce_kernel<<<dim3((outs + 31) / 32, G.ns), kGramRedThreads, 0, st>>>(G.d_slots, which);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

static int launch_umma_multi(const EGroup& G, int which, cudaStream_t st) {
  const bool fused = which == UP_XPNEW || which == UP_AXPNEW;
  const UmmaPlan pl = umma_plan((fused ? 3 : 1) * G.m_max, G.m_max, fused ? 2 : 1, G.m_max, G.m_max);
  if (!pl.nout_pass) { set_error("tcgen05 update plan does not fit shared memory"); return QDKP_ERR_ARG; }
  e_update_umma_kernel<<<std::min(G.utiles, G.nsm), kUmmaThreads, pl.bytes, st>>>(
      G.d_slots, G.ns, which, G.utiles, G.m_max);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

// the updates which .. which + count - 1 (UpdWhich), in one launch where no tcgen05 kernel runs them
static int launch_update_multi(const EGroup& G, int which, cudaStream_t st, int count = 1) {
  if (G.hx_ns[0]) {
    e_update_kernel<double><<<dim3(G.row_ctas, count), kUpdThreads, update_smem_bytes(G.m_max, G.m_max), st>>>(
        G.d_slots, G.ns, which);
    count_launch();
  }
  if (G.hx_ns[1] && c64_update_tcgen05()) {
    for (int i = 0; i < count; ++i) {
      const int rc = launch_umma_multi(G, which + i, st);
      if (rc) return rc;
    }
  } else if (G.hx_ns[1]) {
    e_update_kernel<float><<<dim3(G.row_ctas, count), kUpdThreads, update_tf32_smem_bytes(G.m_max, G.m_max), st>>>(
        G.d_slots, G.ns, which);
    count_launch();
  }
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

static int launch_ritz_multi(const EGroup& G, cudaStream_t st) {
  if (G.hx_ns[0]) {
    e_ritz_kernel<double><<<G.row_ctas, kUpdThreads, ritz_smem_bytes(G.m_max), st>>>(G.d_slots, G.ns);
    count_launch();
  }
  if (G.hx_ns[1] && c64_update_tcgen05()) {
    int rc = launch_umma_multi(G, UP_XPNEW, st);
    if (rc) return rc;
    rc = launch_umma_multi(G, UP_AXPNEW, st);
    if (rc) return rc;
  } else if (G.hx_ns[1]) {
    e_ritz_kernel<float><<<G.row_ctas, kUpdThreads, ritz_tf32_smem_bytes(G.m_max), st>>>(G.d_slots, G.ns);
    count_launch();
  }
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

bool group_umma(const EGroup& G) { return G.hx_ns[1] && c64_update_tcgen05(); }

#define ETRY(x) do { const int rc_ = (x); if (rc_ != QDKP_OK) return rc_; } while (0)

int launch_decide(const EGroup& G, cudaStream_t st) {
  if (group_umma(G)) {
    e_norm_kernel<<<G.row_ctas, kTallThreads, 0, st>>>(G.d_slots, G.ns);
    count_launch();
  }
  e_decide_kernel<<<G.ns, kDecideThreads, 0, st>>>(G.d_slots);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

int launch_p_chain(const EGroup& G, cudaStream_t st) {
  e_row_kernel<<<G.row_ctas, kTallThreads, 0, st>>>(G.d_slots, G.ns, RW_COPYBEST);
  count_launch();
  if (group_umma(G)) {
    e_row_kernel<<<G.row_ctas, kTallThreads, 0, st>>>(G.d_slots, G.ns, RW_GATHERP);
    count_launch();
  }
  ETRY(launch_gram_multi(G, GR_PP, st));
  e_chol_kernel<GR_PP><<<G.ns, kSmallThreads, 2 * (size_t)G.m_max * G.m_max * sizeof(double2), st>>>(G.d_slots);
  count_launch();
  return launch_update_multi(G, UP_PNORM, st, 2);
}

int launch_r_chain(const EGroup& G, cudaStream_t st) {
  e_row_kernel<<<G.row_ctas, kTallThreads, 0, st>>>(G.d_slots, G.ns, RW_RESID);
  count_launch();
  ETRY(launch_gram_multi(G, GR_XR, st));
  ETRY(launch_update_multi(G, UP_RPROJ, st));
  ETRY(launch_gram_multi(G, GR_RR, st));
  e_chol_kernel<GR_RR><<<G.ns, kSmallThreads, 2 * (size_t)G.m_max * G.m_max * sizeof(double2), st>>>(G.d_slots);
  count_launch();
  return launch_update_multi(G, UP_RNORM, st);
}

int launch_ritz_step(const EGroup& G, cudaStream_t st) {
  ETRY(launch_gram_multi(G, GR_RZ, st));
  const size_t rr_smem = 2 * (size_t)(3 * G.m_max) * (3 * G.m_max) * sizeof(double2);
  bool cls[3] = {};
  for (int m : G.widths) cls[rr_class(3 * m)] = true;
  const int c64_ritz = !group_umma(G);
  if (cls[0]) e_rr_kernel<0><<<G.ns, kSmallThreads, rr_smem, st>>>(G.d_slots, c64_ritz);
  if (cls[1]) e_rr_kernel<1><<<G.ns, kSmallThreads, rr_smem, st>>>(G.d_slots, c64_ritz);
  if (cls[2]) e_rr_kernel<2><<<G.ns, kSmallThreads, rr_smem, st>>>(G.d_slots, c64_ritz);
  count_launch(cls[0] + cls[1] + cls[2]);
  QDKP_CUDA_TRY(cudaGetLastError());
  return launch_ritz_multi(G, st);
}

void set_slot_kernel_limits() {
  const int big = 200 * 1024;
  cudaFuncSetAttribute(e_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramMaxSmem);
  cudaFuncSetAttribute(e_update_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_update_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_ritz_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_ritz_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_update_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       kUmmaSmemLimit);
  cudaFuncSetAttribute(e_rr_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_rr_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_rr_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_chol_kernel<GR_RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(e_chol_kernel<GR_PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
}

namespace {

struct SlotHost {
  bool used = false;
  const qdkp_operator* op = nullptr;
  qdkp_lobpcg_params prm{};
  ESlot d{};
  size_t gpart_doubles = 0;
  int64_t applies = 0;
};

// The used slots are split into up to kEGroups groups whose ticks run on streams of their own:
// the groups share no data, so while one group is in its latency-bound kernels (the
// Rayleigh-Ritz eigensolve and the small Cholesky, reduction and decision kernels, one CTA per
// slot) the other group's tall kernels fill the GPU. A slot's kernels and partitions are the
// same in any group, so grouping changes no result.
constexpr int kEGroups = 2;

}  // namespace
}  // namespace qdkp

struct qdkp_engine {
  int device = 0;
  int max_slots = 0;
  std::vector<qdkp::SlotHost> slots;
  qdkp::ESlot* d_slots = nullptr;      // compact array of the used slots (group after group)
  qdkp::HXSlot* d_hx = nullptr;        // H.X descriptors, kEGroups x 8 x max_slots
  int ns = 0;                          // used slots
  int ngroups = 0;
  int nsm = 148;                       // SMs of the device (grid of the tcgen05 updates)
  qdkp::EGroup grp[qdkp::kEGroups];
  bool dirty = true;
  // CUDA graph of one tick of each group over the current slot layout, replayed by qdkp_engine_step on
  // the group's own stream (ordered after and before the caller's stream by events)
  cudaStream_t gstream = nullptr, gstream2 = nullptr;   // group 0 and group 1
  // the work on P of a single group, forked from and joined to the group's stream within a tick
  cudaStream_t pstream = nullptr;
  cudaEvent_t ev_dec = nullptr, ev_p = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr, ev_fork = nullptr, ev_join = nullptr;
  cudaGraphExec_t graph[qdkp::kEGroups] = {};
  bool use_graph = true;
  long long launches_per_tick = 0;     // kernels one tick launches (graph replays count them)
};

namespace qdkp {
namespace {

// Host helpers on a slot's tall blocks, in the slot's precision (the block pointers are typed
// double2 in ESlot and hold complex64 values for a QDKP_C64 slot).
int apply_folded(const SlotHost& h, const void* V, int c, void* out, cudaStream_t st) {
  const ESlot& d = h.d;
  if (h.prm.folded) return launch_folded(h.op, V, c, d.T, out, c, c, h.prm.sigma, d.prec, st);
  return launch_apply(h.op, V, c, out, c, c, 0.0, 0, d.prec, st);
}

template <typename T>
BlockList<T> one(const void* p, int c) {
  BlockList<T> L;
  L.nblk = 1; L.p[0] = static_cast<const cplx<T>*>(p); L.ld[0] = c; L.cols[0] = c;
  return L;
}

int gram1(const SlotHost& h, const void* A, const void* B, int m, double2* out,
          cudaStream_t st) {
  const size_t elems = h.gpart_doubles / 2;
  double2* part = reinterpret_cast<double2*>(h.d.gpart);
  if (h.d.prec == QDKP_C64)
    return launch_gram(one<float>(A, m), one<float>(B, m), h.d.n, part, elems, out, st);
  return launch_gram(one<double>(A, m), one<double>(B, m), h.d.n, part, elems, out, st);
}

// Y (n x q) = A (n x m) C (m x q)
int update1(const SlotHost& h, const void* A, int m, const double2* C, int q, void* Y,
            cudaStream_t st) {
  const double2* Cs[1] = {C};
  if (h.d.prec == QDKP_C64)
    return launch_update(one<float>(A, m), Cs, q, h.d.n, static_cast<float2*>(Y), q, 0, st);
  return launch_update(one<double>(A, m), Cs, q, h.d.n, static_cast<double2*>(Y), q, 0, st);
}

// out[j] = sum_r |A[r, j] - lambda_j B[r, j]|^2, summed on the device into out (device)
int colnorm1(const SlotHost& h, const void* A, const void* B, const double* lam, int m,
             double* out, cudaStream_t st) {
  const ESlot& d = h.d;
  if (d.prec == QDKP_C64)
    return launch_colnorm2<float>(static_cast<const float2*>(A), m, static_cast<const float2*>(B),
                                  m, lam, m, d.n, d.npart, d.nparts, out, st);
  return launch_colnorm2<double>(static_cast<const double2*>(A), m,
                                 static_cast<const double2*>(B), m, lam, m, d.n, d.npart,
                                 d.nparts, out, st);
}

int copy1(const SlotHost& h, const void* src, int m, void* dst, cudaStream_t st) {
  if (h.d.prec == QDKP_C64)
    return launch_copy<float, float>(static_cast<const float2*>(src), m, m, h.d.n,
                                     static_cast<float2*>(dst), m, st);
  return launch_copy<double, double>(static_cast<const double2*>(src), m, m, h.d.n,
                                     static_cast<double2*>(dst), m, st);
}

int read_sync(void* host, const void* dev, size_t bytes, cudaStream_t st) {
  QDKP_CUDA_TRY(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  return QDKP_OK;
}

// descriptors of group g (slots `ids`, compact-array positions from `base` on)
int build_group(qdkp_engine* e, int g, const std::vector<int>& ids, int base, cudaStream_t st) {
  EGroup& G = e->grp[g];
  G = EGroup();
  G.d_slots = e->d_slots + base;
  G.d_hx = e->d_hx + (size_t)g * 8 * e->max_slots;
  std::vector<ESlot> compact;
  std::vector<HXSlot> hx(8 * (size_t)e->max_slots);
  int gram0 = 0, row0 = 0, m_max = 1, utile0 = 0;
  int tile0[2] = {0, 0}, kp[2] = {0, 0}, nf[2] = {0, 0};
  for (int i : ids) {
    SlotHost& h = e->slots[i];
    ESlot d = h.d;
    d.gram0 = gram0; gram0 += d.gparts;
    d.row0 = row0; row0 += (int)((d.n + d.rows_per_cta - 1) / d.rows_per_cta);
    d.utile0 = -1;
    if (d.prec == QDKP_C64) { d.utile0 = utile0; utile0 += (int)((d.n + kUmmaRows - 1) / kUmmaRows); }
    h.d = d;
    compact.push_back(d);
    const int pi = d.prec == QDKP_C64 ? 1 : 0;
    const int k = kp[pi]++;
    nf[pi] += h.prm.folded ? 1 : 0;
    const qdkp_operator* op = h.op;
    m_max = std::max(m_max, d.m);
    const int tiles = apply_tiles(op->n_sites, d.m);
    for (int t = 0; t < 4; ++t) {
      HXSlot x{};
      x.rec = pi ? (const void*)op->rec32 : (const void*)op->rec64;
      x.msk = op->nbmask; x.N = (int)op->n_sites;
      x.sx = op->ny * op->nz; x.sy = op->nz;
      x.tile0 = tile0[pi]; x.cb = apply_cb_weight(op);
      x.sigma = h.prm.sigma;
      x.shifted = h.prm.folded ? 1 : 0;
      const bool recompute = t < 2;
      if (recompute) { x.m = d.m; x.m_dev = nullptr; x.ld_same = 0; x.ldx = d.m; x.ldy = d.m; }
      else { x.m = 0; x.m_dev = &d.st->ma; x.ld_same = 1; }
      const int* skipflag = recompute ? &d.st->skip_recompute : &d.st->r_idle;
      if (h.prm.folded) {
        x.X = (t == 0) ? (const void*)d.X : (t == 2) ? (const void*)d.Ra : (const void*)d.T;
        x.Y = (t == 0 || t == 2) ? (void*)d.T : (t == 1) ? (void*)d.AX : (void*)d.ARa;
        x.skip = skipflag;
      } else {
        x.X = recompute ? (const void*)d.X : (const void*)d.Ra;
        x.Y = recompute ? (void*)d.AX : (void*)d.ARa;
        x.skip = skipflag;                    // phases 1 and 3 are for folded slots only
      }
      hx[((size_t)pi * 4 + t) * e->max_slots + k] = x;
    }
    tile0[pi] += tiles;
  }
  G.ns = (int)compact.size();
  G.gram_ctas = gram0; G.row_ctas = row0;
  G.utiles = utile0;
  G.nsm = e->nsm;
  for (int pi = 0; pi < 2; ++pi) { G.hx_ns[pi] = kp[pi]; G.hx_tiles[pi] = tile0[pi]; G.hx_folded[pi] = nf[pi]; }
  G.m_max = m_max;
  for (const ESlot& d : compact)
    if (std::find(G.widths.begin(), G.widths.end(), d.m) == G.widths.end()) G.widths.push_back(d.m);
  std::sort(G.widths.begin(), G.widths.end());
  if (G.ns) {
    QDKP_CUDA_TRY(cudaMemcpyAsync(G.d_slots, compact.data(), compact.size() * sizeof(ESlot),
                                  cudaMemcpyHostToDevice, st));
    QDKP_CUDA_TRY(cudaMemcpyAsync(G.d_hx, hx.data(), hx.size() * sizeof(HXSlot),
                                  cudaMemcpyHostToDevice, st));
  }
  return QDKP_OK;
}

// Split the used slots into groups, balancing rows x block width greedily in slot order.
int rebuild(qdkp_engine* e, cudaStream_t st) {
  std::vector<int> ids[kEGroups];
  double load[kEGroups] = {};
  int used = 0;
  for (int i = 0; i < e->max_slots; ++i) used += e->slots[i].used ? 1 : 0;
  const int ng = std::max(1, std::min(kEGroups, used));
  for (int i = 0; i < e->max_slots; ++i) {
    const SlotHost& h = e->slots[i];
    if (!h.used) continue;
    int g = 0;
    for (int c = 1; c < ng; ++c) if (load[c] < load[g]) g = c;
    ids[g].push_back(i);
    load[g] += (double)h.d.n * h.d.m;
  }
  e->ns = used;
  e->ngroups = ng;
  int base = 0;
  for (int g = 0; g < kEGroups; ++g) {
    if (g >= ng) { e->grp[g] = EGroup(); continue; }
    const int rc = build_group(e, g, ids[g], base, st);
    if (rc) return rc;
    base += (int)ids[g].size();
  }
  e->dirty = false;
  return QDKP_OK;
}

// One H.X phase of a tick: a multi-slot launch per precision and kind (folded or not) present. The
// recomputation of A X (phases 0 and 1) runs on a forced restart only: a grid of every tile would
// take 18 us a phase (seven slots) to find that out.
int launch_hx_phase(const qdkp_engine* e, const EGroup& G, int phase, cudaStream_t st) {
  for (int pi = 0; pi < 2; ++pi) {
    if (!G.hx_ns[pi]) continue;
    const HXSlot* slots = G.d_hx + ((size_t)pi * 4 + phase) * e->max_slots;
    const int prec = pi ? QDKP_C64 : QDKP_C128, most = phase < 2 ? 4 * e->nsm : G.hx_tiles[pi];
    const int basis = phase % 2 ? HX_X_UNCOUPLED : HX_Y_UNCOUPLED;
    int rc = QDKP_OK;
    if (G.hx_folded[pi]) rc = launch_apply_multi(slots, G.hx_ns[pi], G.hx_tiles[pi], prec, basis, most, st);
    if (rc == QDKP_OK && G.hx_folded[pi] < G.hx_ns[pi] && phase % 2 == 0)
      rc = launch_apply_multi(slots, G.hx_ns[pi], G.hx_tiles[pi], prec, 0, most, st);
    if (rc) return rc;
  }
  return QDKP_OK;
}

// One LOBPCG iteration of every running slot of group g. The work on P needs nothing of the work on R.
// A group by itself runs it beside R's, on a stream forked from st after the decisions and joined
// before the pencil; two groups fill each other's gaps already (a sweep of 14 complex64 slots 28.7 ms
// with the P work in line, 29.7 ms forked).
int tick(const qdkp_engine* e, int g, cudaStream_t st) {
  const EGroup& G = e->grp[g];
  if (!G.ns) return QDKP_OK;
  ETRY(launch_decide(G, st));
  // (two tcgen05 kernels would contend for an SM's tensor memory: one after the other)
  const cudaStream_t ps = e->ngroups > 1 || group_umma(G) ? st : e->pstream;
  if (ps != st) {
    QDKP_CUDA_TRY(cudaEventRecord(e->ev_dec, st));
    QDKP_CUDA_TRY(cudaStreamWaitEvent(ps, e->ev_dec, 0));
  }
  int rc = launch_p_chain(G, ps);
  if (rc == QDKP_OK) rc = launch_r_chain(G, st);
  for (int phase = 0; phase < 4 && rc == QDKP_OK; ++phase) rc = launch_hx_phase(e, G, phase, st);
  if (ps != st) {
    // after an error too, so that a capture in progress ends with no stream left forked
    const cudaError_t r1 = cudaEventRecord(e->ev_p, ps);
    const cudaError_t r2 = cudaStreamWaitEvent(st, e->ev_p, 0);
    if (rc == QDKP_OK) { QDKP_CUDA_TRY(r1); QDKP_CUDA_TRY(r2); }
  }
  if (rc != QDKP_OK) return rc;
  return launch_ritz_step(G, st);
}

}  // namespace
}  // namespace qdkp

namespace qdkp {

// `ticks` ticks of every group: group 0 on `st`, group 1 on the engine's second stream, forked
// from and joined back to `st` (the groups share no data, so their ticks interleave freely)
static int run_ticks(qdkp_engine* e, int ticks, cudaStream_t st) {
  int rc = QDKP_OK;
  if (e->ngroups > 1) {
    QDKP_CUDA_TRY(cudaEventRecord(e->ev_fork, st));
    QDKP_CUDA_TRY(cudaStreamWaitEvent(e->gstream2, e->ev_fork, 0));
  }
  for (int t = 0; t < ticks && rc == QDKP_OK; ++t) rc = tick(e, 0, st);
  for (int t = 0; t < ticks && rc == QDKP_OK && e->ngroups > 1; ++t) rc = tick(e, 1, e->gstream2);
  if (e->ngroups > 1) {
    // join even after an error, so that a capture in progress ends with no stream left forked
    const cudaError_t r1 = cudaEventRecord(e->ev_join, e->gstream2);
    const cudaError_t r2 = cudaStreamWaitEvent(st, e->ev_join, 0);
    if (rc == QDKP_OK && (r1 != cudaSuccess || r2 != cudaSuccess)) {
      set_error(std::string("engine stream join: ") + cudaGetErrorString(r1 != cudaSuccess ? r1 : r2));
      rc = QDKP_ERR_CUDA;
    }
  }
  return rc;
}

static void destroy_pstream(qdkp_engine* e) {
  if (e->pstream) { cudaStreamSynchronize(e->pstream); cudaStreamDestroy(e->pstream); }
  if (e->ev_dec) cudaEventDestroy(e->ev_dec);
  if (e->ev_p) cudaEventDestroy(e->ev_p);
}

static void drop_graph(qdkp_engine* e) {
  for (cudaGraphExec_t& g : e->graph) {
    if (g) cudaGraphExecDestroy(g);
    g = nullptr;
  }
}

// Capture a tick of each group of the current layout, from the group's stream, into e->graph. (One tick,
// replayed: a graph of all of a call's ticks cost 5 us a kernel to build whenever the slots changed.)
static int capture_ticks(qdkp_engine* e) {
  drop_graph(e);
  e->launches_per_tick = 0;
  for (int gi = 0; gi < e->ngroups; ++gi) {
    const cudaStream_t st = gi ? e->gstream2 : e->gstream;
    QDKP_CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const long long l0 = launches_so_far();
    const int rc = tick(e, gi, st);
    // captured launches are not executions: take them back off the counter
    const long long captured = launches_so_far() - l0;
    count_launch((int)-captured);
    e->launches_per_tick += captured;
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(st, &g);
    if (rc != QDKP_OK) { if (g) cudaGraphDestroy(g); drop_graph(e); return rc; }
    if (ce != cudaSuccess) {
      drop_graph(e);
      set_error(std::string("engine graph capture: ") + cudaGetErrorString(ce));
      return QDKP_ERR_CUDA;
    }
    const cudaError_t ie = cudaGraphInstantiate(&e->graph[gi], g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) {
      e->graph[gi] = nullptr;
      drop_graph(e);
      set_error(std::string("engine graph instantiate: ") + cudaGetErrorString(ie));
      return QDKP_ERR_CUDA;
    }
  }
  return QDKP_OK;
}

}  // namespace qdkp

using namespace qdkp;

extern "C" {

int qdkp_engine_create(int max_slots, int device, qdkp_engine** out) {
  QDKP_CHECK_ARG(out && max_slots >= 1 && max_slots <= 4096, "bad engine arguments");
  QDKP_CUDA_TRY(cudaSetDevice(device));
  auto* e = new qdkp_engine();
  e->device = device;
  e->max_slots = max_slots;
  e->slots.resize(max_slots);
  cudaError_t err = cudaMalloc(&e->d_slots, sizeof(ESlot) * max_slots);
  if (err == cudaSuccess) err = cudaMalloc(&e->d_hx, sizeof(HXSlot) * kEGroups * 8 * max_slots);
  if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&e->gstream, cudaStreamNonBlocking);
  if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&e->gstream2, cudaStreamNonBlocking);
  if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->ev_in, cudaEventDisableTiming);
  if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->ev_out, cudaEventDisableTiming);
  if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->ev_fork, cudaEventDisableTiming);
  if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->ev_join, cudaEventDisableTiming);
  if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&e->pstream, cudaStreamNonBlocking);
  if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->ev_dec, cudaEventDisableTiming);
  if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->ev_p, cudaEventDisableTiming);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&e->nsm, cudaDevAttrMultiProcessorCount, device);
  if (err != cudaSuccess) {
    set_error(std::string("engine tables: ") + cudaGetErrorString(err));
    cudaFree(e->d_slots); cudaFree(e->d_hx);
    if (e->gstream) cudaStreamDestroy(e->gstream);
    if (e->gstream2) cudaStreamDestroy(e->gstream2);
    if (e->ev_in) cudaEventDestroy(e->ev_in);
    if (e->ev_out) cudaEventDestroy(e->ev_out);
    if (e->ev_fork) cudaEventDestroy(e->ev_fork);
    if (e->ev_join) cudaEventDestroy(e->ev_join);
    destroy_pstream(e);
    delete e;
    return QDKP_ERR_CUDA;
  }
  set_slot_kernel_limits();
  *out = e;
  return QDKP_OK;
}

int qdkp_engine_destroy(qdkp_engine* e) {
  if (!e) return QDKP_OK;
  cudaSetDevice(e->device);
  drop_graph(e);
  if (e->gstream) { cudaStreamSynchronize(e->gstream); cudaStreamDestroy(e->gstream); }
  if (e->gstream2) { cudaStreamSynchronize(e->gstream2); cudaStreamDestroy(e->gstream2); }
  if (e->ev_in) cudaEventDestroy(e->ev_in);
  if (e->ev_out) cudaEventDestroy(e->ev_out);
  if (e->ev_fork) cudaEventDestroy(e->ev_fork);
  if (e->ev_join) cudaEventDestroy(e->ev_join);
  destroy_pstream(e);
  cudaFree(e->d_slots);
  cudaFree(e->d_hx);
  delete e;
  return QDKP_OK;
}

size_t qdkp_engine_slot_workspace_size(const qdkp_operator* op, const qdkp_lobpcg_params* prm) {
  if (!op || !prm || prm->block < 1 || prm->block > kMaxBlock) return 0;
  if (prm->precision != QDKP_C128 && prm->precision != QDKP_C64) return 0;
  return slot_layout((int64_t)op->n_bands * op->n_sites, prm->block, prm->precision, 10).total;
}

int qdkp_engine_admit(qdkp_engine* e, const qdkp_operator* op, const qdkp_lobpcg_params* prm,
                      const void* X0, void* ws, size_t ws_bytes, void* stream, int* slot_out) {
  QDKP_CHECK_ARG(e && op && prm && X0 && ws && slot_out, "NULL argument");
  QDKP_CHECK_ARG(op->n_bands == 8, "the batched engine serves eight-band operators");
  QDKP_CHECK_ARG(prm->block >= 1 && prm->block <= kMaxBlock, "block must be in [1, 24]");
  QDKP_CHECK_ARG(prm->precision == QDKP_C128 || prm->precision == QDKP_C64,
                 "precision must be QDKP_C128 or QDKP_C64");
  QDKP_CHECK_ARG(op->device == e->device, "operator lives on another device");
  const int64_t n = (int64_t)op->n_bands * op->n_sites;
  const int m = prm->block;
  QDKP_CHECK_ARG(n >= 5 * m, "problem too small for LOBPCG");
  QDKP_CHECK_ARG(n * m < (int64_t(1) << 31), "n * block must stay below 2^31 elements");
  const SlotLayout L = slot_layout(n, m, prm->precision, 10);
  if (ws_bytes < L.total) { set_error("engine slot workspace too small"); return QDKP_ERR_WORKSPACE; }
  int id = -1;
  for (int i = 0; i < e->max_slots; ++i) if (!e->slots[i].used) { id = i; break; }
  if (id < 0) { set_error("no free engine slot"); return QDKP_ERR_WORKSPACE; }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SlotHost& h = e->slots[id];
  h = SlotHost();
  h.op = op;
  h.prm = *prm;
  ESlot& d = h.d;
  slot_carve(d, ws, L, n, m, prm->precision, 10);
  d.fault = device_fault_flag(e->device);
  h.gpart_doubles = L.gpart / sizeof(double);
  int rc;
#define ATRY(x) do { rc = (x); if (rc != QDKP_OK) return rc; } while (0)
  // X = orthonormalise(X0) (lobpcg.py:620-630)
  if (d.prec == QDKP_C64)
    ATRY((launch_copy<double, float>(static_cast<const double2*>(X0), m, m, n,
                                     reinterpret_cast<float2*>(d.X), m, st)));
  else
    ATRY(launch_copy(static_cast<const double2*>(X0), m, m, n, d.X, m, st));
  ATRY(gram1(h, d.X, d.X, m, d.gS, st));
  ATRY(launch_chol_inv(d.gS, m, d.U, (int*)d.w, st));
  int stat = 0;
  ATRY(read_sync(&stat, d.w, sizeof(int), st));
  if (stat) { set_error("Linearly dependent initial approximations"); return QDKP_ERR_NUMERIC; }
  ATRY(update1(h, d.X, m, d.U, m, d.X, st));
  // initial Ritz vectors (lobpcg.py:633-660)
  ATRY(apply_folded(h, d.X, m, d.AX, st));
  ATRY(gram1(h, d.X, d.AX, m, d.gT, st));
  ATRY(launch_eigh(d.gT, nullptr, m, d.w, d.E, d.scr, (int*)d.Up, st));
  ATRY(read_sync(&stat, d.Up, sizeof(int), st));
  // the eigensolve fails only on non-finite input (a NaN or inf in the operator's fields or in
  // X0): the slot is admitted already stopped with status nonfinite, and retires like any other
  const bool nonfinite = stat != 0;
  std::vector<double> w(m, std::numeric_limits<double>::quiet_NaN());
  if (!nonfinite) {
    ATRY(update1(h, d.X, m, d.E, m, d.X, st));
    ATRY(update1(h, d.AX, m, d.E, m, d.AX, st));
    // the first tick's decision kernel reads the partials left in npart
    ATRY(colnorm1(h, d.AX, d.X, d.w, m, d.gpart, st));
    ATRY(read_sync(w.data(), d.w, m * sizeof(double), st));
  }
  EState s0;
  slot_params(d, s0, prm, w.data());
  if (nonfinite) { s0.running = 0; s0.status = QDKP_LOBPCG_NONFINITE; }
  QDKP_CUDA_TRY(cudaMemcpyAsync(d.st, &s0, sizeof(EState), cudaMemcpyHostToDevice, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  ATRY(check_device_fault(e->device));
#undef ATRY
  h.used = true;
  e->dirty = true;
  *slot_out = id;
  return QDKP_OK;
}

int qdkp_engine_step(qdkp_engine* e, int ticks, void* stream) {
  QDKP_CHECK_ARG(e && ticks >= 0, "bad arguments");
  if (const int rc = check_device_fault(e->device)) return rc;      // of earlier ticks
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  QDKP_CUDA_TRY(cudaSetDevice(e->device));
  if (e->dirty) {
    drop_graph(e);
    int rc = rebuild(e, st);
    if (rc) return rc;
  }
  if (ticks == 0 || e->ns == 0) return QDKP_OK;
  if (!e->use_graph) return run_ticks(e, ticks, st);
  // the tick sequence is fixed for a slot layout: replay it as one graph launch
  if (!e->graph[0]) {
    QDKP_CUDA_TRY(cudaStreamSynchronize(st));   // descriptor uploads of rebuild() landed
    int rc = capture_ticks(e);
    if (rc) return rc;
  }
  // the groups' ticks interleave freely: each replays its own graph on its own stream
  QDKP_CUDA_TRY(cudaEventRecord(e->ev_in, st));
  QDKP_CUDA_TRY(cudaStreamWaitEvent(e->gstream, e->ev_in, 0));
  if (e->ngroups > 1) QDKP_CUDA_TRY(cudaStreamWaitEvent(e->gstream2, e->ev_in, 0));
  cudaError_t le = cudaSuccess;
  for (int t = 0; t < ticks && le == cudaSuccess; ++t) {
    le = cudaGraphLaunch(e->graph[0], e->gstream);
    if (le == cudaSuccess && e->ngroups > 1) le = cudaGraphLaunch(e->graph[1], e->gstream2);
  }
  count_launch(e->launches_per_tick * ticks);
  QDKP_CUDA_TRY(cudaEventRecord(e->ev_out, e->gstream));
  QDKP_CUDA_TRY(cudaStreamWaitEvent(st, e->ev_out, 0));
  if (e->ngroups > 1) {
    QDKP_CUDA_TRY(cudaEventRecord(e->ev_join, e->gstream2));
    QDKP_CUDA_TRY(cudaStreamWaitEvent(st, e->ev_join, 0));
  }
  QDKP_CUDA_TRY(le);
  return QDKP_OK;
}

int qdkp_engine_set_graphs(qdkp_engine* e, int enable) {
  QDKP_CHECK_ARG(e != nullptr, "NULL engine");
  e->use_graph = enable != 0;
  if (!e->use_graph) drop_graph(e);
  return QDKP_OK;
}

int qdkp_engine_poll(qdkp_engine* e, int* state, int* status, int* iterations, void* stream) {
  QDKP_CHECK_ARG(e && state, "bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  std::vector<EState> hs(e->max_slots);
  for (int i = 0; i < e->max_slots; ++i) {
    const SlotHost& h = e->slots[i];
    if (!h.used) continue;
    QDKP_CUDA_TRY(cudaMemcpyAsync(&hs[i], h.d.st, sizeof(EState), cudaMemcpyDeviceToHost, st));
  }
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  for (int i = 0; i < e->max_slots; ++i) {
    const SlotHost& h = e->slots[i];
    state[i] = !h.used ? -1 : (hs[i].running ? 1 : 0);
    if (status) status[i] = h.used ? hs[i].status : -1;
    if (iterations) iterations[i] = h.used ? hs[i].iter + 1 : 0;
  }
  return check_device_fault(e->device);
}

int qdkp_engine_retire(qdkp_engine* e, int slot, double* lambda_out, void* V,
                       double* residuals_out, qdkp_lobpcg_info* info, void* stream) {
  QDKP_CHECK_ARG(e && slot >= 0 && slot < e->max_slots && e->slots[slot].used, "bad slot");
  QDKP_CHECK_ARG(lambda_out && V && info, "NULL argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SlotHost& h = e->slots[slot];
  ESlot& d = h.d;
  const int m = d.m;
  const int64_t n = d.n;
  int rc;
#define RTRY(x) do { rc = (x); if (rc != QDKP_OK) return rc; } while (0)
  EState s;
  RTRY(read_sync(&s, d.st, sizeof(EState), st));
  std::vector<double> lam(s.lam, s.lam + m), rn2(m), norms(m);
  // residuals of the last iterate; it becomes the best one if it improved (lobpcg.py:975-995)
  double* dl = d.w;
  QDKP_CUDA_TRY(cudaMemcpyAsync(dl, lam.data(), m * sizeof(double), cudaMemcpyHostToDevice, st));
  RTRY(colnorm1(h, d.AX, d.X, dl, m, d.gpart, st));
  RTRY(read_sync(rn2.data(), d.gpart, m * sizeof(double), st));
  double mean = 0.0;
  for (int j = 0; j < m; ++j) mean += std::sqrt(std::fabs(rn2[j]));
  mean /= m;
  int best_iter = s.best_iter;
  if (s.status != QDKP_LOBPCG_NONFINITE && mean < s.smallest) {
    RTRY(copy1(h, d.X, m, d.best, st));
    best_iter = s.iter + 1;
  }
  if (s.status == QDKP_LOBPCG_NONFINITE) {
    // a non-finite residual: no Rayleigh-Ritz on it; the last iterate is returned as it is with
    // NaN Ritz values and residuals, and the slot is freed for the next request
    if (d.prec == QDKP_C64)
      RTRY((launch_copy<float, double>(reinterpret_cast<const float2*>(d.X), m, m, n,
                                       static_cast<double2*>(V), m, st)));
    else
      RTRY((launch_copy<double, double>(reinterpret_cast<const double2*>(d.X), m, m, n,
                                        static_cast<double2*>(V), m, st)));
    QDKP_CUDA_TRY(cudaStreamSynchronize(st));
    for (int j = 0; j < m; ++j) lambda_out[j] = std::numeric_limits<double>::quiet_NaN();
    if (residuals_out)
      for (int j = 0; j < m; ++j) residuals_out[j] = std::numeric_limits<double>::quiet_NaN();
    std::memset(info, 0, sizeof(*info));
    info->iterations = std::min(s.iter + 1, h.prm.maxiter + 3);
    info->best_iteration = best_iter;
    info->status = s.status;
    info->explicit_gram = s.explicit_gram;
    info->best_mean_residual = s.smallest;
    h.used = false;
    e->dirty = true;
    return check_device_fault(e->device);
  }
  // final Rayleigh-Ritz on the best iterate (lobpcg.py:1009-1060)
  RTRY(apply_folded(h, d.best, m, d.AX, st));
  RTRY(gram1(h, d.best, d.AX, m, d.gT, st));
  RTRY(gram1(h, d.best, d.best, m, d.gS, st));
  {
    std::vector<double2> t((size_t)m * m), s2((size_t)m * m), a((size_t)m * m), bb((size_t)m * m);
    RTRY(read_sync(t.data(), d.gT, t.size() * sizeof(double2), st));
    RTRY(read_sync(s2.data(), d.gS, s2.size() * sizeof(double2), st));
    for (int i = 0; i < m; ++i)
      for (int j = 0; j < m; ++j) {
        const double2 x = t[(size_t)i * m + j], y = t[(size_t)j * m + i];
        a[(size_t)i * m + j] = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
        const double2 u = s2[(size_t)i * m + j], v = s2[(size_t)j * m + i];
        bb[(size_t)i * m + j] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
      }
    QDKP_CUDA_TRY(cudaMemcpyAsync(d.gA, a.data(), a.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
    QDKP_CUDA_TRY(cudaMemcpyAsync(d.gB, bb.data(), bb.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
  }
  RTRY(launch_eigh(d.gA, d.gB, m, d.w, d.E, d.scr, (int*)d.Up, st));
  int stat = 0;
  RTRY(read_sync(&stat, d.Up, sizeof(int), st));
  if (stat) { set_error("eigh has failed in lobpcg postprocessing"); return QDKP_ERR_NUMERIC; }
  RTRY(read_sync(lam.data(), d.w, m * sizeof(double), st));
  // Ritz vectors of the best iterate; a complex64 slot forms them in its own precision (in the
  // free folded scratch T) and widens them into the caller's complex128 V
  void* Vs = d.prec == QDKP_C64 ? static_cast<void*>(d.T) : V;
  RTRY(update1(h, d.best, m, d.E, m, Vs, st));
  RTRY(update1(h, d.AX, m, d.E, m, d.AX, st));
  RTRY(colnorm1(h, d.AX, Vs, d.w, m, d.gpart, st));
  if (d.prec == QDKP_C64)
    RTRY((launch_copy<float, double>(reinterpret_cast<const float2*>(d.T), m, m, n,
                                     static_cast<double2*>(V), m, st)));
  RTRY(read_sync(rn2.data(), d.gpart, m * sizeof(double), st));
  bool all = true;
  for (int j = 0; j < m; ++j) {
    norms[j] = std::sqrt(std::fabs(rn2[j]));
    all = all && norms[j] <= d.tol;
  }
  std::memcpy(lambda_out, lam.data(), m * sizeof(double));
  if (residuals_out) std::memcpy(residuals_out, norms.data(), m * sizeof(double));
  int status = s.status;
  if (status == QDKP_LOBPCG_MAXITER && all) status = QDKP_LOBPCG_CONVERGED;
  std::memset(info, 0, sizeof(*info));
  info->iterations = std::min(best_iter + 2, h.prm.maxiter + 3);
  info->best_iteration = best_iter;
  info->status = status;
  info->explicit_gram = s.explicit_gram;
  info->best_mean_residual = s.smallest;
#undef RTRY
  h.used = false;
  e->dirty = true;
  return check_device_fault(e->device);
}

}  // extern "C"
