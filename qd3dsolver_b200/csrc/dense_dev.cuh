// Device building blocks shared by the single-solve and batched LOBPCG kernels: FP64 MMA,
// block-list element access, and the one-CTA Cholesky / triangular inverse / Hermitian
// eigensolver routines.
#pragma once
#include "blockops.cuh"
#include "gram_dev.cuh"

namespace qdkp {

// Eigen-decomposition of the Hermitian C in S0 (n x n, shared memory), with S1 = I on entry:
// Householder reduction to tridiagonal form (C <- H C H, Q <- Q H, H = I - tau v v^H, one column
// per step), a diagonal phase that makes the sub-diagonal real, and the implicit QL iteration
// with shifts of Bowdler, Martin, Reinsch and Wilkinson (the tql2 scheme) on the real symmetric
// tridiagonal matrix. One thread runs the QL recurrences and records each sweep's plane
// rotations; then every row of the eigenvector matrix Z applies them, so the rotations stay
// exactly orthogonal even inside clusters of (near-)equal eigenvalues. On return S0's diagonal
// holds the eigenvalues (unsorted) and S1 the eigenvectors of C (columns). gtmp: n * n global
// double2 of scratch. Returns nonzero (block-uniform) if an eigenvalue needed more than 60 QL
// iterations (only non-finite input gets there).
static __device__ int block_tql(double2* S0, double2* S1, int n, double2* gtmp) {
  __shared__ double2 hv[kMaxSmall], hp[kMaxSmall], hq[kMaxSmall], ph[kMaxSmall];
  __shared__ double td[kMaxSmall], tb[kMaxSmall], rc[kMaxSmall], rs[kMaxSmall];
  __shared__ int ri[kMaxSmall];
  __shared__ double s_tau, s_K;
  __shared__ int s_nrot, s_state;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // ---- Householder reduction ----
  for (int k = 0; k + 2 < n; ++k) {
    if (warp == 0) {
      double nx2 = 0.0;
      for (int i = k + 1 + lane; i < n; i += 32) {
        const double2 x = S0[i * n + k];
        nx2 += x.x * x.x + x.y * x.y;
      }
      for (int o = 16; o > 0; o >>= 1) nx2 += __shfl_xor_sync(0xffffffffu, nx2, o);
      const double2 x0 = S0[(k + 1) * n + k];
      const double ax0 = sqrt(x0.x * x0.x + x0.y * x0.y);
      const double nx = sqrt(nx2);
      // alpha = -phase(x0) |x|; v = x - alpha e_1; v^H v = 2 |x| (|x| + |x0|)
      const double2 phs = ax0 > 0.0 ? make_double2(x0.x / ax0, x0.y / ax0) : make_double2(1.0, 0.0);
      for (int i = lane; i < n; i += 32) {
        double2 v = make_double2(0.0, 0.0);
        if (i == k + 1) v = make_double2(x0.x + phs.x * nx, x0.y + phs.y * nx);
        else if (i > k + 1) v = S0[i * n + k];
        hv[i] = v;
      }
      // a column whose |x| (|x| + |x0|) is below the smallest normal double is left as it is
      // (entries of that size do not change a tridiagonal of a matrix of ordinary scale; 1 / it
      // would overflow)
      const double den = nx * (nx + ax0);
      if (lane == 0) s_tau = den >= 2.2250738585072014e-308 ? 1.0 / den : 0.0;
    }
    __syncthreads();
    const double tau = s_tau;
    // every thread has read tau before warp 0 can move on to the next column and rewrite it
    __syncthreads();
    if (tau == 0.0) continue;                      // column already reduced (uniform)
    // p = tau C v and q = Q v, a warp per row
    for (int i = warp; i < n; i += nwarps) {
      double2 sp = make_double2(0.0, 0.0), sq = make_double2(0.0, 0.0);
      for (int j = k + 1 + lane; j < n; j += 32) {
        const double2 v = hv[j];
        cfma(sp, S0[i * n + j], v);
        cfma(sq, S1[i * n + j], v);
      }
      for (int o = 16; o > 0; o >>= 1) {
        sp.x += __shfl_xor_sync(0xffffffffu, sp.x, o); sp.y += __shfl_xor_sync(0xffffffffu, sp.y, o);
        sq.x += __shfl_xor_sync(0xffffffffu, sq.x, o); sq.y += __shfl_xor_sync(0xffffffffu, sq.y, o);
      }
      if (lane == 0) { hp[i] = make_double2(tau * sp.x, tau * sp.y); hq[i] = sq; }
    }
    __syncthreads();
    if (warp == 0) {                               // K = tau / 2 v^H p
      double2 s = make_double2(0.0, 0.0);
      for (int i = k + 1 + lane; i < n; i += 32) cfmac(s, hv[i], hp[i]);
      for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      }
      // v^H C v is real for Hermitian C; its rounding residue in s.y is dropped
      if (lane == 0) s_K = 0.5 * tau * s.x;
    }
    __syncthreads();
    const double K = s_K;
    // C <- C - v w^H - w v^H with w = p - K v;  Q <- Q - tau q v^H
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e - i * n;
      const double2 vi = hv[i], vj = hv[j];
      const double2 wi = make_double2(hp[i].x - K * vi.x, hp[i].y - K * vi.y);
      const double2 wj = make_double2(hp[j].x - K * vj.x, hp[j].y - K * vj.y);
      double2 c = S0[e];
      // c -= vi conj(wj) + wi conj(vj)
      c.x -= vi.x * wj.x + vi.y * wj.y + wi.x * vj.x + wi.y * vj.y;
      c.y -= vi.y * wj.x - vi.x * wj.y + wi.y * vj.x - wi.x * vj.y;
      S0[e] = c;
      const double2 qi = hq[i];
      double2 q = S1[e];
      q.x -= tau * (qi.x * vj.x + qi.y * vj.y);
      q.y -= tau * (qi.y * vj.x - qi.x * vj.y);
      S1[e] = q;
    }
    __syncthreads();
  }
  // ---- real tridiagonal form: D^H T D with D = diag(ph), ph_{i+1} = ph_i e_i / |e_i| ----
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    td[i] = S0[i * n + i].x;
    hv[i] = i + 1 < n ? S0[(i + 1) * n + i] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double2 p = make_double2(1.0, 0.0);
    for (int i = 0; i < n; ++i) {
      ph[i] = p;
      const double2 e = hv[i];
      const double ae = sqrt(e.x * e.x + e.y * e.y);
      tb[i] = ae;
      if (ae > 0.0) p = cmul(p, make_double2(e.x / ae, e.y / ae));
    }
    tb[n - 1] = 0.0;
  }
  __syncthreads();
  double* Z = reinterpret_cast<double*>(S0);       // S0 is free now: n x n real
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e - i * n;
    S1[e] = cmul(S1[e], ph[j]);
    Z[e] = i == j ? 1.0 : 0.0;
  }
  // ---- implicit QL; thread 0 carries the iteration state across sweeps ----
  int l = 0, it = 0, fail = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      int nrot = 0, state = 0;                     // 0: a sweep to apply, 1: finished
      for (;;) {
        if (l >= n) { state = 1; break; }
        int m = l;
        for (; m < n - 1; ++m) {
          const double dd = fabs(td[m]) + fabs(td[m + 1]);
          if (fabs(tb[m]) <= 2.220446049250313e-16 * dd || fabs(tb[m]) < 1e-300) break;
        }
        if (m == l) { ++l; it = 0; continue; }
        if (++it > 60) { fail = 1; state = 1; break; }
        double g = (td[l + 1] - td[l]) / (2.0 * tb[l]);
        double r = sqrt(g * g + 1.0);
        g = td[m] - td[l] + tb[l] / (g + (g >= 0.0 ? r : -r));
        double s = 1.0, c = 1.0, p = 0.0;
        bool early = false;
        for (int i = m - 1; i >= l; --i) {
          const double f = s * tb[i], bb = c * tb[i];
          const double h2 = f * f + g * g;
          if (h2 == 0.0) { td[i + 1] -= p; tb[i + 1] = 0.0; tb[m] = 0.0; early = true; break; }
          const double inv = rsqrt(h2);
          tb[i + 1] = h2 * inv;
          s = f * inv; c = g * inv;
          g = td[i + 1] - p;
          r = (td[i] - g) * s + 2.0 * c * bb;
          p = s * r;
          td[i + 1] = g + p;
          g = c * r - bb;
          ri[nrot] = i; rc[nrot] = c; rs[nrot] = s; ++nrot;
        }
        if (!early) { td[l] -= p; tb[l] = g; tb[m] = 0.0; }
        break;
      }
      s_nrot = nrot; s_state = state | (fail << 1);
    }
    __syncthreads();
    const int nrot = s_nrot, state = s_state;
    for (int row = threadIdx.x; row < n; row += blockDim.x) {
      double* z = Z + row * n;
      for (int u = 0; u < nrot; ++u) {
        const int i = ri[u];
        const double c = rc[u], s = rs[u];
        const double f = z[i + 1];
        z[i + 1] = s * z[i] + c * f;
        z[i] = c * z[i] - s * f;
      }
    }
    __syncthreads();
    if (state & 1) { fail = state >> 1; break; }
  }
  // ---- V = (Q D) Z into S1, eigenvalues onto S0's diagonal ----
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e - i * n;
    double2 v = make_double2(0.0, 0.0);
    for (int k = 0; k < n; ++k) caxpy(v, Z[k * n + j], S1[i * n + k]);
    gtmp[e] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) S1[e] = gtmp[e];
  for (int i = threadIdx.x; i < n; i += blockDim.x) S0[i * n + i] = make_double2(td[i], 0.0);
  __syncthreads();
  return fail;
}


// =============================================================================================
// Rayleigh-Ritz eigensolve for the wanted eigenpairs only: LOBPCG keeps the m smallest of the
// 3m Ritz pairs, so the tridiagonal problem is solved for those alone, by multisection with
// Sturm counts and inverse iteration, which run in parallel where the QL recurrence is serial.
// Every routine is CTA-wide for 512 threads (16 warps); block-uniform return codes.
// =============================================================================================
constexpr int kRrWarps = 16;

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// integer mixing (xorshift-multiply) for deterministic pseudo-random start vectors
__device__ __forceinline__ unsigned mix32(unsigned x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}
__device__ __forceinline__ double start_value(int i, int j) {
  return (double)(mix32((unsigned)(i * 131 + j * 7919 + 17)) >> 8) * (1.0 / 8388608.0) - 1.0;
}

struct RrShared {
  double td[kMaxSmall], tb[kMaxSmall], tau[kMaxSmall], rinv[kMaxSmall];
  double lam[kMaxSmall];
  double ds[kMaxSmall], es[kMaxSmall];       // the tridiagonal scaled for the Sturm counts
  double2 esub[kMaxSmall], ph[kMaxSmall], xcol[kMaxSmall], psm[kMaxSmall];
  double G[kMaxBlock * kMaxBlock];
  double lo, hi;
  int bad;
};

// Upper Cholesky B = U^H U in place (S, ld n), one barrier per column: step k subtracts
// conj(S_ki) S_kj / S_kk from S_ij (k < i <= j) with the unscaled pivot row; the rows are scaled
// by 1 / sqrt(S_kk) at the end. rinv = 1 / U_kk. Returns nonzero on a bad pivot. The leading k0
// columns are the identity's (S = [I V; V^H W] with V of k0 rows): their steps touch the trailing
// block alone and are taken together, four lanes an entry. A pivot must exceed least[k] (NULL: 0).
static __device__ int rr_cholesky(double2* __restrict__ S, int n, double* __restrict__ rinv, int k0,
                                  const double* __restrict__ least = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwp = blockDim.x >> 5;
  if (k0) {
    const int np = n - k0;
    for (int e0 = 0; e0 < np * np; e0 += blockDim.x / 4) {
      const int e = e0 + (threadIdx.x >> 2), i = k0 + e / np, j = k0 + e % np;
      const bool in = e < np * np && i <= j;
      double sx = 0.0, sy = 0.0;
      if (in)
        for (int k = threadIdx.x & 3; k < k0; k += 4) {
          const double2 a = S[k * n + i], b = S[k * n + j];
          sx += a.x * b.x + a.y * b.y;
          sy += a.x * b.y - a.y * b.x;
        }
      for (int o = 1; o < 4; o <<= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
      }
      if (in && (threadIdx.x & 3) == 0) { S[i * n + j].x -= sx; S[i * n + j].y -= sy; }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int k = k0; k < n; ++k) {
    const double d = S[k * n + k].x;
    if (!(d > (least ? least[k] : 0.0)) || !isfinite(d)) { __syncthreads(); return 1; }
    const double inv = 1.0 / d;
    for (int i = k + 1 + warp; i < n; i += nwp) {
      const double2 a = S[k * n + i];
      for (int j = i + lane; j < n; j += 32) {
        const double2 b = S[k * n + j];
        double2 t = S[i * n + j];
        t.x -= (a.x * b.x + a.y * b.y) * inv;
        t.y -= (a.x * b.y - a.y * b.x) * inv;
        S[i * n + j] = t;
      }
    }
    __syncthreads();
  }
  for (int k = threadIdx.x; k < n; k += blockDim.x) rinv[k] = 1.0 / sqrt(S[k * n + k].x);
  __syncthreads();
  for (int i = k0 + warp; i < n; i += nwp)
    for (int j = i + lane; j < n; j += 32) {
      const double r = rinv[i];
      if (j == i) S[i * n + j] = make_double2(1.0 / r, 0.0);
      else { S[i * n + j].x *= r; S[i * n + j].y *= r; }
    }
  __syncthreads();
  return 0;
}

// U^-1 of the upper triangle of S (pivots as reciprocals rinv) into out (ld n, zero below the diagonal):
// a warp per column, the column in registers (lane l holds rows l + 32 q), by back substitution
static __device__ void rr_upper_inverse(const double2* __restrict__ S, int n, const double* __restrict__ rinv,
                                        double2* __restrict__ out) {
  constexpr int CC = (kMaxSmall + 31) / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwp = blockDim.x >> 5;
  for (int j = warp; j < n; j += nwp) {
    double2 y[CC];
#pragma unroll
    for (int q = 0; q < CC; ++q) y[q] = make_double2(lane + 32 * q == j ? 1.0 : 0.0, 0.0);
#pragma unroll 1
    for (int k = j; k >= 0; --k) {
      double2 yk = y[0];
#pragma unroll
      for (int q = 1; q < CC; ++q) if (k >> 5 == q) yk = y[q];
      const double r = rinv[k];
      const double2 xk = make_double2(__shfl_sync(0xffffffffu, yk.x, k & 31) * r,
                                      __shfl_sync(0xffffffffu, yk.y, k & 31) * r);
#pragma unroll
      for (int q = 0; q < CC; ++q) {
        const int i = lane + 32 * q;
        if (i == k) y[q] = xk;
        const double2 u = i < k ? S[i * n + k] : make_double2(0.0, 0.0);
        y[q].x -= u.x * xk.x - u.y * xk.y;
        y[q].y -= u.x * xk.y + u.y * xk.x;
      }
    }
#pragma unroll
    for (int q = 0; q < CC; ++q) {
      const int i = lane + 32 * q;
      if (i < n) out[i * n + j] = y[q];
    }
  }
  __syncthreads();
}

// Rows of A (ld n) times U^-1 (U upper, pivots as reciprocals rinv): a warp per row (rows
// warp + 16 r), the row in registers (lane l holds columns l + 32 q), w_k = a_k / U_kk broadcast
// by a shuffle, then a_j -= w_k U_kj. Written conjugate-transposed (row i into column i) when
// `trans`, in place otherwise; every row is read before any is written.
template <int R, int CC>
static __device__ void rr_rows_solve(double2* __restrict__ A, const double2* __restrict__ U,
                                     int n, const double* __restrict__ rinv, bool trans) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2 a[R][CC];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int q = 0; q < CC; ++q) {
      const int i = warp + kRrWarps * r, j = lane + 32 * q;
      a[r][q] = (i < n && j < n) ? A[i * n + j] : make_double2(0.0, 0.0);
    }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const int kl = k & 31, kq = k >> 5;
    const double rk = rinv[k];
    double2 u[CC];
#pragma unroll
    for (int q = 0; q < CC; ++q) {
      const int j = lane + 32 * q;
      u[q] = (j > k && j < n) ? U[k * n + j] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double2 ak = a[r][0];
#pragma unroll
      for (int q = 1; q < CC; ++q) if (kq == q) ak = a[r][q];
      ak.x = __shfl_sync(0xffffffffu, ak.x, kl) * rk;
      ak.y = __shfl_sync(0xffffffffu, ak.y, kl) * rk;
#pragma unroll
      for (int q = 0; q < CC; ++q) {
        if (lane + 32 * q == k) a[r][q] = ak;
        a[r][q].x -= ak.x * u[q].x - ak.y * u[q].y;
        a[r][q].y -= ak.x * u[q].y + ak.y * u[q].x;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int q = 0; q < CC; ++q) {
      const int i = warp + kRrWarps * r, j = lane + 32 * q;
      if (i < n && j < n) {
        if (trans) A[j * n + i] = make_double2(a[r][q].x, -a[r][q].y);
        else A[i * n + j] = a[r][q];
      }
    }
  __syncthreads();
}

// rr_rows_solve with U = [I V; 0 U'] (k0 identity rows, n - k0 <= 32): rows a of A become
// [a_1 | (a_2 - a_1 V) U'^-1], in place; row i's entry j stands at A[i si + j sj], and with CONJ the
// rows are those of A^T and U is conjugated (A <- U^-H A).
template <bool CONJ>
static __device__ void rr_rows_solve_tail(double2* __restrict__ A, int si, int sj, const double2* __restrict__ U,
                                          int n, const double* __restrict__ rinv, int k0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, np = n - k0;
  for (int e = threadIdx.x; e < n * np; e += blockDim.x) {
    const int i = e / np, j = k0 + e - i * np;
    double rx = 0.0, ry = 0.0, ix = 0.0, iy = 0.0;          // four chains of FMAs
#pragma unroll 4
    for (int k = 0; k < k0; ++k) {
      const double2 a = A[i * si + k * sj];
      double2 u = U[k * n + j];
      if (CONJ) u.y = -u.y;
      rx = fma(a.x, u.x, rx); ry = fma(a.y, u.y, ry);
      ix = fma(a.x, u.y, ix); iy = fma(a.y, u.x, iy);
    }
    double2 t = A[i * si + j * sj];
    t.x -= rx - ry;
    t.y -= ix + iy;
    A[i * si + j * sj] = t;
  }
  __syncthreads();
  for (int i0 = 0; i0 < n; i0 += 3 * kRrWarps) {
    double2 a[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int i = i0 + warp + kRrWarps * r;
      a[r] = i < n && lane < np ? A[i * si + (k0 + lane) * sj] : make_double2(0.0, 0.0);
    }
    for (int k = 0; k < np; ++k) {
      const double rk = rinv[k0 + k];
      double2 u = lane > k && lane < np ? U[(k0 + k) * n + k0 + lane] : make_double2(0.0, 0.0);
      if (CONJ) u.y = -u.y;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double wx = __shfl_sync(0xffffffffu, a[r].x, k) * rk, wy = __shfl_sync(0xffffffffu, a[r].y, k) * rk;
        if (lane == k) a[r] = make_double2(wx, wy);
        a[r].x -= wx * u.x - wy * u.y;
        a[r].y -= wx * u.y + wy * u.x;
      }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int i = i0 + warp + kRrWarps * r;
      if (i < n && lane < np) A[i * si + (k0 + lane) * sj] = a[r];
    }
  }
  __syncthreads();
}

// sum over aligned groups of L lanes
template <int L>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Householder tridiagonalisation of the Hermitian part of Csm (read once), held in registers: L
// lanes a row, lane c columns c + L q, rows (thread / L) + RP r. Step k forms the reflector
// H = I - tau v v^H (v^H v = 2 / tau) from column k in every group (identical butterfly sums),
// p = tau C v row-wise, K = tau / 2 v^H p, w = p - K v and C <- C - v w^H - w v^H; two barriers
// per column; warps whose rows are reduced already, or past n, only wait. A step is a chain of
// three sums, a reciprocal and a root: eight lanes a row leave three shuffles a sum and a matrix of
// 36 fills nine warps without padding columns (a warp a row: five shuffles, twice the FMAs). Above 64
// the rows of eight lanes would not fit the registers: sixteen.
// Reflector k (v_j, j > k) is stored in row n - 1 - k of Rf's strict lower triangle
// (v_j at column j - k - 1), tau_k in sh.tau. On return sh.td / sh.tb hold the real
// tridiagonal T = D^H (Q^H C Q) D, sh.ph the phases D (the off-diagonal made real and >= 0).
template <int L, int R, int Q>
static __device__ void rr_tridiag(const double2* __restrict__ Csm, int n,
                                  double2* __restrict__ Rf, RrShared& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int RW = 32 / L, RP = RW * kRrWarps;   // rows of a warp, and of the block, a round
  const int c = threadIdx.x % L, row0 = threadIdx.x / L;
  double2 a[R][Q];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = row0 + RP * r, j = c + L * q;
      if (i < n && j < n) {
        const double2 u = Csm[i * n + j], v = Csm[j * n + i];
        a[r][q] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
      } else {
        a[r][q] = make_double2(0.0, 0.0);
      }
    }
  if (row0 == 0)                                   // column 0 is row 0 conjugated
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = c + L * q;
      if (j < n) sh.xcol[j] = j > 0 ? make_double2(a[0][q].x, -a[0][q].y) : make_double2(0.0, 0.0);
    }
  __syncthreads();
  int wlast = -1;                                  // the warp's last row of the matrix, about
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (RW * warp + RP * r < n) wlast = RW * warp + RP * r + RW - 1;
  for (int k = 0; k + 2 < n; ++k) {
    const bool live = wlast >= k;                  // uniform over the warp
    const int j0 = k + 1;
    double2 vs[Q], vr[R], pr[R];
    double tau = 0.0;
    if (live) {
      double n0 = 0.0, n1 = 0.0;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = c + L * q;
        vs[q] = (j > k && j < n) ? sh.xcol[j] : make_double2(0.0, 0.0);
        n0 = fma(vs[q].x, vs[q].x, n0);
        n1 = fma(vs[q].y, vs[q].y, n1);
      }
      const double nx2 = group_sum<L>(n0 + n1);
      const double2 x0 = sh.xcol[j0];
      // alpha = -phase(x0) |x|, v = x - alpha e_1
      const double a2 = x0.x * x0.x + x0.y * x0.y;
      const double ia = rsqrt(a2), ax0 = a2 > 0.0 ? a2 * ia : 0.0;
      const double nx = nx2 > 0.0 ? nx2 * rsqrt(nx2) : 0.0;
      const double2 phs = a2 > 0.0 ? make_double2(x0.x * ia, x0.y * ia) : make_double2(1.0, 0.0);
      // below the smallest normal double the column is left as it is (1 / den would overflow)
      const double den = nx * (nx + ax0);
      tau = den >= 2.2250738585072014e-308 ? 1.0 / den : 0.0;
      const double2 v0 = make_double2(x0.x + phs.x * nx, x0.y + phs.y * nx);
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (c + L * q == j0) vs[q] = v0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = row0 + RP * r;
        vr[r] = (i > j0 && i < n) ? sh.xcol[i] : (i == j0 ? v0 : make_double2(0.0, 0.0));
        double s0 = 0.0, s1 = 0.0, t0 = 0.0, t1 = 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          s0 = fma(a[r][q].x, vs[q].x, s0); s1 = fma(a[r][q].y, vs[q].y, s1);
          t0 = fma(a[r][q].x, vs[q].y, t0); t1 = fma(a[r][q].y, vs[q].x, t1);
        }
        pr[r] = make_double2(s0 - s1, t0 + t1);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        pr[r].x = tau * group_sum<L>(pr[r].x);
        pr[r].y = tau * group_sum<L>(pr[r].y);
        const int i = row0 + RP * r;
        if (i < k) pr[r] = make_double2(0.0, 0.0);     // reduced already
        if (c == 0 && i < n) sh.psm[i] = pr[r];
      }
    }
    __syncthreads();
    if (live) {
      // the reflector, kept by the last warp of the matrix (it stays live)
      if ((n - 1) % RP / RW == warp && lane < L) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int j = c + L * q;
          if (j > k && j < n) Rf[(n - 1 - k) * n + (j - k - 1)] = vs[q];
        }
        if (lane == 0) sh.tau[k] = tau;
      }
      double2 pc[Q];
      double s0 = 0.0, s1 = 0.0;                   // Re v^H p (v^H C v is real)
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = c + L * q;
        pc[q] = (j >= k && j < n) ? sh.psm[j] : make_double2(0.0, 0.0);
        s0 = fma(vs[q].x, pc[q].x, s0);
        s1 = fma(vs[q].y, pc[q].y, s1);
      }
      const double K = 0.5 * tau * group_sum<L>(s0 + s1);
#pragma unroll
      for (int q = 0; q < Q; ++q) pc[q] = make_double2(pc[q].x - K * vs[q].x, pc[q].y - K * vs[q].y);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double2 wi = make_double2(pr[r].x - K * vr[r].x, pr[r].y - K * vr[r].y);
        const double2 vi = vr[r];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const double2 vj = vs[q], wj = pc[q];
          a[r][q].x -= vi.x * wj.x + vi.y * wj.y + wi.x * vj.x + wi.y * vj.y;
          a[r][q].y -= vi.y * wj.x - vi.x * wj.y + wi.y * vj.x - wi.x * vj.y;
        }
        // row k is final (diagonal and sub-diagonal); row k + 1, conjugated, is the next column
        const int i = row0 + RP * r;
        if (i == k || i == k + 1)
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const int j = c + L * q;
            const double2 v = make_double2(a[r][q].x, -a[r][q].y);
            if (i == k) {
              if (j == k) sh.td[k] = v.x;
              if (j == k + 1) sh.esub[k] = v;
            } else if (j < n) {
              sh.xcol[j] = j > k + 1 ? v : make_double2(0.0, 0.0);
            }
          }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {                    // the last two rows
    const int i = row0 + RP * r;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = c + L * q;
      if (n >= 2 && i == n - 2) {
        if (j == n - 2) sh.td[n - 2] = a[r][q].x;
        if (j == n - 1) sh.esub[n - 2] = make_double2(a[r][q].x, -a[r][q].y);
      }
      if (i == n - 1 && j == n - 1) sh.td[n - 1] = a[r][q].x;
    }
  }
  __syncthreads();
  // the off-diagonal's moduli, and its phases' running products (a warp scan)
  if (warp == 0) {
    double2 carry = make_double2(1.0, 0.0);
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      double2 u = make_double2(1.0, 0.0);
      if (i < n) {
        double ae = 0.0;
        if (i + 1 < n) {
          const double2 e = sh.esub[i];
          ae = sqrt(e.x * e.x + e.y * e.y);
          if (ae > 0.0) u = make_double2(e.x / ae, e.y / ae);
        }
        sh.tb[i] = ae;
      }
      for (int o = 1; o < 32; o <<= 1) {
        const double2 t = make_double2(__shfl_up_sync(0xffffffffu, u.x, o), __shfl_up_sync(0xffffffffu, u.y, o));
        if (lane >= o) u = cmul(t, u);
      }
      u = cmul(carry, u);
      if (i0 == 0 && lane == 0) sh.ph[0] = make_double2(1.0, 0.0);
      if (i + 1 < n) sh.ph[i + 1] = u;
      carry = make_double2(__shfl_sync(0xffffffffu, u.x, 31), __shfl_sync(0xffffffffu, u.y, 31));
    }
  }
  __syncthreads();
}

// Eigenvalues of the tridiagonal below x: sign changes of the leading-minor determinants
// p_{i+1} = (d_i - x) p_i - e_{i-1}^2 p_{i-1} (the Sturm sequence; an FMA per step where the
// ratio form needs a division). The caller scales T to at most 2 and keeps the e^2 above 2^-120, so
// that a zero determinant is followed by one of the other sign (it counts once whichever sign it
// is given) and four steps cannot leave the exponent range: the pair is rescaled by a power of two
// after every fourth, and the chain is otherwise an FMA a step (signs are counted in integers).
static __device__ __forceinline__ int rr_sturm(const double* __restrict__ ds,
                                               const double* __restrict__ es, int n, double x) {
  double pm = 1.0, p = ds[0] - x;
  int c = (unsigned)__double2hiint(p) >> 31;
#pragma unroll 4
  for (int i = 1; i < n; ++i) {
    const double pn = fma(ds[i] - x, p, -es[i - 1] * pm);
    c += (unsigned)(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
    pm = p;
    p = pn;
    if ((i & 3) == 0) {
      const int e = max(__double2hiint(p) & 0x7ff00000, __double2hiint(pm) & 0x7ff00000);
      const double f = __hiloint2double(0x7fe00000 - e, 0);
      p *= f;
      pm *= f;
    }
  }
  return c;
}

// The nwant smallest eigenpairs of A x = lambda B x (B = nullptr: the identity), A and B n x n
// Hermitian (global, ld n): w[0..nwant) ascending and Vout[:, 0..nwant) (ld n; the other columns
// are zeroed). Steps: B = U^H U (rr_cholesky); C^H = (U^-H A U^-1)^H by two row solves
// (rr_rows_solve); Householder to the real tridiagonal T (rr_tridiag); eigenvalues by
// multisection (G lanes per eigenvalue, Sturm counts, G + 1 sub-intervals per round, down to
// 2 eps ||T||); eigenvectors by two inverse-iteration steps (a thread per eigenvalue, LU of
// T - lambda I with partial pivoting, pseudo-random start), orthonormalised by two Cholesky-QR
// passes; V = U^-1 Q D Z with the reflectors applied in reverse order. Returns 0, 1 (B not
// positive definite), 2 (non-finite T) or 3 (inverse-iteration vectors not independent: the
// caller then solves the full problem). S0 / S1: n x n shared matrices. The leading k0 columns of
// B are the identity's. Rows and columns a thread holds: R x CC in rr_rows_solve, RT x QC (L lanes a
// row) in rr_tridiag. S0 is the kernel's dynamic shared memory.
extern __shared__ double2 rr_dynamic[];
template <int R, int CC, int L, int RT, int QC>
static __device__ __forceinline__ int rr_wanted(const double2* __restrict__ A, const double2* __restrict__ B,
                                                int k0, int n, int nwant, double* __restrict__ w,
                                                double2* __restrict__ Vout) {
  __shared__ RrShared sh;
  double2 *S0 = rr_dynamic, *S1 = rr_dynamic + n * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwp = blockDim.x >> 5;
  const double eps = 1.1102230246251565e-16;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) S1[e] = A[e];
  if (!B) k0 = n;
  if (k0 < n) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) S0[e] = B[e];
    __syncthreads();
    if (n - k0 > 32) k0 = 0;                               // more trailing columns than lanes
    if (rr_cholesky(S0, n, sh.rinv, k0)) return 1;
    if (k0) {
      rr_rows_solve_tail<false>(S1, n, 1, S0, n, sh.rinv, k0);   // W = A U^-1
      rr_rows_solve_tail<true>(S1, 1, n, S0, n, sh.rinv, k0);    // C = U^-H W
    } else {
      rr_rows_solve<R, CC>(S1, S0, n, sh.rinv, true);      // W^H with W = A U^-1
      rr_rows_solve<R, CC>(S1, S0, n, sh.rinv, false);     // W^H U^-1 = C^H
    }
  } else {
    __syncthreads();
  }
  rr_tridiag<L, RT, QC>(S1, n, S0, sh);    // reflectors below S0's diagonal, U above it
  // ---- Gershgorin bounds ----
  if (warp == 0) {
    double lo = INFINITY, hi = -INFINITY;
    for (int i = lane; i < n; i += 32) {
      const double r = (i > 0 ? sh.tb[i - 1] : 0.0) + (i + 1 < n ? sh.tb[i] : 0.0);
      lo = fmin(lo, sh.td[i] - r);
      hi = fmax(hi, sh.td[i] + r);
    }
    lo = warp_min(lo);
    hi = warp_max(hi);
    if (lane == 0) {
      const double tn = fmax(fabs(lo), fabs(hi));
      sh.lo = lo - 4.0 * eps * tn * n - 1e-300;
      sh.hi = hi + 4.0 * eps * tn * n + 1e-300;
      sh.bad = !(isfinite(lo) && isfinite(hi));
    }
  }
  __syncthreads();
  if (sh.bad) return 2;
  const double tn = fmax(fabs(sh.lo), fabs(sh.hi));
  // T scaled by a power of two to at most 2 (an exact scaling) for the Sturm counts
  const double scale = __hiloint2double(max(0x00100000, 0x7fe00000 - (__double2hiint(tn) & 0x7ff00000)), 0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double e = sh.tb[i] * scale;
    sh.ds[i] = sh.td[i] * scale;
    sh.es[i] = fmax(e * e, 0x1p-120);
  }
  __syncthreads();
  // ---- multisection: lanes t of group g evaluate a + (b - a)(t + 1) / (G + 1) ----
  int G = 32;
  while (G > 1 && nwant * G > (int)blockDim.x) G >>= 1;
  {
    const int g = threadIdx.x / G, t = threadIdx.x % G;
    const int base = lane / G * G;
    const unsigned gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u) << base);
    const bool act = g < nwant;
    const double part = (double)(t + 1) / (double)(G + 1);
    double a = sh.lo, b = sh.hi;
    for (int round = 0; round < 64; ++round) {
      const bool conv = !act || (b - a) <= fmax(2.0 * eps * tn, 4.0 * eps * fmax(fabs(a), fabs(b)));
      if (__all_sync(0xffffffffu, conv)) break;
      const double x = a + (b - a) * part;
      const int cnt = rr_sturm(sh.ds, sh.es, n, x * scale);
      const unsigned below = __ballot_sync(0xffffffffu, cnt <= g) & gmask;   // x below lambda_g
      const int hiT = below ? 31 - __clz(below) : -1;
      const unsigned above = ~below & gmask;
      const int loT = above ? __ffs(above) - 1 : -1;
      const double xh = __shfl_sync(0xffffffffu, x, max(hiT, 0)), xl = __shfl_sync(0xffffffffu, x, max(loT, 0));
      const double na = hiT >= 0 ? xh : a;
      const double nb = loT >= 0 ? xl : b;
      a = conv ? a : na;
      b = conv ? b : nb;
    }
    if (act && t == 0) sh.lam[g] = 0.5 * (a + b);
  }
  __syncthreads();
  // ---- inverse iteration: arrays interleaved [i][j] in S1 (free after the tridiagonalisation) ----
  const int zs = (n * nwant + 1) & ~1;
  double* Z = reinterpret_cast<double*>(S1);
  double* ur = Z + zs;                  // 1 / pivot of U's row i
  double* u1 = ur + n * nwant;          // U_{i,i+1}
  double* ll = u1 + n * nwant;          // L's multiplier
  const double tiny = eps * tn + 1e-300;
  if ((int)threadIdx.x < nwant) {
    const int j = threadIdx.x;
    const double mu = sh.lam[j];
    // T - mu I factored row by row, rows exchanged when the sub-diagonal is larger (a bit each in sw:
    // U_{i,i+2} is then the next off-diagonal), and the right-hand side eliminated alongside
    unsigned sw[(kMaxSmall + 31) / 32] = {};
    {
      double a = sh.td[0] - mu, bcur = n > 1 ? sh.tb[0] : 0.0;
      double y = start_value(0, j);
#pragma unroll 1
      for (int i = 0; i + 1 < n; ++i) {
        const double cc = sh.tb[i];
        const double an = sh.td[i + 1] - mu;
        const double bn = i + 2 < n ? sh.tb[i + 1] : 0.0;
        const double yn = start_value(i + 1, j);
        const bool s = fabs(a) < fabs(cc);
        const double ap = fabs(a) < tiny ? (a < 0.0 ? -tiny : tiny) : a;
        const double ri = 1.0 / (s ? cc : ap);
        const double l = (s ? a : cc) * ri;
        ur[i * nwant + j] = ri;
        u1[i * nwant + j] = s ? an : bcur;
        ll[i * nwant + j] = l;
#pragma unroll
        for (int q = 0; q < (kMaxSmall + 31) / 32; ++q)
          if (q == i >> 5) sw[q] |= (unsigned)s << (i & 31);
        Z[i * nwant + j] = s ? yn : y;
        const double na = s ? bcur - l * an : an - l * bcur;
        const double ny = s ? y - l * yn : yn - l * y;
        bcur = s ? -l * bn : bn;
        a = na;
        y = ny;
      }
      const double ap = fabs(a) < tiny ? (a < 0.0 ? -tiny : tiny) : a;
      ur[(n - 1) * nwant + j] = 1.0 / ap;
      u1[(n - 1) * nwant + j] = 0.0;
      Z[(n - 1) * nwant + j] = y;
    }
    auto exchanged = [&](int i) {
      unsigned w = sw[0];
#pragma unroll
      for (int q = 1; q < (kMaxSmall + 31) / 32; ++q) if (q == i >> 5) w = sw[q];
      return (w >> (i & 31) & 1u) != 0;
    };
    for (int step = 0; step < 2; ++step) {
      double x1 = 0.0, x2 = 0.0, mx = 0.0;          // back substitution
#pragma unroll 2
      for (int i = n - 1; i >= 0; --i) {
        const double u2 = i + 2 < n && exchanged(i) ? sh.tb[i + 1] : 0.0;
        const double x = (Z[i * nwant + j] - u2 * x2 - u1[i * nwant + j] * x1) * ur[i * nwant + j];
        Z[i * nwant + j] = x;
        x2 = x1;
        x1 = x;
        mx = fmax(mx, fabs(x));
      }
      const double sc = mx > 0.0 && isfinite(mx) ? 1.0 / mx : 0.0;
      if (step == 1) {
        for (int i = 0; i < n; ++i) Z[i * nwant + j] *= sc;
      } else {                                      // the second right-hand side, eliminated
        double y = Z[j] * sc;
#pragma unroll 2
        for (int i = 0; i + 1 < n; ++i) {
          const double l = ll[i * nwant + j], yn = Z[(i + 1) * nwant + j] * sc;
          const bool s = exchanged(i);
          Z[i * nwant + j] = s ? yn : y;
          y = s ? y - l * yn : yn - l * y;
        }
        Z[(n - 1) * nwant + j] = y;
      }
    }
  }
  __syncthreads();
  // ---- Cholesky-QR, twice: G = Z^T Z (a thread per entry), G = R^T R with unscaled rows (row k of R is
  //      G_k / sqrt(G_kk)), Z <- Z R^-1 (eight lanes a row). The loops stay rolled: unrolled over the
  //      widest block they ran as fast when their code was cached, and 22 us longer after the tall
  //      kernels of an iteration had pushed it out of L2 ----
  double* rs = sh.es;
  for (int pass = 0; pass < 2; ++pass) {
    for (int e = threadIdx.x; e < nwant * nwant; e += blockDim.x) {
      const int a = e / nwant, b = e - a * nwant;
      if (b < a) continue;
      double d0 = 0.0, d1 = 0.0, d2 = 0.0;
#pragma unroll 1
      for (int i = 0; i < n; i += 3) {
        d0 = fma(Z[i * nwant + a], Z[i * nwant + b], d0);
        if (i + 1 < n) d1 = fma(Z[(i + 1) * nwant + a], Z[(i + 1) * nwant + b], d1);
        if (i + 2 < n) d2 = fma(Z[(i + 2) * nwant + a], Z[(i + 2) * nwant + b], d2);
      }
      sh.G[e] = d0 + d1 + d2;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < nwant; ++k) {
      const double d0 = sh.G[k * nwant + k];
      // the vectors have max-abs 1 (first pass) or unit norm (second): a pivot this small means
      // a vector (nearly) in the span of the previous ones
      if (!(d0 > 1e-10) || !isfinite(d0)) return 3;
      const double inv = 1.0 / d0;
      for (int e = threadIdx.x; e < nwant * nwant; e += blockDim.x) {
        const int a = e / nwant, b = e - a * nwant;
        if (a > k && b >= a) sh.G[e] -= sh.G[k * nwant + a] * sh.G[k * nwant + b] * inv;
      }
      __syncthreads();
    }
    if ((int)threadIdx.x < nwant) rs[threadIdx.x] = rsqrt(sh.G[threadIdx.x * (nwant + 1)]);
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += 64) {
      const int i = i0 + (threadIdx.x >> 3), c = threadIdx.x & 7;
      constexpr int QZ = kMaxBlock / 8;
      double z[QZ];
#pragma unroll
      for (int q = 0; q < QZ; ++q) z[q] = i < n && c + 8 * q < nwant ? Z[i * nwant + c + 8 * q] : 0.0;
#pragma unroll 1
      for (int k = 0; k < nwant; ++k) {
        double zk = z[0];
#pragma unroll
        for (int q = 1; q < QZ; ++q) if (q == k >> 3) zk = z[q];
        zk = __shfl_sync(0xffffffffu, zk, (lane & 24) | (k & 7)) * rs[k];
        const double f = zk * rs[k];
#pragma unroll
        for (int q = 0; q < QZ; ++q) {
          const int j = c + 8 * q;
          if (j == k) z[q] = zk;
          else if (j > k && j < nwant) z[q] -= f * sh.G[k * nwant + j];
        }
      }
#pragma unroll
      for (int q = 0; q < QZ; ++q) if (i < n && c + 8 * q < nwant) Z[i * nwant + c + 8 * q] = z[q];
    }
    __syncthreads();
  }
  // ---- V = U^-1 Q D Z: a warp per column, the column in registers (lane l holds rows l + 32 q):
  //      phases, reflectors n-3 .. 0, back substitution ----
  for (int j = warp; j < nwant; j += nwp) {
    double2 y[CC];
#pragma unroll
    for (int q = 0; q < CC; ++q) {
      const int i = lane + 32 * q;
      const double z = i < n ? Z[i * nwant + j] : 0.0;
      y[q] = i < n ? make_double2(sh.ph[i].x * z, sh.ph[i].y * z) : make_double2(0.0, 0.0);
    }
#pragma unroll 1
    for (int k = n - 3; k >= 0; --k) {
      const double tk = sh.tau[k];
      const double2* vrow = S0 + (n - 1 - k) * n - (k + 1);   // v_i at vrow[i], i > k
      double2 v[CC];
      double sx = 0.0, sy = 0.0;                                // v^H y
#pragma unroll
      for (int q = 0; q < CC; ++q) {
        const int i = lane + 32 * q;
        v[q] = (i > k && i < n) ? vrow[i] : make_double2(0.0, 0.0);
        sx += v[q].x * y[q].x + v[q].y * y[q].y;
        sy += v[q].x * y[q].y - v[q].y * y[q].x;
      }
      sx = tk * warp_sum(sx);
      sy = tk * warp_sum(sy);
#pragma unroll
      for (int q = 0; q < CC; ++q) {
        y[q].x -= v[q].x * sx - v[q].y * sy;
        y[q].y -= v[q].x * sy + v[q].y * sx;
      }
    }
    if (k0 < n) {
#pragma unroll 1
      for (int k = n - 1; k >= k0; --k) {
        const int kl = k & 31, kq = k >> 5;
        double2 yk = y[0];
#pragma unroll
        for (int q = 1; q < CC; ++q) if (kq == q) yk = y[q];
        const double r = sh.rinv[k];
        const double2 xk = make_double2(__shfl_sync(0xffffffffu, yk.x, kl) * r,
                                        __shfl_sync(0xffffffffu, yk.y, kl) * r);
#pragma unroll
        for (int q = 0; q < CC; ++q) {
          const int i = lane + 32 * q;
          if (i == k) y[q] = xk;
          const double2 u = i < k ? S0[i * n + k] : make_double2(0.0, 0.0);
          y[q].x -= u.x * xk.x - u.y * xk.y;
          y[q].y -= u.x * xk.y + u.y * xk.x;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < CC; ++q) {
      const int i = lane + 32 * q;
      if (i < n) Vout[i * n + j] = y[q];
    }
  }
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e - i * n;
    if (j >= nwant) Vout[e] = make_double2(0.0, 0.0);
  }
  for (int j = threadIdx.x; j < nwant; j += blockDim.x) w[j] = sh.lam[j];
  __syncthreads();
  return 0;
}

// Sizes of the eigensolve, each a kernel of its own: with all of them in one body the small ones' loops
// spilled registers (36 rows: 355k clocks for 230k), and as functions they still did.
__host__ __device__ __forceinline__ int rr_class(int n) { return n <= 40 ? 0 : (n <= 64 ? 1 : 2); }

// doubles that rr_wanted's inverse iteration takes in S1
__host__ __device__ __forceinline__ int rr_s1_doubles(int n, int nwant) {
  return ((n * nwant + 1) & ~1) + 3 * n * nwant;
}

// rr_wanted when it applies (its arrays fit the s1 doubles of S1, 512 threads); returns -1 when it does
// not
template <int CLASS>
static __device__ __forceinline__ int block_eigh_wanted(const double2* __restrict__ A,
                                                        const double2* __restrict__ B, int k0, int n, int nwant,
                                                        int s1, double* __restrict__ w,
                                                        double2* __restrict__ Vout) {
  if (nwant < 1 || nwant > n || nwant > kMaxBlock || (int)blockDim.x != 32 * kRrWarps ||
      rr_s1_doubles(n, nwant) > s1)
    return -1;
  if (CLASS == 0) return rr_wanted<3, 2, 8, 1, 5>(A, B, k0, n, nwant, w, Vout);
  if (CLASS == 1) return rr_wanted<4, 2, 8, 1, 8>(A, B, k0, n, nwant, w, Vout);
  return rr_wanted<5, 3, 16, 3, 5>(A, B, k0, n, nwant, w, Vout);
}

// The full problem by the QL iteration (block_eigh's arguments)
static __device__ __noinline__ int block_eigh_full(const double2* __restrict__ A,
                                                   const double2* __restrict__ B, int n,
                                                   double* __restrict__ w, double2* __restrict__ Vout,
                                                   double2* __restrict__ scratch) {
  double2 *S0 = rr_dynamic, *S1 = rr_dynamic + n * n;
  double2* Ug = scratch;           // Uinv (global)
  double2* Tg = scratch + n * n;   // A Uinv (global)
  __shared__ int rank[kMaxSmall];
  __shared__ double wd[kMaxSmall];
  if (B) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) S0[e] = B[e];
    __syncthreads();
    __shared__ double rinv[kMaxSmall];
    if (rr_cholesky(S0, n, rinv, 0)) return 1;
    rr_upper_inverse(S0, n, rinv, S1);          // Uinv in shared memory
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) Ug[e] = S1[e];
    // T = A Uinv  (Uinv upper: k <= j), A staged into S0
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) S0[e] = A[e];
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e % n;
      double2 s = make_double2(0.0, 0.0);
      for (int k = 0; k <= j; ++k) cfma(s, S0[i * n + k], S1[k * n + j]);
      Tg[e] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) S0[e] = Tg[e];
    __syncthreads();
    // C = Uinv^H T (k <= i) into Tg, then Hermitised into S0
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e % n;
      double2 s = make_double2(0.0, 0.0);
      for (int k = 0; k <= i; ++k) cfmac(s, S1[k * n + i], S0[k * n + j]);
      Tg[e] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) S1[e] = Tg[e];
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e % n;
      const double2 a = S1[i * n + j], b = S1[j * n + i];
      S0[e] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    }
    __syncthreads();
  } else {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e % n;
      const double2 a = A[i * n + j], b = A[j * n + i];
      S0[e] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < n * n; e += blockDim.x)
    S1[e] = make_double2((e / n == e % n) ? 1.0 : 0.0, 0.0);
  __syncthreads();
  if (block_tql(S0, S1, n, Tg)) return 2;
  for (int i = threadIdx.x; i < n; i += blockDim.x) wd[i] = S0[i * n + i].x;
  __syncthreads();
  int bad = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    int r = 0;
    const double wi = wd[i];
    if (!isfinite(wi)) bad = 1;
    for (int j = 0; j < n; ++j) {
      const double wj = wd[j];
      r += (wj < wi) || (wj == wi && j < i);
    }
    rank[i] = r;
    w[r] = wi;
  }
  bad = __syncthreads_or(bad);
  // Vout[:, rank[j]] = (Uinv) W[:, j]
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e % n;
    double2 s;
    if (B) {
      s = make_double2(0.0, 0.0);
      for (int k = i; k < n; ++k) cfma(s, Ug[i * n + k], S1[k * n + j]);
    } else {
      s = S1[i * n + j];
    }
    Vout[i * n + rank[j]] = s;
  }
  __syncthreads();
  return bad ? 2 : 0;
}

// w ascending, V columns permuted accordingly; generalized problem through B = U^H U.
// Returns 0 (ok), 1 (B not positive definite) or 2 (non-finite eigenvalue); block-uniform.
// The kernel's dynamic shared memory: two n x n matrices, the second of s1 >= 2 n^2 doubles; scratch:
// 2 n^2 global elements. Only the nwant smallest pairs are required (w[0..nwant), V's first nwant
// columns): block_eigh_wanted computes them, block_eigh_full is taken when it does not apply or its
// vectors collapse. The leading k0 columns of B are known to be the identity's. CLASS: rr_class of
// n or more.
template <int CLASS>
static __device__ int block_eigh(const double2* __restrict__ A, const double2* __restrict__ B,
                                 int n, double* __restrict__ w, double2* __restrict__ Vout,
                                 double2* __restrict__ scratch, int nwant, int s1, int k0 = 0) {
  const int r = block_eigh_wanted<CLASS>(A, B, k0, n, nwant, s1, w, Vout);
  if (r == 0 || r == 1) return r;                  // else: the full problem
  return block_eigh_full(A, B, n, w, Vout, scratch);
}



// ---------------------------------------------------------------------------------------------
// Block updates of complex128 blocks on the FP64 MMA (mma.sync.m8n8k4.f64): Y' = A' C'' with A'
// (rows x 2P) the real view of [A_0 | A_1 | A_2] and C'' (2P x 2q) the real representation of the
// stacked complex coefficients: C''_{2i,2j} = Re C_ij, C''_{2i,2j+1} = Im C_ij, C''_{2i+1,2j} =
// -Im C_ij, C''_{2i+1,2j+1} = Re C_ij. A warp owns MT 8-row M tiles at a time. The k order is permuted
// over pairs of k steps: a pair covers complex columns c0 .. c0 + 3 of one block, MMA k = t of its
// first step is Re A[.][c0 + t] and of its second step Im A[.][c0 + t] (g = lane / 4, t = lane % 4),
// so a lane's A values of the pair are one 16-byte load, A[row g][c0 + t]. Those loads stream
// through a ring of pairs in shared memory private to the warp: each lane cp.async-copies exactly
// the 16 bytes it later reads, so its own cp.async.wait_group orders them and no barrier is needed.
// C'' is stored in the pair's k order as one 16-byte word per (pair, 8-column N tile, lane):
// {C''[2 (c0 + t)][n g], C''[2 (c0 + t) + 1][n g]}. A row is read (by the four lanes of its quad)
// before any of its outputs is written and no other warp touches it, so outputs may alias inputs.
// ---------------------------------------------------------------------------------------------
constexpr int kUpdThreads = 256;
constexpr int kUpdWarps = kUpdThreads / 32;
constexpr int kUpdChunk = 16 * kUpdWarps;           // row granularity of a CTA's span: two tiles a warp
// ... of an update alone: complex128 outputs of more than 12 columns go by one tile a warp (80,000 rows of
// 60 columns to 20: spans of 256 rows make 313 CTAs for the 296 that run at once, 72 us; of 192 rows 63)
template <typename T> __host__ __device__ __forceinline__ int update_chunk(int q) {
  return sizeof(T) == 8 && q > 12 ? kUpdChunk / 2 : kUpdChunk;
}
constexpr int kDmRing = 16;                         // 16-byte words in flight per lane
constexpr size_t kDmRingBytes = (size_t)kUpdWarps * kDmRing * 32 * sizeof(double2);

// k-step pairs of a list of at most three blocks with P columns in all (ceil(cols / 4) each)
__host__ __device__ __forceinline__ int dmma_pairs_bound(int P) { return (P + 3) / 4 + 2; }
// the warps' load rings, then the packed coefficients
__host__ __device__ __forceinline__ size_t update_smem_bytes(int P, int q) {
  return kDmRingBytes + (size_t)dmma_pairs_bound(P) * ((q + 3) / 4) * 32 * sizeof(double2);
}

// One k-step pair of an update's A list: up to four columns of a block. 16 bytes, read as one word: with the
// four places as integers, indexed by the lane, the step went through local memory and a complex64 update of
// 650,000 rows of 51 columns took 175 us, 157 us so.
template <typename T>
struct KStep {
  const cplx<T>* p;
  int ld;
  unsigned col;     // a byte a column: its place in a row of p, 255 where there is none
  // element of column t (0..3) of row `row`, or NULL
  __device__ __forceinline__ const cplx<T>* at(int t, long long row, long long end) const {
    const unsigned c = col >> (8 * t) & 255u;
    return c != 255u && row < end ? p + row * ld + c : nullptr;
  }
};
static_assert(sizeof(KStep<float>) == 16 && kMaxBlock < 255, "a word; places fit a byte");

// Appends the k steps of block p (ld, cols columns; gather: column c at gather[c]); one thread.
template <typename T>
static __device__ __forceinline__ int add_ksteps(KStep<T>* k, int s, const cplx<T>* p, long long ld,
                                                 int cols, const int* gather) {
  for (int c0 = 0; c0 < cols; c0 += 4, ++s) {
    k[s].p = gather ? p : p + c0; k[s].ld = (int)ld; k[s].col = 0;
    for (int t = 0; t < 4; ++t)
      k[s].col |= (unsigned)(c0 + t < cols ? (gather ? gather[c0 + t] : t) : 255) << (8 * t);
  }
  return s;
}

// Packs the cols x q row-major complex coefficients C of one block (k steps s0 .. of the list) for
// the FP64 MMA; every thread of the CTA
static __device__ __forceinline__ void pack_dmma(double2* __restrict__ sB, int s0, const double2* __restrict__ C,
                                                 int cols, int q, double sg) {
  const int NT = (q + 3) / 4, KS = (cols + 3) / 4;
  for (int e = threadIdx.x; e < KS * NT * 32; e += blockDim.x) {
    const int s = e / (NT * 32), r = e - s * NT * 32;
    const int j = r >> 5, ln = r & 31, gg = ln >> 2, tt = ln & 3;
    const int i = 4 * s + tt, jj = j * 4 + (gg >> 1);
    double2 w = make_double2(0.0, 0.0);
    if (i < cols && jj < q) {
      const double2 c = C[(size_t)i * q + jj];
      const double re = sg * c.x, im = sg * c.y;
      w = (gg & 1) ? make_double2(im, re)          // C''[2i][2jj+1], C''[2i+1][2jj+1]
                   : make_double2(re, -im);        // C''[2i][2jj],   C''[2i+1][2jj]
    }
    sB[(size_t)s0 * NT * 32 + e] = w;
  }
}

// A warp's stream of A fragments: items are (tile group of MT 8-row tiles, k step), kDmRing / MT in
// flight. take() gives item `it`'s fragments, done() refills its slot.
template <int MT>
struct DmStream {
  static constexpr int DEPTH = kDmRing / MT;
  const KStep<double>* k;       // in shared memory
  double2* ring;
  int KS, nitems, nw, g, t, l_group, l_s;
  long long r0, r1;
  __device__ __forceinline__ DmStream(const KStep<double>* k_, double2* ring_, int KS_, long long r0_,
                                      long long r1_)
      : k(k_), KS(KS_), r0(r0_), r1(r1_) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    g = lane >> 2; t = lane & 3; nw = blockDim.x >> 5;
    const int groups = (int)((r1 - r0 + 8 * MT - 1) / (8 * MT));
    nitems = (groups > warp ? (groups - warp + nw - 1) / nw : 0) * KS;
    ring = ring_ + (size_t)warp * kDmRing * 32 + lane;
    l_group = warp; l_s = 0;
    for (int d = 0; d < DEPTH; ++d) fetch(d, d < nitems);
  }
  __device__ __forceinline__ void fetch(int slot, bool any) {
    if (any) {
      const KStep<double> ks = k[l_s];
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const long long ra = r0 + (long long)l_group * (8 * MT) + 8 * i + g;
        double2* dst = ring + (slot * MT + i) * 32;
        if (const double2* src = ks.at(t, ra, r1)) {
          const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(sa), "l"(src) : "memory");
        } else {
          *dst = make_double2(0.0, 0.0);
        }
      }
      if (++l_s == KS) { l_s = 0; l_group += nw; }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  __device__ __forceinline__ void take(int it, double2 (&a)[MT]) const {
    // item it's group is complete once at most DEPTH - 1 younger groups are pending
    asm volatile("cp.async.wait_group %0;\n" :: "n"(DEPTH - 1) : "memory");
#pragma unroll
    for (int i = 0; i < MT; ++i) a[i] = ring[((it & (DEPTH - 1)) * MT + i) * 32];
  }
  // after the MMAs on item it: their reads of its slot are done
  __device__ __forceinline__ void done(int it) { fetch(it & (DEPTH - 1), it + DEPTH < nitems); }
};

template <int NT, int MT>
static __device__ __forceinline__ void dm_step(const double2 (&a)[MT], const double2* __restrict__ bp,
                                               double (&acc)[MT][NT][2]) {
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const double2 b = bp[j * 32];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      dmma(acc[i][j][0], acc[i][j][1], a[i].x, b.x);
      dmma(acc[i][j][0], acc[i][j][1], a[i].y, b.y);
    }
  }
}

template <int NT, bool ACC>
static __device__ __forceinline__ void update_dmma_core(const KStep<double>* __restrict__ sK,
                                                        const double2* __restrict__ sB,
                                                        double2* __restrict__ ring, int KS, int q,
                                                        long long r0, long long r1, double2* Y,
                                                        long long ldy) {
  constexpr int MT = NT <= 3 ? 2 : 1;               // wide outputs hold more accumulators
  DmStream<MT> st(sK, ring, KS, r0, r1);
  const int lane = threadIdx.x & 31;
  double acc[MT][NT][2];
  int group = threadIdx.x >> 5, c_s = 0;
  for (int it = 0; it < st.nitems; ++it) {
    double2 a[MT];
    if (c_s == 0) {
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const long long ra = r0 + (long long)group * (8 * MT) + 8 * i + st.g;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int col = j * 4 + st.t;
          double2 y = make_double2(0.0, 0.0);
          if (ACC && col < q && ra < r1) y = Y[ra * ldy + col];
          acc[i][j][0] = y.x; acc[i][j][1] = y.y;
        }
      }
    }
    st.take(it, a);
    dm_step<NT, MT>(a, sB + (size_t)c_s * NT * 32 + lane, acc);
    st.done(it);
    if (++c_s == KS) {
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const long long ra = r0 + (long long)group * (8 * MT) + 8 * i + st.g;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int col = j * 4 + st.t;
          if (col < q && ra < r1) Y[ra * ldy + col] = make_double2(acc[i][j][0], acc[i][j][1]);
        }
      }
      c_s = 0;
      group += st.nw;
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

#define QDKP_NT_SWITCH(NT, CALL)                                                                  \
  switch (NT) {                                                                                  \
    case 1: { CALL(1) break; } case 2: { CALL(2) break; } case 3: { CALL(3) break; }              \
    case 4: { CALL(4) break; } case 5: { CALL(5) break; } case 6: { CALL(6) break; }              \
    default: break;                                                                              \
  }

// Y (+)= sg A C over rows [r0, r1). C[b] is the cols_b x q row-major coefficient block of A's block
// b; gather: columns of block 0 (NULL: as they stand); q <= kMaxBlock. Called by every thread of
// the CTA; smem holds update_smem_bytes.
static __device__ void update_rows(const BlockList<double>& A, const double2* const* C, int q,
                                   long long r0, long long r1, double2* Y, long long ldy,
                                   int accumulate, int neg, unsigned char* smem,
                                   const int* gather = nullptr) {
  __shared__ KStep<double> sK[kMaxSmall / 4 + 3];
  double2* ring = reinterpret_cast<double2*>(smem);
  double2* sB = reinterpret_cast<double2*>(smem + kDmRingBytes);
  int KS = 0;
  for (int b = 0; b < A.nblk; ++b) {
    if (threadIdx.x == 0) add_ksteps(sK, KS, A.p[b], A.ld[b], A.cols[b], b ? nullptr : gather);
    pack_dmma(sB, KS, C[b], A.cols[b], q, neg ? -1.0 : 1.0);
    KS += (A.cols[b] + 3) / 4;
  }
  __syncthreads();
#define QDKP_UPD(nt)                                                                              \
  if (accumulate) update_dmma_core<nt, true>(sK, sB, ring, KS, q, r0, r1, Y, ldy);                \
  else update_dmma_core<nt, false>(sK, sB, ring, KS, q, r0, r1, Y, ldy);
  QDKP_NT_SWITCH((q + 3) / 4, QDKP_UPD)
#undef QDKP_UPD
}

// ---------------------------------------------------------------------------------------------
// The Ritz update of an iteration in one pass over [X | R | P] and [AX | AR | AP] (lobpcg.py:
// 921-973): P = R Cr + P Cp, X = X Cx + P, the same for AP and AX, all in place, and with them the
// residuals A X - X lambda of the new iterate: their squared norms per column, and, if Rout is not
// NULL, the block itself. Six blocks are read and four (five) written, where two two-output updates,
// the norm and the residual kernels read ten and write five. P's sum is carried on into X's, so
// the six products are six block multiplications, not ten. Memory bounds it: 1.13 M rows of 12
// columns, complex128 (seven slots), 408 us at 5.9 TB/s; the four kernels took 960 us. The FP64 MMAs
// need 220 us of that; two M tiles a warp share the coefficient fragments while the accumulators and
// the kept X rows fit the registers (12 columns).
// ---------------------------------------------------------------------------------------------
template <typename T>
struct RitzArgs {
  cplx<T> *X, *R, *P, *AX, *AR, *AP;   // X, P, AX, AP: n x m (outputs); R, AR: n x ma; P, AP in: Pin, APin
  const cplx<T> *Pin, *APin;           // n x mp
  cplx<T>* Rout;                       // n x m, may be R when ma == m
  const double2 *Cx, *Cr, *Cp;
  const double* lam;
  double* npart;                       // m sums of this CTA
  int m, ma, mp;
};

constexpr int kRitzMaxKs = 2 * (kMaxSmall / 4 + 3);

// sum over the CTA's rows of nacc (lane: columns 4 j + t) into npart
template <int NT>
static __device__ __forceinline__ void ritz_norms(double (&nacc)[NT], int m, double* __restrict__ npart) {
  __shared__ double red[kUpdWarps][4 * NT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    double v = nacc[j];
    for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane < 4) red[warp][4 * j + lane] = v;
  }
  __syncthreads();
  if ((int)threadIdx.x < m) {
    double v = 0.0;
    for (int w = 0; w < kUpdWarps; ++w) v += red[w][threadIdx.x];
    npart[threadIdx.x] = v;
  }
}

template <int NT>
static __device__ __forceinline__ void ritz_dmma_core(const RitzArgs<double>& t, const KStep<double>* __restrict__ sK,
                                                      const double2* __restrict__ sB, double2* __restrict__ ring,
                                                      int KP, int KX, long long r0, long long r1) {
  constexpr int MT = NT <= 3 ? 2 : 1;
  const int KH = KP + KX;                           // k steps of one side
  DmStream<MT> st(sK, ring, 2 * KH, r0, r1);
  const int lane = threadIdx.x & 31, m = t.m;
  double lam[NT], nacc[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    nacc[j] = 0.0;
    lam[j] = j * 4 + st.t < m ? t.lam[j * 4 + st.t] : 0.0;
  }
  double acc[MT][NT][2], xs[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  int group = threadIdx.x >> 5, c_s = 0, k = 0;     // k step of the item, and within its side
  for (int it = 0; it < st.nitems; ++it) {
    double2 a[MT];
    st.take(it, a);
    dm_step<NT, MT>(a, sB + (size_t)k * NT * 32 + lane, acc);
    st.done(it);
    ++c_s;
    ++k;
    if (k == KP || k == KH) {
      const bool ax = c_s > KH;
      double2* out = k == KP ? (ax ? t.AP : t.P) : (ax ? t.AX : t.X);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const long long ra = r0 + (long long)group * (8 * MT) + 8 * i + st.g;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int col = j * 4 + st.t;
          const double2 v = make_double2(acc[i][j][0], acc[i][j][1]);
          if (col < m && ra < r1) {
            out[ra * m + col] = v;
            if (c_s == 2 * KH) {
              const double re = v.x - lam[j] * xs[i][j][0], im = v.y - lam[j] * xs[i][j][1];
              nacc[j] = fma(re, re, fma(im, im, nacc[j]));
              if (t.Rout) t.Rout[ra * m + col] = make_double2(re, im);
            }
          }
          if (k == KH) {
            xs[i][j][0] = v.x; xs[i][j][1] = v.y;
            acc[i][j][0] = acc[i][j][1] = 0.0;
          }
        }
      }
      if (k == KH) k = 0;
      if (c_s == 2 * KH) { c_s = 0; group += st.nw; }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  ritz_norms<NT>(nacc, m, t.npart);
}

__host__ __device__ __forceinline__ size_t ritz_smem_bytes(int m) { return update_smem_bytes(3 * m, m); }

static __device__ void ritz_rows(const RitzArgs<double>& t, long long r0, long long r1, unsigned char* smem) {
  __shared__ KStep<double> sK[kRitzMaxKs];
  double2* ring = reinterpret_cast<double2*>(smem);
  double2* sB = reinterpret_cast<double2*>(smem + kDmRingBytes);
  const int kr = (t.ma + 3) / 4, kp = (t.mp + 3) / 4, KX = (t.m + 3) / 4, KP = kr + kp;
  if (threadIdx.x == 0) {
    int s = add_ksteps<double>(sK, 0, t.R, t.ma, t.ma, nullptr);
    s = add_ksteps<double>(sK, s, t.Pin, t.mp, t.mp, nullptr);
    s = add_ksteps<double>(sK, s, t.X, t.m, t.m, nullptr);
    s = add_ksteps<double>(sK, s, t.AR, t.ma, t.ma, nullptr);
    s = add_ksteps<double>(sK, s, t.APin, t.mp, t.mp, nullptr);
    add_ksteps<double>(sK, s, t.AX, t.m, t.m, nullptr);
  }
  pack_dmma(sB, 0, t.Cr, t.ma, t.m, 1.0);
  pack_dmma(sB, kr, t.Cp, t.mp, t.m, 1.0);
  pack_dmma(sB, KP, t.Cx, t.m, t.m, 1.0);
  __syncthreads();
#define QDKP_RITZ(nt) ritz_dmma_core<nt>(t, sK, sB, ring, KP, KX, r0, r1);
  QDKP_NT_SWITCH(KX, QDKP_RITZ)
#undef QDKP_RITZ
}

// ---------------------------------------------------------------------------------------------
// complex64 blocks: split-precision TF32 tensor-core products (mma.sync.m16n8k8 .tf32, FP32
// accumulation). Every FP32 value x is split into x = hi + lo with hi, lo TF32 (10-bit
// mantissas; cvt.rna), and a product is formed as lo*hi + hi*lo + hi*hi (the lo*lo term is below
// FP32 rounding), which keeps the FP32 accuracy of the inputs. A CTA accumulates its rows in
// FP32 registers and writes an FP64 partial; partials are summed in FP64.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned tf32_round(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void tf32_split(float x, unsigned& hi, unsigned& lo) {
  hi = tf32_round(x);
  lo = tf32_round(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], unsigned a0, unsigned a1, unsigned a2,
                                         unsigned a3, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// d += (ahi + alo)(bhi + blo) without the lo * lo term
__device__ __forceinline__ void mma_tf32x3(float (&d)[4], const unsigned (&ah)[4],
                                           const unsigned (&al)[4], const unsigned (&bh)[2],
                                           const unsigned (&bl)[2]) {
  mma_tf32(d, al[0], al[1], al[2], al[3], bh[0], bh[1]);
  mma_tf32(d, ah[0], ah[1], ah[2], ah[3], bl[0], bl[1]);
  mma_tf32(d, ah[0], ah[1], ah[2], ah[3], bh[0], bh[1]);
}

// Y' = A' C'' for rows [r0, r1) of complex64 blocks on TF32 tensor cores (split as above).
// Nothing is staged: a warp owns 16-row M tiles (tiles warp, warp + warps, ... of the CTA's
// rows) and loads its A fragments from global memory into registers, a ring of k steps ahead of
// the MMAs, so a CTA needs no barrier after its coefficient setup. The MMA's k order is
// permuted so that a lane's two k values of a fragment row are the real and imaginary part of
// one complex element: k step s covers complex columns c0 .. c0 + 3 of one block, and
// MMA k = t <-> Re A[.][c0 + t], k = t + 4 <-> Im A[.][c0 + t] (g = lane / 4, t = lane % 4), so
// a0 a2 = A[row g][c0 + t] and a1 a3 = A[row g + 8][c0 + t] are one 8-byte load each. C'' (the
// real representation of the stacked complex coefficients, as in update_rows) is stored in that
// k order as one 16-byte word per (k step, 8-column N tile, lane): {hi b0, hi b1, lo b0, lo b1}
// with b0 = C''[k t][n g], b1 = C''[k t + 4][n g]. A row is read (by the four lanes of its quad)
// before any of its outputs is written and no other warp touches it, so Y may alias an input.
constexpr int kTfRing = 8;         // k steps of A fragments in flight per warp (narrow outputs)

// k steps of a list of at most three blocks with P columns in all (ceil(cols / 4) per block)
__host__ __device__ __forceinline__ int tf32_ksteps_bound(int P) { return (P + 3) / 4 + 2; }

__host__ __device__ __forceinline__ size_t update_tf32_smem_bytes(int P, int q) {
  return (size_t)tf32_ksteps_bound(P) * ((q + 3) / 4) * 32 * sizeof(uint4);
}

// Packs one block's coefficients for the TF32 MMA (k steps s0 .. of the list); every thread
static __device__ __forceinline__ void pack_tf32(uint4* __restrict__ sB, int s0, const double2* __restrict__ C,
                                                 int cols, int q, float sg) {
  const int NT = (q + 3) / 4, KS = (cols + 3) / 4;
  for (int e = threadIdx.x; e < KS * NT * 32; e += blockDim.x) {
    const int s = e / (NT * 32), r = e - s * NT * 32;
    const int j = r >> 5, ln = r & 31, gg = ln >> 2, tt = ln & 3;
    const int i = 4 * s + tt, jj = j * 4 + (gg >> 1);
    float v0 = 0.f, v1 = 0.f;
    if (i < cols && jj < q) {
      const double2 c = C[(size_t)i * q + jj];
      const float re = sg * (float)c.x, im = sg * (float)c.y;
      if (gg & 1) { v0 = im; v1 = re; }          // C''[2i][2jj+1], C''[2i+1][2jj+1]
      else { v0 = re; v1 = -im; }                // C''[2i][2jj],   C''[2i+1][2jj]
    }
    uint4 w;
    tf32_split(v0, w.x, w.z);
    tf32_split(v1, w.y, w.w);
    sB[(size_t)s0 * NT * 32 + e] = w;
  }
}

// A warp's stream of A fragments over (16-row tile, k step) items, RING in flight in registers
template <int RING>
struct TfStream {
  const KStep<float>* k;
  int KS, nitems, nw, g, t, l_tile, l_s;
  long long r0, r1;
  float2 fa[RING], fb[RING];
  __device__ __forceinline__ TfStream(const KStep<float>* k_, int KS_, long long r0_, long long r1_)
      : k(k_), KS(KS_), r0(r0_), r1(r1_) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    g = lane >> 2; t = lane & 3; nw = blockDim.x >> 5;
    const int ntiles = (int)((r1 - r0 + 15) / 16);
    nitems = (ntiles > warp ? (ntiles - warp + nw - 1) / nw : 0) * KS;
    l_tile = warp; l_s = 0;
#pragma unroll
    for (int d = 0; d < RING; ++d)
      if (d < nitems) fetch(d);
  }
  __device__ __forceinline__ void fetch(int d) {
    const KStep<float> ks = k[l_s];
    const long long ra = r0 + (long long)l_tile * 16 + g, rb = ra + 8;
    const float2 *pa = ks.at(t, ra, r1), *pb = ks.at(t, rb, r1);
    fa[d] = pa ? __ldcs(pa) : make_float2(0.f, 0.f);
    fb[d] = pb ? __ldcs(pb) : make_float2(0.f, 0.f);
    if (++l_s == KS) { l_s = 0; l_tile += nw; }
  }
  // item `it` in slot d: its split fragments; the slot is refilled
  __device__ __forceinline__ void take(int it, int d, unsigned (&ah)[4], unsigned (&al)[4]) {
    tf32_split(fa[d].x, ah[0], al[0]);
    tf32_split(fb[d].x, ah[1], al[1]);
    tf32_split(fa[d].y, ah[2], al[2]);
    tf32_split(fb[d].y, ah[3], al[3]);
    if (it + RING < nitems) fetch(d);
  }
};

template <int NT>
static __device__ __forceinline__ void tf_step(const unsigned (&ah)[4], const unsigned (&al)[4],
                                               const uint4* __restrict__ bp, float (&acc)[NT][4]) {
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const uint4 b = bp[j * 32];
    const unsigned bh[2] = {b.x, b.y}, bl[2] = {b.z, b.w};
    mma_tf32x3(acc[j], ah, al, bh, bl);
  }
}

template <int NT, bool ACC>
static __device__ __forceinline__ void update_tf32_core(const KStep<float>* __restrict__ sK,
                                                        const uint4* __restrict__ sB, int KS,
                                                        int q, long long r0, long long r1,
                                                        float2* Y, long long ldy) {
  constexpr int RING = kTfRing;
  TfStream<RING> st(sK, KS, r0, r1);
  const int lane = threadIdx.x & 31;
  float acc[NT][4];
  float2 yo[ACC ? NT : 1][2];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  int c_s = 0, tile = threadIdx.x >> 5;
  for (int base = 0; base < st.nitems; base += RING) {
#pragma unroll
    for (int d = 0; d < RING; ++d) {
      const int it = base + d;
      if (it >= st.nitems) break;
      unsigned ah[4], al[4];
      st.take(it, d, ah, al);
      const long long ra = r0 + (long long)tile * 16 + st.g, rb = ra + 8;
      if (ACC && c_s == 0) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int col = j * 4 + st.t;
          yo[j][0] = (col < q && ra < r1) ? Y[ra * ldy + col] : make_float2(0.f, 0.f);
          yo[j][1] = (col < q && rb < r1) ? Y[rb * ldy + col] : make_float2(0.f, 0.f);
        }
      }
      tf_step<NT>(ah, al, sB + (size_t)c_s * NT * 32 + lane, acc);
      if (++c_s == KS) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int col = j * 4 + st.t;
          if (col < q) {
            float2 va = make_float2(acc[j][0], acc[j][1]), vb = make_float2(acc[j][2], acc[j][3]);
            if (ACC) {
              va.x += yo[j][0].x; va.y += yo[j][0].y;
              vb.x += yo[j][1].x; vb.y += yo[j][1].y;
            }
            if (ra < r1) Y[ra * ldy + col] = va;
            if (rb < r1) Y[rb * ldy + col] = vb;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
        }
        c_s = 0;
        tile += st.nw;
      }
    }
  }
}

// Y (+)= sg A C over rows [r0, r1) of complex64 blocks; arguments as update_rows. smem holds
// update_tf32_smem_bytes.
static __device__ void update_rows_tf32(const BlockList<float>& A, const double2* const* C, int q,
                                        long long r0, long long r1, float2* Y, long long ldy,
                                        int accumulate, int neg, unsigned char* smem,
                                        const int* gather = nullptr) {
  __shared__ KStep<float> sK[kMaxSmall / 4 + 3];
  uint4* sB = reinterpret_cast<uint4*>(smem);
  int KS = 0;
  for (int b = 0; b < A.nblk; ++b) {
    if (threadIdx.x == 0) add_ksteps(sK, KS, A.p[b], A.ld[b], A.cols[b], b ? nullptr : gather);
    pack_tf32(sB, KS, C[b], A.cols[b], q, neg ? -1.f : 1.f);
    KS += (A.cols[b] + 3) / 4;
  }
  __syncthreads();
#define QDKP_UPD(nt)                                                                              \
  if (accumulate) update_tf32_core<nt, true>(sK, sB, KS, q, r0, r1, Y, ldy);                      \
  else update_tf32_core<nt, false>(sK, sB, KS, q, r0, r1, Y, ldy);
  QDKP_NT_SWITCH((q + 3) / 4, QDKP_UPD)
#undef QDKP_UPD
}

// the Ritz update (ritz_rows) of complex64 blocks; the residual in FP64 from the rounded X and A X
template <int NT>
static __device__ __forceinline__ void ritz_tf32_core(const RitzArgs<float>& t, const KStep<float>* __restrict__ sK,
                                                      const uint4* __restrict__ sB, int KP, int KX,
                                                      long long r0, long long r1) {
  constexpr int RING = NT <= 3 ? kTfRing : kTfRing / 2;
  const int KH = KP + KX;
  TfStream<RING> st(sK, 2 * KH, r0, r1);
  const int lane = threadIdx.x & 31, m = t.m;
  double nacc[NT];
  float acc[NT][4], xs[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    nacc[j] = 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  }
  int c_s = 0, k = 0, tile = threadIdx.x >> 5;
  for (int base = 0; base < st.nitems; base += RING) {
#pragma unroll
    for (int d = 0; d < RING; ++d) {
      const int it = base + d;
      if (it >= st.nitems) break;
      unsigned ah[4], al[4];
      st.take(it, d, ah, al);
      tf_step<NT>(ah, al, sB + (size_t)k * NT * 32 + lane, acc);
      ++c_s;
      ++k;
      if (k == KP || k == KH) {
        const bool ax = c_s > KH;
        float2* out = k == KP ? (ax ? t.AP : t.P) : (ax ? t.AX : t.X);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const long long ra = r0 + (long long)tile * 16 + st.g + 8 * h;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const int col = j * 4 + st.t;
            const float2 v = make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
            if (col < m && ra < r1) {
              out[ra * m + col] = v;
              if (c_s == 2 * KH) {
                const double l = t.lam[col];
                const double re = (double)v.x - l * (double)xs[j][2 * h];
                const double im = (double)v.y - l * (double)xs[j][2 * h + 1];
                nacc[j] = fma(re, re, fma(im, im, nacc[j]));
                if (t.Rout) t.Rout[ra * m + col] = make_float2((float)re, (float)im);
              }
            }
            if (k == KH) {
              xs[j][2 * h] = v.x; xs[j][2 * h + 1] = v.y;
              acc[j][2 * h] = acc[j][2 * h + 1] = 0.f;
            }
          }
        }
        if (k == KH) k = 0;
        if (c_s == 2 * KH) { c_s = 0; tile += st.nw; }
      }
    }
  }
  ritz_norms<NT>(nacc, m, t.npart);
}

__host__ __device__ __forceinline__ size_t ritz_tf32_smem_bytes(int m) { return update_tf32_smem_bytes(3 * m, m); }

static __device__ void ritz_rows_tf32(const RitzArgs<float>& t, long long r0, long long r1, unsigned char* smem) {
  __shared__ KStep<float> sK[kRitzMaxKs];
  uint4* sB = reinterpret_cast<uint4*>(smem);
  const int kr = (t.ma + 3) / 4, kp = (t.mp + 3) / 4, KX = (t.m + 3) / 4, KP = kr + kp;
  if (threadIdx.x == 0) {
    int s = add_ksteps<float>(sK, 0, t.R, t.ma, t.ma, nullptr);
    s = add_ksteps<float>(sK, s, t.Pin, t.mp, t.mp, nullptr);
    s = add_ksteps<float>(sK, s, t.X, t.m, t.m, nullptr);
    s = add_ksteps<float>(sK, s, t.AR, t.ma, t.ma, nullptr);
    s = add_ksteps<float>(sK, s, t.APin, t.mp, t.mp, nullptr);
    add_ksteps<float>(sK, s, t.AX, t.m, t.m, nullptr);
  }
  pack_tf32(sB, 0, t.Cr, t.ma, t.m, 1.f);
  pack_tf32(sB, kr, t.Cp, t.mp, t.m, 1.f);
  pack_tf32(sB, KP, t.Cx, t.m, t.m, 1.f);
  __syncthreads();
#define QDKP_RITZ(nt) ritz_tf32_core<nt>(t, sK, sB, KP, KX, r0, r1);
  QDKP_NT_SWITCH(KX, QDKP_RITZ)
#undef QDKP_RITZ
}

}  // namespace qdkp
