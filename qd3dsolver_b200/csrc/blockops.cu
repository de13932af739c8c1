// Tall-skinny block kernels (norms, residual gather, Gram, block update) and one-CTA FP64
// small dense kernels (Cholesky + triangular inverse, Hermitian generalized eigensolver by
// Householder reduction and implicit QL) for the LOBPCG driver.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>
#include <cstdlib>
#include <cstring>

#include "dense_dev.cuh"
#include "gram_dev.cuh"
#include "gram_tf32_dev.cuh"
#include "umma_dev.cuh"

namespace qdkp {

// ------------------------------------------------------------------------------------------------
// Column norms: out[j] = sum_r |A[r, j] - lambda_j B[r, j]|^2 (B may be NULL).
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kTallThreads)
colnorm2_partial(const cplx<T>* __restrict__ A, long long lda, const cplx<T>* __restrict__ B,
                 long long ldb, const double* __restrict__ lam, int m, long long n,
                 double* __restrict__ partial) {
  double acc[kMaxBlock];
#pragma unroll
  for (int j = 0; j < kMaxBlock; ++j) acc[j] = 0.0;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n;
       r += (long long)gridDim.x * blockDim.x) {
#pragma unroll
    for (int j = 0; j < kMaxBlock; ++j) {
      if (j < m) {
        const cplx<T> av = A[r * lda + j];
        double2 a = make_double2((double)av.x, (double)av.y);
        if (B) {
          const cplx<T> b = B[r * ldb + j];
          a.x -= lam[j] * (double)b.x;
          a.y -= lam[j] * (double)b.y;
        }
        acc[j] = fma(a.x, a.x, fma(a.y, a.y, acc[j]));
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
    partial[(long long)blockIdx.x * m + threadIdx.x] = s;
  }
}

// a warp per column (a thread per column took 20 us for 296 parts: one load after the other)
__global__ void __launch_bounds__(32 * kMaxBlock)
reduce_partials(const double* __restrict__ partial, int nparts, int m, double* __restrict__ out) {
  const int j = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0;
  for (int b = lane; b < nparts; b += 32) s += partial[(long long)b * m + j];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[j] = s;
}

template <typename T>
int launch_colnorm2(const cplx<T>* A, long long lda, const cplx<T>* B, long long ldb,
                    const double* lambda, int m, long long n, double* partial, int nparts,
                    double* out, cudaStream_t st) {
  if (m > kMaxBlock) { set_error("block wider than kMaxBlock"); return QDKP_ERR_ARG; }
  colnorm2_partial<T><<<nparts, kTallThreads, 0, st>>>(A, lda, B, ldb, lambda, m, n, partial);
  count_launch();
  reduce_partials<<<1, 32 * m, 0, st>>>(partial, nparts, m, out);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

template <typename TS, typename TD>
__global__ void copy_kernel(const cplx<TS>* __restrict__ src, long long lds, int cols, long long n,
                            cplx<TD>* __restrict__ dst, long long ldd) {
  const long long total = n * cols;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long r = e / cols;
    const int c = (int)(e - r * cols);
    const cplx<TS> v = src[r * lds + c];
    dst[r * ldd + c] = mk<TD>((TD)v.x, (TD)v.y);
  }
}

template <typename TS, typename TD>
int launch_copy(const cplx<TS>* src, long long lds, int cols, long long n, cplx<TD>* dst,
                long long ldd, cudaStream_t st) {
  if (std::is_same<TS, TD>::value && lds == cols && ldd == cols) {
    QDKP_CUDA_TRY(cudaMemcpyAsync(dst, src, (size_t)n * cols * sizeof(cplx<TD>),
                                  cudaMemcpyDeviceToDevice, st));
    return QDKP_OK;
  }
  copy_kernel<TS, TD><<<1184, 256, 0, st>>>(src, lds, cols, n, dst, ldd);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

// ------------------------------------------------------------------------------------------------
// Gram: out = A^H B over concatenated column lists, FP64 accumulation, deterministic (gram_dev.cuh).
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(32 * (kGramMaxWarps + 1), 1)
gram_kernel(const GramTask<T> t, int parts, double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char gsm_d[];
  gram_core(t, (int)blockIdx.x, parts, (int)blockIdx.y, partial, gsm_d);
}

// out row-major with leading dimension Q (GK_FULL, GK_HERM: both triangles)
template <typename T>
__global__ void __launch_bounds__(kGramRedThreads)
gram_reduce_kernel(const GramTask<T> t, int parts, const double* __restrict__ partial,
                   double2* __restrict__ out) {
  gram_reduce_core(t, parts, partial, (int)blockIdx.x, (int)gridDim.x,
                   [&](int i, int j, double2 v) { gram_put(t, i, j, v, out, out); });
}

size_t gram_partial_elems(int P, int Q) {
  const size_t rects = (size_t)((P + kGramRect - 1) / kGramRect) * ((Q + kGramRect - 1) / kGramRect);
  return rects * kGramMaxParts * kGramRectElems / 2;
}

// ... of a qdkp_block_gram, in either precision, and of any narrower one: split TF32 takes products of up to
// kTfMaxRects rectangles and more room for the widest of them than FP64 for some wider ones
static size_t block_gram_elems(int P, int Q) {
  size_t e = gram_partial_elems(P, Q);
  for (int r = 1; r <= kTfMaxRects && kGramRect * (r - 1) < P; ++r)
    e = std::max(e, gram_tf32_doubles(std::min(P, kGramRect * r), std::min(Q, kGramRect * (kTfMaxRects / r))) / 2);
  return e;
}

__global__ void __launch_bounds__(512)
gram_tf32_kernel(const BlockList<float> A, const BlockList<float> B, long long n, long long rows_per_part,
                 double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char gsm_f[];
  const long long r0 = blockIdx.x * rows_per_part;
  const int RP = (2 * A.total() + 7) / 8 * 8, RQ = (2 * B.total() + 7) / 8 * 8;
  gram_core_tf32(A, B, r0, min(n, r0 + rows_per_part), partial + (long long)blockIdx.x * RP * RQ, gsm_f);
}

// out = the parts' sum as a complex P x Q product, 32 entries a CTA: each of 16 warps adds a sixteenth of the
// parts in order, then the sixteenths are added in order. Latency bounds it: 80,000
// rows of 18 x 12 columns took 59 us with eight warps of four parts' loads in flight, 49 us so (product, sums
// and the copy of the result).
constexpr int kTfRedWarps = 16;
__global__ void __launch_bounds__(32 * kTfRedWarps)
gram_tf32_reduce_kernel(const double* __restrict__ partial, int parts, int P, int Q, double2* __restrict__ out) {
  __shared__ double2 s_sum[kTfRedWarps][32];
  const int RP = (2 * P + 7) / 8 * 8, RQ = (2 * Q + 7) / 8 * 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, o = blockIdx.x * 32 + lane;
  const int i = o / Q, j = o - i * Q, per = (parts + kTfRedWarps - 1) / kTfRedWarps;
  double2 v = make_double2(0.0, 0.0);
  if (o < P * Q)
    v = gram_add_parts(partial + (long long)(2 * i) * RQ + 2 * j, (long long)RP * RQ, warp * per,
                       min(parts, (warp + 1) * per), RQ);
  s_sum[warp][lane] = v;
  __syncthreads();
  if (warp || o >= P * Q) return;
  for (int w = 1; w < kTfRedWarps; ++w) { v.x += s_sum[w][lane].x; v.y += s_sum[w][lane].y; }
  out[o] = v;
}

static int launch_gram_tf32(const BlockList<float>& A, const BlockList<float>& B, long long n, int threads,
                            double2* partial, size_t partial_elems, double2* out, cudaStream_t st) {
  const int P = A.total(), Q = B.total();
  if (gram_tf32_doubles(P, Q) > 2 * partial_elems) {
    set_error("gram partial buffer too small");
    return QDKP_ERR_WORKSPACE;
  }
  long long parts = std::max(1LL, std::min<long long>((n + 255) / 256, kGramTfParts));
  const long long rpp = ((n + parts - 1) / parts + 3) / 4 * 4;
  parts = (n + rpp - 1) / rpp;
  const size_t smem = gram_smem_bytes(P, Q, (int)sizeof(float2));
  QDKP_CUDA_TRY(cudaFuncSetAttribute(gram_tf32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  double* pd = reinterpret_cast<double*>(partial);
  gram_tf32_kernel<<<(unsigned)parts, threads, smem, st>>>(A, B, n, rpp, pd);
  gram_tf32_reduce_kernel<<<(P * Q + 31) / 32, 32 * kTfRedWarps, 0, st>>>(pd, (int)parts, P, Q, out);
  count_launch(2);
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

template <typename T>
static int launch_gram_task(const GramTask<T>& t, double2* partial, size_t partial_elems, double2* out,
                            cudaStream_t st) {
  const GramShape sh = gram_shape(t.kind, t.P, t.Q, t.m, t.ma, t.mp);
  const int parts = gram_parts(t.n);
  if (gram_partial_doubles(sh.rects, parts) > 2 * partial_elems) {
    set_error("gram partial buffer too small");
    return QDKP_ERR_WORKSPACE;
  }
  const size_t smem = gram_smem<T>(t.tc, sh.warps);
  QDKP_CUDA_TRY(cudaFuncSetAttribute(gram_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramMaxSmem));
  double* pd = reinterpret_cast<double*>(partial);
  gram_kernel<T><<<dim3((unsigned)parts, (unsigned)sh.panels), 32 * (sh.warps + 1), smem, st>>>(t, parts, pd);
  gram_reduce_kernel<T><<<(t.P * t.Q + 31) / 32, kGramRedThreads, 0, st>>>(t, parts, pd, out);
  count_launch(2);
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

template <typename T>
int launch_gram(const BlockList<T>& A, const BlockList<T>& B, long long n,
                double2* partial, size_t partial_elems, double2* out, cudaStream_t st) {
  const int P = A.total(), Q = B.total();
  if (P > kMaxSmall || Q > kMaxSmall || P <= 0 || Q <= 0) {
    set_error("gram dimensions out of range");
    return QDKP_ERR_ARG;
  }
  bool same = A.nblk == B.nblk;
  for (int b = 0; b < A.nblk && same; ++b)
    same = A.p[b] == B.p[b] && A.cols[b] == B.cols[b] && A.ld[b] == B.ld[b];
  GramTask<T> t{};
  for (int side = 0; side < (same ? 1 : 2); ++side) {
    const BlockList<T>& L = side ? B : A;
    for (int b = 0; b < L.nblk; ++b) {
      t.p[t.nblk] = L.p[b]; t.ld[t.nblk] = L.ld[b]; t.cols[t.nblk] = L.cols[b];
      ++t.nblk;
    }
  }
  t.tc = same ? P : P + Q;
  t.a0 = 0; t.P = P; t.b0 = same ? 0 : P; t.Q = Q;
  t.kind = same ? GK_HERM : GK_FULL;
  t.n = n;
  int device = 0;
  QDKP_CUDA_TRY(cudaGetDevice(&device));
  t.fault = device_fault_flag(device);
  return launch_gram_task(t, partial, partial_elems, out, st);
}

// ------------------------------------------------------------------------------------------------
// Block update: Y = beta Y + sum_k A_k C_k  (C_k row-major cols_k x q)
// ------------------------------------------------------------------------------------------------
struct CoefList {
  const double2* c[3];
};

template <typename T>
__global__ void __launch_bounds__(kUpdThreads, 2)
update_kernel(const BlockList<T> A, const CoefList C, int q, long long n, cplx<T>* Y,
              long long ldy, int accumulate) {
  extern __shared__ __align__(16) unsigned char usm[];
  const double2* Cf[3] = {C.c[0], C.c[1], C.c[2]};
  const int chunk = update_chunk<T>(q);
  const long long per = ((n + gridDim.x - 1) / gridDim.x + chunk - 1) / chunk * chunk;
  const long long r0 = (long long)blockIdx.x * per;
  if (r0 >= n) return;
  if constexpr (std::is_same<T, float>::value)
    update_rows_tf32(A, Cf, q, r0, min(n, r0 + per), Y, ldy, accumulate, 0, usm);
  else
    update_rows(A, Cf, q, r0, min(n, r0 + per), Y, ldy, accumulate, 0, usm);
}

// complex64 blocks on the tcgen05 tensor cores (umma_dev.cuh): one CTA per SM at most, each a
// contiguous range of 128-row tiles run as one pipeline
__global__ void __launch_bounds__(kUmmaThreads, 1)
update_umma_kernel(const BlockList<float> A, const CoefList C, int q, long long n, float2* Y,
                   long long ldy, int accumulate, int cmax, int ldmax, int* fault) {
  extern __shared__ __align__(128) unsigned char usm_u[];
  const double2* Cf[3] = {C.c[0], C.c[1], C.c[2]};
  const UmmaPlan pl = umma_plan(A.total(), q, 1, cmax, ldmax);
  const long long tiles = (n + kUmmaRows - 1) / kUmmaRows;
  const long long per = (tiles + gridDim.x - 1) / gridDim.x * kUmmaRows;
  const long long r0 = (long long)blockIdx.x * per;
  if (r0 >= n) return;
  UmmaCtx cx;
  umma_ctx_init(cx, pl);
  const bool ok = update_rows_umma(pl, cx, A, Cf, q, r0, min(n, r0 + per), Y, ldy, accumulate, 0, usm_u);
  if (!ok && threadIdx.x == 0) raise_device_fault(fault);
  umma_ctx_free(cx);
}

bool c64_update_tcgen05() {
  static const bool on = [] {
    const char* v = std::getenv("QDKP_C64_UPDATE");
    if (v && std::strcmp(v, "mma") == 0) return false;
    if (v && std::strcmp(v, "tcgen05") == 0) return true;
    return kC64UpdateTcgen05Default;
  }();
  return on;
}

template <typename T>
int launch_update(const BlockList<T>& A, const double2* const* C, int q, long long n,
                  cplx<T>* Y, long long ldy, int accumulate, cudaStream_t st) {
  if (q > kMaxBlock || A.total() > kMaxSmall || q < 1) { set_error("update dimensions out of range"); return QDKP_ERR_ARG; }
  CoefList cl;
  for (int b = 0; b < 3; ++b) cl.c[b] = b < A.nblk ? C[b] : nullptr;
  const int P = A.total();
  if constexpr (std::is_same<T, float>::value) if (c64_update_tcgen05()) {
    static bool uattr = false;
    if (!uattr) {
      QDKP_CUDA_TRY(cudaFuncSetAttribute(update_umma_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kUmmaSmemLimit));
      uattr = true;
    }
    // blocks are split into sub-blocks of at most kMaxBlock columns (the operand buffers' width),
    // three to a launch; a list that needs more sub-blocks is formed by launches that accumulate
    // (there Y must not alias an input). Raw stages hold rows of up to 32 complex values; a
    // block with a longer row is read directly.
    struct Sub { const float2* p; long long ld; int cols; const double2* c; };
    std::vector<Sub> subs;
    for (int b = 0; b < A.nblk; ++b)
      for (int c0 = 0; c0 < A.cols[b]; c0 += kMaxBlock)
        subs.push_back({A.p[b] + c0, A.ld[b], std::min(kMaxBlock, A.cols[b] - c0),
                        C[b] ? C[b] + (size_t)c0 * q : nullptr});
    int nsm = 148, device = 0;
    QDKP_CUDA_TRY(cudaGetDevice(&device));
    QDKP_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, 0));
    long long ublocks = (n + kUmmaRows - 1) / kUmmaRows;
    if (ublocks > nsm) ublocks = nsm;
    for (size_t s0 = 0; s0 < subs.size(); s0 += 3) {
      BlockList<float> L;
      CoefList cs;
      L.nblk = (int)std::min<size_t>(3, subs.size() - s0);
      int cmax = 1, ldmax = 1, Ps = 0;
      for (int b = 0; b < 3; ++b) cs.c[b] = nullptr;
      for (int b = 0; b < L.nblk; ++b) {
        const Sub& u = subs[s0 + b];
        L.p[b] = u.p; L.ld[b] = u.ld; L.cols[b] = u.cols; cs.c[b] = u.c;
        cmax = std::max(cmax, u.cols);
        if (u.ld <= 32) ldmax = std::max(ldmax, (int)u.ld);
        Ps += u.cols;
      }
      ldmax = std::max(ldmax, cmax);
      const UmmaPlan pl = umma_plan(Ps, q, 1, cmax, ldmax);
      if (!pl.nout_pass) { set_error("tcgen05 update plan does not fit shared memory"); return QDKP_ERR_ARG; }
      update_umma_kernel<<<(unsigned)ublocks, kUmmaThreads, pl.bytes, st>>>(
          L, cs, q, n, Y, ldy, s0 == 0 ? accumulate : 1, cmax, ldmax, device_fault_flag(device));
      count_launch();
      QDKP_CUDA_TRY(cudaGetLastError());
    }
    return QDKP_OK;
  }
  const size_t smem = std::is_same<T, float>::value ? update_tf32_smem_bytes(P, q)
                                                    : update_smem_bytes(P, q);
  static bool attr = false;
  if (!attr) {
    QDKP_CUDA_TRY(cudaFuncSetAttribute(update_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       200 * 1024));
    attr = true;
  }
  const int chunk = update_chunk<T>(q);
  long long blocks = (n + chunk - 1) / chunk;
  if (blocks > 148 * 4) blocks = 148 * 4;
  update_kernel<T><<<(unsigned)blocks, kUpdThreads, smem, st>>>(A, cl, q, n, Y, ldy, accumulate);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

// ------------------------------------------------------------------------------------------------
// Small dense FP64 (one CTA).
// ------------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(kSmallThreads)
chol_inv_kernel(const double2* __restrict__ G, int n, double2* __restrict__ Uinv,
                int* __restrict__ status) {
  extern __shared__ double2 ssm[];
  double2* S1 = ssm + n * n;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) ssm[e] = G[e];
  __syncthreads();
  __shared__ double rinv[kMaxSmall], least[kMaxSmall];
  // A repeated column's entries of the Gram matrix are the same bits as the first one's; its pivot is then the
  // rounding of |G_ab|^2 / G_aa, at most three units (square, reciprocal, product) of 2^-53 of its diagonal
  // and of either sign. Beyond that a column counts as its own: one 3e-8 off another leaves 9e-16, give or
  // take the rounding of the sums.
  for (int k = threadIdx.x; k < n; k += blockDim.x) least[k] = 3.4e-16 * ssm[k * n + k].x;
  __syncthreads();
  const int fail = rr_cholesky(ssm, n, rinv, 0, least);
  if (threadIdx.x == 0) *status = fail;
  if (fail) return;
  rr_upper_inverse(ssm, n, rinv, S1);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) Uinv[e] = S1[e];
}

// The shared-memory limit of the kernels below: the widest matrix's, whatever this call needs. It is a property
// of the kernel that every thread of the process shares; a call that lowered it to its own size made a wider
// one's launch on another thread fail.
constexpr int kSmallSmem = 2 * kMaxSmall * kMaxSmall * (int)sizeof(double2);

int launch_chol_inv(const double2* G, int n, double2* Uinv, int* status, cudaStream_t st) {
  if (n < 1 || n > kMaxSmall) { set_error("chol_inv dimension out of range"); return QDKP_ERR_ARG; }
  const size_t smem = 2 * (size_t)n * n * sizeof(double2);
  QDKP_CUDA_TRY(cudaFuncSetAttribute(chol_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem));
  chol_inv_kernel<<<1, kSmallThreads, smem, st>>>(G, n, Uinv, status);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

// w ascending, V columns permuted accordingly; generalized problem through B = U^H U (with
// 0 < nwant < n only the first nwant pairs are computed).
template <int CLASS>
__global__ void __launch_bounds__(kSmallThreads)
eigh_kernel(const double2* __restrict__ A, const double2* __restrict__ B, int n,
            double* __restrict__ w, double2* __restrict__ Vout, double2* __restrict__ scratch,
            int* __restrict__ status, int nwant, int s1) {
  const int st = block_eigh<CLASS>(A, B, n, w, Vout, scratch, nwant, s1);
  if (threadIdx.x == 0) *status = st;
}

int launch_eigh(const double2* A, const double2* B, int n, double* w, double2* V,
                double2* scratch, int* status, cudaStream_t st, int nwant) {
  if (n < 1 || n > kMaxSmall) { set_error("eigh dimension out of range"); return QDKP_ERR_ARG; }
  // all pairs of a block's own matrix (the first and the last Rayleigh-Ritz of a solve) by the same
  // parallel route as a wanted few, with room for its arrays: 12 x 12 105 us by the QL iteration, 55 us so
  const int want = nwant > 0 && nwant < n ? nwant : n;
  const int s1 = std::max(2 * n * n, want <= kMaxBlock ? rr_s1_doubles(n, want) : 0);
  const size_t smem = (size_t)n * n * sizeof(double2) + (size_t)s1 * sizeof(double);
  const auto kernel = rr_class(n) == 0 ? eigh_kernel<0> : (rr_class(n) == 1 ? eigh_kernel<1> : eigh_kernel<2>);
  QDKP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem));
  kernel<<<1, kSmallThreads, smem, st>>>(A, B, n, w, V, scratch, status, want, s1);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

// complex128 (plain form, refinement) and complex64 (mixed-precision search) blocks
#define QDKP_BLOCKOPS_INST(T)                                                                      \
  template int launch_colnorm2<T>(const cplx<T>*, long long, const cplx<T>*, long long,          \
                                  const double*, int, long long, double*, int, double*,          \
                                  cudaStream_t);                                                 \
  template int launch_gram<T>(const BlockList<T>&, const BlockList<T>&, long long, double2*,     \
                              size_t, double2*, cudaStream_t);                                   \
  template int launch_update<T>(const BlockList<T>&, const double2* const*, int, long long,       \
                                cplx<T>*, long long, int, cudaStream_t);
QDKP_BLOCKOPS_INST(double)
QDKP_BLOCKOPS_INST(float)
#undef QDKP_BLOCKOPS_INST
template int launch_copy<double, double>(const double2*, long long, int, long long, double2*,
                                         long long, cudaStream_t);
template int launch_copy<float, float>(const float2*, long long, int, long long, float2*,
                                       long long, cudaStream_t);
template int launch_copy<double, float>(const double2*, long long, int, long long, float2*,
                                        long long, cudaStream_t);
template int launch_copy<float, double>(const float2*, long long, int, long long, double2*,
                                        long long, cudaStream_t);

}  // namespace qdkp

using namespace qdkp;

extern "C" {

size_t qdkp_block_gram_workspace_size(int P, int Q) {
  if (P < 1 || Q < 1 || P > kMaxSmall || Q > kMaxSmall) return 0;
  return block_gram_elems(P, Q) * sizeof(double2) + (size_t)P * Q * sizeof(double2) + 256;
}

int qdkp_block_gram(const void* A, int64_t lda, int P, const void* B, int64_t ldb, int Q,
                    int64_t n, int precision, double* out, void* ws, size_t ws_bytes,
                    void* stream) {
  QDKP_CHECK_ARG(A && B && out && ws, "NULL argument");
  QDKP_CHECK_ARG(P >= 1 && Q >= 1 && P <= kMaxSmall && Q <= kMaxSmall && n >= 1 && lda >= P &&
                 ldb >= Q, "bad block shapes");
  QDKP_CHECK_ARG(precision == QDKP_C128 || precision == QDKP_C64, "bad precision");
  if (ws_bytes < qdkp_block_gram_workspace_size(P, Q)) {
    set_error("qdkp_block_gram: workspace too small");
    return QDKP_ERR_WORKSPACE;
  }
  int device = 0;
  QDKP_CUDA_TRY(cudaGetDevice(&device));
  if (const int rc = init_device_fault()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t pe = block_gram_elems(P, Q);
  double2* part = static_cast<double2*>(ws);
  double2* dout = part + pe;
  int rc;
  if (precision == QDKP_C64) {
    BlockList<float> La, Lb;
    La.nblk = 1; La.p[0] = static_cast<const float2*>(A); La.ld[0] = lda; La.cols[0] = P;
    Lb.nblk = 1; Lb.p[0] = static_cast<const float2*>(B); Lb.ld[0] = ldb; Lb.cols[0] = Q;
    const int threads = gram_tf32_threads(P, Q);
    rc = threads ? launch_gram_tf32(La, Lb, n, threads, part, pe, dout, st)
                 : launch_gram(La, Lb, n, part, pe, dout, st);
  } else {
    BlockList<double> La, Lb;
    La.nblk = 1; La.p[0] = static_cast<const double2*>(A); La.ld[0] = lda; La.cols[0] = P;
    Lb.nblk = 1; Lb.p[0] = static_cast<const double2*>(B); Lb.ld[0] = ldb; Lb.cols[0] = Q;
    rc = launch_gram(La, Lb, n, part, pe, dout, st);
  }
  if (rc != QDKP_OK) return rc;
  QDKP_CUDA_TRY(cudaMemcpyAsync(out, dout, (size_t)P * Q * sizeof(double2), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  return check_device_fault(device);
}

size_t qdkp_block_eigh_workspace_size(int n) {
  if (n < 1 || n > kMaxSmall) return 0;
  const size_t mat = ((size_t)n * n * sizeof(double2) + 255) / 256 * 256;
  return 5 * mat + ((size_t)n * sizeof(double) + 255) / 256 * 256 + 256;
}

int qdkp_block_eigh(const double* A, const double* B, int n, int nwant, double* w, double* V,
                    void* ws, size_t ws_bytes, void* stream) {
  QDKP_CHECK_ARG(A && w && V && ws, "NULL argument");
  QDKP_CHECK_ARG(n >= 1 && n <= kMaxSmall, "n must be in [1, 72]");
  QDKP_CHECK_ARG(nwant >= 1 && nwant <= n, "nwant must be in [1, n]");
  if (ws_bytes < qdkp_block_eigh_workspace_size(n)) {
    set_error("qdkp_block_eigh: workspace too small");
    return QDKP_ERR_WORKSPACE;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t mb = (size_t)n * n * sizeof(double2);
  const size_t mat = (mb + 255) / 256 * 256;
  char* p = static_cast<char*>(ws);
  double2* dA = reinterpret_cast<double2*>(p);
  double2* dB = reinterpret_cast<double2*>(p + mat);
  double2* dV = reinterpret_cast<double2*>(p + 2 * mat);
  double2* scr = reinterpret_cast<double2*>(p + 3 * mat);     // 2 n^2
  double* dw = reinterpret_cast<double*>(p + 5 * mat);
  int* dstat = reinterpret_cast<int*>(p + 5 * mat + ((size_t)n * sizeof(double) + 255) / 256 * 256);
  QDKP_CUDA_TRY(cudaMemcpyAsync(dA, A, mb, cudaMemcpyHostToDevice, st));
  if (B) QDKP_CUDA_TRY(cudaMemcpyAsync(dB, B, mb, cudaMemcpyHostToDevice, st));
  const int rc = launch_eigh(dA, B ? dB : nullptr, n, dw, dV, scr, dstat, st, nwant < n ? nwant : 0);
  if (rc != QDKP_OK) return rc;
  int hstat = 0;
  QDKP_CUDA_TRY(cudaMemcpyAsync(w, dw, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaMemcpyAsync(V, dV, mb, cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaMemcpyAsync(&hstat, dstat, sizeof(int), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  if (hstat != 0) {
    set_error(hstat == 1 ? "qdkp_block_eigh: B is not positive definite"
                         : "qdkp_block_eigh: non-finite spectrum");
    return QDKP_ERR_NUMERIC;
  }
  return QDKP_OK;
}

size_t qdkp_block_update_workspace_size(int P, int q) {
  if (P < 1 || q < 1 || P > kMaxSmall || q > kMaxBlock) return 0;
  return (size_t)P * q * sizeof(double2) + 256;
}

int qdkp_block_update(const void* A, int64_t lda, int P, const double* C, int q, int64_t n,
                      void* Y, int64_t ldy, int precision, void* ws, size_t ws_bytes,
                      void* stream) {
  QDKP_CHECK_ARG(A && C && Y && ws, "NULL argument");
  QDKP_CHECK_ARG(P >= 1 && q >= 1 && P <= kMaxSmall && q <= kMaxBlock && n >= 1 && lda >= P &&
                 ldy >= q, "bad block shapes");
  QDKP_CHECK_ARG(precision == QDKP_C128 || precision == QDKP_C64, "bad precision");
  if (ws_bytes < qdkp_block_update_workspace_size(P, q)) {
    set_error("qdkp_block_update: workspace too small");
    return QDKP_ERR_WORKSPACE;
  }
  int device = 0;
  QDKP_CUDA_TRY(cudaGetDevice(&device));
  if (const int rc2 = init_device_fault()) return rc2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double2* dC = static_cast<double2*>(ws);
  QDKP_CUDA_TRY(cudaMemcpyAsync(dC, C, (size_t)P * q * sizeof(double2), cudaMemcpyHostToDevice, st));
  const double2* Cs[1] = {dC};
  int rc;
  if (precision == QDKP_C64) {
    BlockList<float> La;
    La.nblk = 1; La.p[0] = static_cast<const float2*>(A); La.ld[0] = lda; La.cols[0] = P;
    rc = launch_update(La, Cs, q, n, static_cast<float2*>(Y), ldy, 0, st);
  } else {
    BlockList<double> La;
    La.nblk = 1; La.p[0] = static_cast<const double2*>(A); La.ld[0] = lda; La.cols[0] = P;
    rc = launch_update(La, Cs, q, n, static_cast<double2*>(Y), ldy, 0, st);
  }
  if (rc != QDKP_OK) return rc;
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  return check_device_fault(device);
}

}  // extern "C"
