// Homogeneous Fourier strain and the first-order piezoelectric potential on the device (sm_100a).
//
//   strain_fourier.solve_strain (strain_fourier.py:142-235): chi = dot mask; u_k = -i eps_T
//     (C11 + 2 C12) chi_k K(k)^-1 k with K the cubic Christoffel matrix K_ik = C_ijkl k_j k_l
//     (its inverse by cofactors, 0 where det K = 0, i.e. the k = 0 mode); total strain = the
//     symmetric spectral gradient of u; elastic = total - eps_T chi on the diagonal
//     (eps_T = -eps_star).
//   piezoelectric.potential (piezoelectric.py:59-99): P = 2 e14 (eyz, ezx, exy) sign;
//     rho = -Re ifft(i k . fft P) CHARGE_UNIT; phi = Re ifft(fft(rho) POISSON_CONST / (eps_r k^2))
//     with the k = 0 mode dropped.
// k = 2 pi fftfreq(n, h) on a C-ordered (nx, ny, nz) grid: the same periodic cell as numpy's fftn.
// The plain 3-D transforms are cuFFT double-precision plans (complex, and real for the FD elasticity;
// one per grid shape, kept for reuse, work area in the caller's workspace); the Christoffel inverse, the spectral derivatives, the
// Poisson filter and the real parts are this file's kernels. Every step is a fixed-order
// computation: the result does not depend on other work on the GPU.
#include <cufft.h>

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "qdkp_common.cuh"

namespace qdkp {

constexpr double kEcharge = 1.602176634e-19;                 // C (poisson_solver.py:25)
constexpr double kEps0 = 8.8541878128e-12;                   // F/m (poisson_solver.py:26)
constexpr double kPoissonConst = kEcharge * 1e9 / kEps0;     // V nm (poisson_solver.py:30)
constexpr double kChargeUnit = 1.0 / (kEcharge * 1e18);      // piezoelectric.py:50

struct Grid3 { int nx, ny, nz; double h; };

__device__ __forceinline__ double kcomp(int i, int n, double h) {
  const int f = (i <= (n - 1) / 2) ? i : i - n;                // numpy fftfreq order
  return 6.283185307179586476925286766559 * (double)f / ((double)n * h);
}

__device__ __forceinline__ void kvec(long long s, Grid3 g, double& kx, double& ky, double& kz) {
  const int iz = (int)(s % g.nz);
  const long long t = s / g.nz;
  const int iy = (int)(t % g.ny), ix = (int)(t / g.ny);
  kx = kcomp(ix, g.nx, g.h); ky = kcomp(iy, g.ny, g.h); kz = kcomp(iz, g.nz, g.h);
}

__global__ void mask_to_complex(const unsigned char* __restrict__ mask, long long N,
                                double2* __restrict__ chi) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x)
    chi[s] = make_double2(mask[s] ? 1.0 : 0.0, 0.0);
}

// six strain spectra from chi_k (cubic Christoffel inverse by cofactors, strain_fourier.py:142-173)
__global__ void strain_spectra(const double2* __restrict__ chik, long long N, Grid3 g,
                               double C11, double C12, double C44, double eps_T,
                               double2* __restrict__ out) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    double kx, ky, kz;
    kvec(s, g, kx, ky, kz);
    const double cs = C12 + C44;
    const double k11 = C11 * kx * kx + C44 * (ky * ky + kz * kz);
    const double k22 = C11 * ky * ky + C44 * (kx * kx + kz * kz);
    const double k33 = C11 * kz * kz + C44 * (kx * kx + ky * ky);
    const double k12 = cs * kx * ky, k13 = cs * kx * kz, k23 = cs * ky * kz;
    const double c11 = k22 * k33 - k23 * k23, c12 = k13 * k23 - k12 * k33;
    const double c13 = k12 * k23 - k13 * k22, c22 = k11 * k33 - k13 * k13;
    const double c23 = k12 * k13 - k11 * k23, c33 = k11 * k22 - k12 * k12;
    const double det = k11 * c11 + k12 * c12 + k13 * c13;
    const double inv = det != 0.0 ? 1.0 / det : 0.0;
    const double i11 = c11 * inv, i12 = c12 * inv, i13 = c13 * inv;
    const double i22 = c22 * inv, i23 = c23 * inv, i33 = c33 * inv;
    // pref = -i eps_T (C11 + 2 C12) chi_k
    const double a = eps_T * (C11 + 2.0 * C12);
    const double2 ck = chik[s];
    const double2 pref = make_double2(a * ck.y, -a * ck.x);
    const double gx = i11 * kx + i12 * ky + i13 * kz;
    const double gy = i12 * kx + i22 * ky + i23 * kz;
    const double gz = i13 * kx + i23 * ky + i33 * kz;
    const double2 ux = make_double2(pref.x * gx, pref.y * gx);
    const double2 uy = make_double2(pref.x * gy, pref.y * gy);
    const double2 uz = make_double2(pref.x * gz, pref.y * gz);
    // i c w = (-c w.y, c w.x)
    auto ic = [](double c, double2 w) { return make_double2(-c * w.y, c * w.x); };
    auto add = [](double2 p, double2 q) { return make_double2(p.x + q.x, p.y + q.y); };
    out[0 * N + s] = ic(kx, ux);
    out[1 * N + s] = ic(ky, uy);
    out[2 * N + s] = ic(kz, uz);
    out[3 * N + s] = ic(0.5, add(make_double2(ky * ux.x, ky * ux.y), make_double2(kx * uy.x, kx * uy.y)));
    out[4 * N + s] = ic(0.5, add(make_double2(kz * uy.x, kz * uy.y), make_double2(ky * uz.x, ky * uz.y)));
    out[5 * N + s] = ic(0.5, add(make_double2(kx * uz.x, kx * uz.y), make_double2(kz * ux.x, kz * ux.y)));
  }
}

// strain[c] = Re(spec[c]) / N - (c < 3 ? eps_T chi : 0)
__global__ void strain_real(const double2* __restrict__ spec, const unsigned char* __restrict__ mask,
                            long long N, double eps_T, double* __restrict__ strain) {
  const double invN = 1.0 / (double)N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < 6 * N;
       e += (long long)gridDim.x * blockDim.x) {
    const long long c = e / N, s = e - c * N;
    double v = spec[e].x * invN;
    if (c < 3 && mask[s]) v -= eps_T;
    strain[e] = v;
  }
}

// P components as complex: (eyz, ezx, exy) * 2 e14 sign
__global__ void polarization_k(const double* __restrict__ strain, const double* __restrict__ e14,
                               long long N, double sign, double2* __restrict__ P) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    const double f = 2.0 * e14[s] * sign;
    P[s] = make_double2(f * strain[4 * N + s], 0.0);             // eyz
    P[N + s] = make_double2(f * strain[5 * N + s], 0.0);         // ezx
    P[2 * N + s] = make_double2(f * strain[3 * N + s], 0.0);     // exy
  }
}

// div_k = i kx P0 + i ky P1 + i kz P2
__global__ void divergence_k(const double2* __restrict__ P, long long N, Grid3 g,
                             double2* __restrict__ div) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    double kx, ky, kz;
    kvec(s, g, kx, ky, kz);
    const double2 a = P[s], b = P[N + s], c = P[2 * N + s];
    div[s] = make_double2(-(kx * a.y + ky * b.y + kz * c.y), kx * a.x + ky * b.x + kz * c.x);
  }
}

// rho = -Re(ifft div) CHARGE_UNIT, as complex input of the next forward transform
__global__ void charge_density(double2* __restrict__ d, long long N) {
  const double f = -kChargeUnit / (double)N;
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x)
    d[s] = make_double2(d[s].x * f, 0.0);
}

__global__ void poisson_filter(double2* __restrict__ r, long long N, Grid3 g, double eps_r) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    double kx, ky, kz;
    kvec(s, g, kx, ky, kz);
    const double k2 = kx * kx + ky * ky + kz * kz;
    const double inv = k2 != 0.0 ? 1.0 / k2 : 0.0;
    const double f = kPoissonConst * inv / eps_r;
    r[s] = make_double2(r[s].x * f, r[s].y * f);
  }
}

__global__ void real_part(const double2* __restrict__ z, long long N, double* __restrict__ out) {
  const double invN = 1.0 / (double)N;
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x)
    out[s] = z[s].x * invN;
}

// ---- cuFFT plans: one per (shape, batch), no automatic allocation ------------------------------
struct Plan { cufftHandle h; size_t work; };
static std::mutex g_plan_mu;
static std::map<std::tuple<int, int, int, int, int, int>, Plan> g_plans;

static int get_plan(int device, int nx, int ny, int nz, int batch, cufftType type, Plan* out) {
  std::lock_guard<std::mutex> lk(g_plan_mu);
  const auto key = std::make_tuple(device, nx, ny, nz, batch, (int)type);
  auto it = g_plans.find(key);
  if (it != g_plans.end()) { *out = it->second; return QDKP_OK; }
  Plan p;
  if (cufftCreate(&p.h) != CUFFT_SUCCESS) { set_error("cufftCreate failed"); return QDKP_ERR_CUDA; }
  cufftSetAutoAllocation(p.h, 0);
  // real transforms: the half spectrum along z, packed
  int n[3] = {nx, ny, nz}, half[3] = {nx, ny, nz / 2 + 1};
  const int N = nx * ny * nz, M = nx * ny * (nz / 2 + 1);
  int* in = type == CUFFT_Z2D ? half : n;
  int* ou = type == CUFFT_D2Z ? half : n;
  if (cufftMakePlanMany(p.h, 3, n, in, 1, type == CUFFT_Z2D ? M : N, ou, 1, type == CUFFT_D2Z ? M : N,
                        type, batch, &p.work) != CUFFT_SUCCESS) {
    cufftDestroy(p.h);
    set_error("cufftMakePlanMany failed");
    return QDKP_ERR_CUDA;
  }
  g_plans[key] = p;
  *out = p;
  return QDKP_OK;
}

// exec(handle) on the plan, with the call's stream and work area
template <typename F>
static int run_plan(int device, int nx, int ny, int nz, int batch, cufftType type, void* work,
                    size_t work_bytes, cudaStream_t st, F exec) {
  Plan p;
  int rc = get_plan(device, nx, ny, nz, batch, type, &p);
  if (rc != QDKP_OK) return rc;
  if (p.work > work_bytes) { set_error("FFT work area larger than the workspace"); return QDKP_ERR_WORKSPACE; }
  std::lock_guard<std::mutex> lk(g_plan_mu);      // the plan's stream and work area are per call
  if (cufftSetStream(p.h, st) != CUFFT_SUCCESS || cufftSetWorkArea(p.h, work) != CUFFT_SUCCESS ||
      exec(p.h) != CUFFT_SUCCESS) {
    set_error("cuFFT execution failed");
    return QDKP_ERR_CUDA;
  }
  return QDKP_OK;
}

static int run_fft(int device, int nx, int ny, int nz, int batch, double2* data, int dir,
                   void* work, size_t work_bytes, cudaStream_t st) {
  auto* z = reinterpret_cast<cufftDoubleComplex*>(data);
  return run_plan(device, nx, ny, nz, batch, CUFFT_Z2Z, work, work_bytes, st,
                  [&](cufftHandle h) { return cufftExecZ2Z(h, z, z, dir); });
}

// three real components to and from their half spectra; the inverse overwrites its input
static int run_fft_d2z(int device, int nx, int ny, int nz, double* in, double2* out, void* work,
                       size_t work_bytes, cudaStream_t st) {
  return run_plan(device, nx, ny, nz, 3, CUFFT_D2Z, work, work_bytes, st, [&](cufftHandle h) {
    return cufftExecD2Z(h, in, reinterpret_cast<cufftDoubleComplex*>(out));
  });
}

static int run_fft_z2d(int device, int nx, int ny, int nz, double2* in, double* out, void* work,
                       size_t work_bytes, cudaStream_t st) {
  return run_plan(device, nx, ny, nz, 3, CUFFT_Z2D, work, work_bytes, st, [&](cufftHandle h) {
    return cufftExecZ2D(h, reinterpret_cast<cufftDoubleComplex*>(in), out);
  });
}

static size_t plan_work(int device, int nx, int ny, int nz, int batch, cufftType type = CUFFT_Z2Z) {
  Plan p;
  if (get_plan(device, nx, ny, nz, batch, type, &p) != QDKP_OK) return 0;
  return p.work;
}

static int grid_blocks(long long N) { return (int)std::min<long long>((N + 255) / 256, 148 * 16); }

static size_t al(size_t b) { return (b + 255) / 256 * 256; }


// ---- inhomogeneous FD elasticity (elasticity_fd.solve_strain_fd, elasticity_fd.py:211-419) ----
// Trilinear (Q1) hexahedral elements with 2x2x2 Gauss quadrature on the periodic cell:
// displacements u (3 x N, component-major) on nodes, materials (chi in {0, 1}) and strain on
// elements; element e spans the nodes e + c for the corners c in {0,1}^3 (corner index
// 4 cx + 2 cy + cz). The stiffness of a node p gathers, over the eight elements e = p - c_a,
// sum_{b,l} K_{mat(e)}[a,b,j,l] u_l[p + c_b - c_a] (element arrays computed on the host from C11,
// C12, C44 and h, elasticity_fd.py:90-153). Where the eight elements are of one material that is a
// 27-point stencil with eight distinct weights, since cubic constants on cubes leave it the
// symmetry of the cube: K_jj depends on |d_j| and the number of other offsets, K_jl (j != l) is
// sign(d_j d_l) times a weight of the third |offset|, and no other entry exists. Preconditioner: the
// exact inverse of the symbol of the volume-averaged homogeneous stencil, S(k) = sum_d Kavg_d
// exp(i k.d), real and symmetric by the same symmetry, per wavevector, zero where the reference's
// scale-free test calls it singular (elasticity_fd.py:179-241). It is formed once per solve: an
// iteration reads six doubles per wavevector (4 us at 96 x 96 x 72) where evaluating 27 phases and the
// adjugate took 87 us, and real transforms halve the FFTs.

struct FdStencil {
  double c[8];                  // K_jj at [3 |d_j| + others], K_jl at [6 + |d_third|]
};

struct FdArrays {
  double Km[8][8][3][3];        // matrix element stiffness
  double Kd[8][8][3][3];        // dot element stiffness
  double Wd[8][3];              // eigenstrain load shape of a dot element
  double G0[8][3];              // shape-function gradients at the element centre
  FdStencil m, d;               // the assembled stencils of either material
};

// scalars of a solve (device doubles)
enum { FD_FF = 0, FD_PAP, FD_RR, FD_RZ_USED, FD_HOST, FD_TRMAX = FD_HOST, FD_FRAC, FD_MEAN,
       FD_RZ = FD_MEAN + 3, FD_SCALARS = FD_RZ + 2 };
constexpr int kFdThreads = 256;
constexpr int kFdMaxBlocks = 148 * 16;

__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// Deterministic reduction of one value a thread over the grid (OP 0: sum, 1: max): a partial per
// block, and the block that arrives last reduces them in order of their index. Returns to that
// block's threads true, with out[0] written. Every thread of the block calls.
template <int OP>
__device__ __forceinline__ bool fd_reduce(double v, double* __restrict__ part, unsigned* __restrict__ ticket,
                                          double* __restrict__ out) {
  __shared__ double red[kFdThreads / 32];
  __shared__ bool last;
  auto op = [](double a, double b) { return OP == 1 ? fmax(a, b) : a + b; };
  auto block = [&](double w) {
    for (int o = 16; o > 0; o >>= 1) w = op(w, __shfl_xor_sync(0xffffffffu, w, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = w;
    __syncthreads();
    w = red[0];
    for (int i = 1; i < (int)blockDim.x >> 5; ++i) w = op(w, red[i]);
    return w;
  };
  v = block(v);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v;
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double w = OP == 1 ? -INFINITY : 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) w = op(w, __ldcg(part + i));
  w = block(w);
  if (threadIdx.x == 0) out[0] = w;
  return true;
}

// nodes of a block of fd_codes and fd_list: contiguous, so that the list is in order of the node
__host__ __device__ __forceinline__ int fd_chunk(int N, int blocks) {
  return ((N + blocks - 1) / blocks + kFdThreads - 1) / kFdThreads * kFdThreads;
}

__device__ __forceinline__ bool fd_mixed(int code) { return code != 0 && code != 255; }

// code[p]: bit a set where element p - c_a is dot; the nodes of both materials in each block's chunk;
// the dot's volume fraction
__global__ void __launch_bounds__(kFdThreads)
fd_codes(const unsigned char* __restrict__ chi, Grid3 g, unsigned char* __restrict__ code,
         int* __restrict__ counts, double* __restrict__ part, unsigned* __restrict__ ticket,
         double* __restrict__ sc) {
  const int N = g.nx * g.ny * g.nz, chunk = fd_chunk(N, gridDim.x);
  const long long end = min((long long)N, (blockIdx.x + 1LL) * chunk);
  double dot = 0.0;
  int mixed = 0;
  for (long long q = (long long)blockIdx.x * chunk + threadIdx.x; q < end; q += blockDim.x) {
    const int p = (int)q, t = p / g.nz, z = p - t * g.nz, x = t / g.ny, y = t - x * g.ny;
    int c = 0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int ex = wrapi(x - (a >> 2), g.nx), ey = wrapi(y - ((a >> 1) & 1), g.ny), ez = wrapi(z - (a & 1), g.nz);
      if (chi[(ex * g.ny + ey) * g.nz + ez]) c |= 1 << a;
    }
    code[p] = (unsigned char)c;
    dot += c & 1;
    mixed += fd_mixed(c);
  }
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  atomicAdd(&total, mixed);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
  if (fd_reduce<0>(dot, part, ticket, sc + FD_FRAC) && threadIdx.x == 0) sc[FD_FRAC] /= (double)N;
}

// the nodes of both materials in order, and their number in *nmixed; same grid as fd_codes
__global__ void __launch_bounds__(kFdThreads)
fd_list(const unsigned char* __restrict__ code, int N, const int* __restrict__ counts, int* __restrict__ list,
        int* __restrict__ nmixed) {
  __shared__ int base;
  __shared__ int warps[kFdThreads / 32];
  const int chunk = fd_chunk(N, gridDim.x), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long first = (long long)blockIdx.x * chunk, end = min((long long)N, first + chunk);
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  int before = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += blockDim.x) before += counts[b];
  if (before) atomicAdd(&base, before);
  __syncthreads();
  int at = base;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *nmixed = at + counts[blockIdx.x];
  if (counts[blockIdx.x] == 0) return;
  for (long long q0 = first; q0 < end; q0 += blockDim.x) {
    const long long q = q0 + threadIdx.x;
    const bool mine = q < end && fd_mixed(code[q]);
    const unsigned vote = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) warps[warp] = __popc(vote);
    __syncthreads();
    int mid = at;
    for (int w = 0; w < kFdThreads / 32; ++w) {
      mid += w < warp ? warps[w] : 0;
      at += warps[w];
    }
    if (mine) list[mid + __popc(vote & ((1u << lane) - 1u))] = (int)q;
    __syncthreads();
  }
}

// F = K u on the nodes and u.F. A thread marches along x over kFdMarch nodes of one (y, z) and reads
// each plane's nine neighbours once (27 loads a node and plane instead of 81): a plane at offset
// dx of the output enters through A (dx = 0), and through a part even and a part odd in dx
// (dx = +-1), nine sums that the three outputs share. They are formed with the matrix's weights
// and, in warps that meet nodes wholly inside the dot, with the dot's too. Nodes whose eight
// elements are of both materials are listed once per solve and done through the element arrays by
// eight lanes each, a lane an element, spread over all blocks (36 us where each block did its own). 82 us at 96 x 96 x 72 with the element arrays read from shared
// memory for every node, 52 us with a thread per node on the 27-point stencil, 28 us so (inputs not in L2).
constexpr int kFdApplyThreads = 128;
constexpr int kFdApplyBlocks = 4 * 148;  // resident at once
constexpr int kFdMarchMin = 4, kFdMarchMax = 16;

// plane sums of the uniform stencil: A[j] for dx = 0, E[j] even and O[j] odd in dx
struct FdPlane {
  double x00, x01, x02;                  // u_x: centre row and column, edges, corners
  double y00, y01, y10, y11;             // u_y: [own y offset][z offset]
  double z00, z01, z10, z11;             // u_z: [own z offset][y offset]
  double xy0, xy1, yx0, yx1;             // odd in y, of u_y and of u_x; [z offset]
  double xz0, xz1, zx0, zx1;             // odd in z, of u_z and of u_x; [y offset]
  double yz, zy;                         // odd in y and z, of u_z and of u_y
};

__device__ __forceinline__ void fd_plane_weights(const FdPlane& s, const FdStencil& S, double (&A)[3],
                                                 double (&E)[3], double (&O)[3]) {
  const double* c = S.c;
  const double o0 = c[6], o1 = c[7];
  A[0] = fma(c[0], s.x00, fma(c[1], s.x01, c[2] * s.x02));
  E[0] = fma(c[3], s.x00, fma(c[4], s.x01, c[5] * s.x02));
  A[1] = fma(c[0], s.y00, fma(c[1], s.y01, fma(c[3], s.y10, fma(c[4], s.y11, o0 * s.yz))));
  E[1] = fma(c[1], s.y00, fma(c[2], s.y01, fma(c[4], s.y10, fma(c[5], s.y11, o1 * s.yz))));
  A[2] = fma(c[0], s.z00, fma(c[1], s.z01, fma(c[3], s.z10, fma(c[4], s.z11, o0 * s.zy))));
  E[2] = fma(c[1], s.z00, fma(c[2], s.z01, fma(c[4], s.z10, fma(c[5], s.z11, o1 * s.zy))));
  O[0] = fma(o0, s.xy0 + s.xz0, o1 * (s.xy1 + s.xz1));
  O[1] = fma(o0, s.yx0, o1 * s.yx1);
  O[2] = fma(o0, s.zx0, o1 * s.zx1);
}

__global__ void __launch_bounds__(kFdApplyThreads, 4)
fd_apply(const double* __restrict__ u, const unsigned char* __restrict__ code, Grid3 g, int march,
         const int* __restrict__ list, const int* __restrict__ nmixed, const FdArrays* __restrict__ arr,
         double* __restrict__ f, double* __restrict__ part,
         unsigned* __restrict__ ticket, double* __restrict__ sc) {
  __shared__ double sK[2][8][8][3][3];
  const int N = g.nx * g.ny * g.nz, nyz = g.ny * g.nz;
  const int columns = (nyz + kFdApplyThreads - 1) / kFdApplyThreads;
  const int tasks = columns * ((g.nx + march - 1) / march);
  FdStencil Sm;
#pragma unroll
  for (int i = 0; i < 8; ++i) Sm.c[i] = arr->m.c[i];
  double dot = 0.0;
  for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
    const int yz = (task % columns) * kFdApplyThreads + threadIdx.x;
    const int x0 = (task / columns) * march, nxs = min(march, g.nx - x0);
    const bool live = yz < nyz;
    const int y = live ? yz / g.nz : 0, z = live ? yz - y * g.nz : 0;
    unsigned inner = 0, mixed = 0;                          // bit per x
    if (live)
      for (int i = 0; i < nxs; ++i) {
        const int cd = code[(x0 + i) * nyz + yz];
        mixed |= fd_mixed(cd) ? 1u << i : 0u;
        inner |= cd == 255 ? 1u << i : 0u;
      }
    const bool dots = __any_sync(0xffffffffu, inner != 0);
    if (live) {
      const int dzm = z ? -1 : g.nz - 1, dzp = z + 1 < g.nz ? 1 : 1 - g.nz;
      const int dym = (y ? -1 : g.ny - 1) * g.nz, dyp = (y + 1 < g.ny ? 1 : 1 - g.ny) * g.nz;
      double am[3] = {0, 0, 0}, bm[3] = {0, 0, 0}, ad[3] = {0, 0, 0}, bd[3] = {0, 0, 0};
      double uc[3] = {0, 0, 0};                             // u at the output's node
      for (int i = -1; i <= nxs; ++i) {
        const double* ux = u + wrapi(x0 + i, g.nx) * nyz + yz;
        const double *uy = ux + N, *uz = uy + N;
        FdPlane s;
        double cx, cy, cz;
        {
          const double a0 = ux[dym + dzm], a1 = ux[dym], a2 = ux[dym + dzp];
          const double b0 = ux[dzm], b1 = ux[0], b2 = ux[dzp];
          const double c0 = ux[dyp + dzm], c1 = ux[dyp], c2 = ux[dyp + dzp];
          cx = b1;
          s.x00 = b1; s.x01 = (b0 + b2) + (a1 + c1); s.x02 = (a0 + a2) + (c0 + c2);
          s.yx0 = c1 - a1; s.yx1 = (c0 + c2) - (a0 + a2);
          s.zx0 = b2 - b0; s.zx1 = (a2 - a0) + (c2 - c0);
        }
        {
          const double a0 = uy[dym + dzm], a1 = uy[dym], a2 = uy[dym + dzp];
          const double b0 = uy[dzm], b1 = uy[0], b2 = uy[dzp];
          const double c0 = uy[dyp + dzm], c1 = uy[dyp], c2 = uy[dyp + dzp];
          cy = b1;
          s.y00 = b1; s.y01 = b0 + b2; s.y10 = a1 + c1; s.y11 = (a0 + a2) + (c0 + c2);
          s.xy0 = c1 - a1; s.xy1 = (c0 + c2) - (a0 + a2);
          s.zy = (c2 - c0) - (a2 - a0);
        }
        {
          const double a0 = uz[dym + dzm], a1 = uz[dym], a2 = uz[dym + dzp];
          const double b0 = uz[dzm], b1 = uz[0], b2 = uz[dzp];
          const double c0 = uz[dyp + dzm], c1 = uz[dyp], c2 = uz[dyp + dzp];
          cz = b1;
          s.z00 = b1; s.z01 = a1 + c1; s.z10 = b0 + b2; s.z11 = (a0 + a2) + (c0 + c2);
          s.xz0 = b2 - b0; s.xz1 = (a2 - a0) + (c2 - c0);
          s.yz = (c2 - c0) - (a2 - a0);
        }
        double A[3], E[3], O[3], om[3], od[3] = {0, 0, 0};
        fd_plane_weights(s, Sm, A, E, O);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          om[j] = am[j] + (E[j] + O[j]);
          am[j] = A[j] + bm[j];
          bm[j] = E[j] - O[j];
        }
        if (dots) {
          fd_plane_weights(s, arr->d, A, E, O);
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            od[j] = ad[j] + (E[j] + O[j]);
            ad[j] = A[j] + bd[j];
            bd[j] = E[j] - O[j];
          }
        }
        if (i >= 1 && !((mixed >> (i - 1)) & 1)) {
          const bool in = (inner >> (i - 1)) & 1;
          const int p = (x0 + i - 1) * nyz + yz;
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const double v = in ? od[j] : om[j];
            f[j * (long long)N + p] = v;
            dot = fma(uc[j], v, dot);
          }
        }
        uc[0] = cx; uc[1] = cy; uc[2] = cz;
      }
    }
  }
  const int total = *nmixed;
  if (blockIdx.x * (kFdApplyThreads / 8) < total) {
    for (int t = threadIdx.x; t < 2 * 576; t += blockDim.x)
      (&sK[0][0][0][0][0])[t] = t < 576 ? (&arr->Km[0][0][0][0])[t] : (&arr->Kd[0][0][0][0])[t - 576];
    __syncthreads();
    for (int i0 = blockIdx.x * (kFdApplyThreads / 8); i0 < total; i0 += gridDim.x * (kFdApplyThreads / 8)) {
      const int i = i0 + (threadIdx.x >> 3), a = threadIdx.x & 7;
      double f0 = 0.0, f1 = 0.0, f2 = 0.0;
      const int q0 = list[min(i, total - 1)];
      const int qx = q0 / nyz, r = q0 - qx * nyz, qy = r / g.nz, qz = r - qy * g.nz;
      const double (*K)[3][3] = sK[(code[q0] >> a) & 1][a];
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const int ox = (b >> 2) - (a >> 2), oy = ((b >> 1) & 1) - ((a >> 1) & 1), oz = (b & 1) - (a & 1);
        const double* uq = u + wrapi(qx + ox, g.nx) * nyz + wrapi(qy + oy, g.ny) * g.nz + wrapi(qz + oz, g.nz);
        const double u0 = uq[0], u1 = uq[N], u2 = uq[2 * (long long)N];
        f0 += K[b][0][0] * u0 + K[b][0][1] * u1 + K[b][0][2] * u2;
        f1 += K[b][1][0] * u0 + K[b][1][1] * u1 + K[b][1][2] * u2;
        f2 += K[b][2][0] * u0 + K[b][2][1] * u1 + K[b][2][2] * u2;
      }
      for (int o = 1; o < 8; o <<= 1) {
        f0 += __shfl_xor_sync(0xffffffffu, f0, o);
        f1 += __shfl_xor_sync(0xffffffffu, f1, o);
        f2 += __shfl_xor_sync(0xffffffffu, f2, o);
      }
      if (a == 0 && i < total) {
        const long long q = q0, n = N;
        f[q] = f0; f[n + q] = f1; f[2 * n + q] = f2;
        dot = fma(u[q], f0, fma(u[n + q], f1, fma(u[2 * n + q], f2, dot)));
      }
    }
  }
  fd_reduce<0>(dot, part, ticket, sc + FD_PAP);
}

// the eigenstrain load F_j[p] = sum_a W_d[a, j] bulk[p - c_a], bulk = eps_T (C11 + 2 C12)_dot chi,
// and its component means
__global__ void __launch_bounds__(kFdThreads)
fd_load(const unsigned char* __restrict__ code, long long N, const FdArrays* __restrict__ arr,
        double bulk, double* __restrict__ f, double* __restrict__ part, unsigned* __restrict__ ticket,
        double* __restrict__ sc) {
  double s[3] = {0.0, 0.0, 0.0};
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N;
       p += (long long)gridDim.x * blockDim.x) {
    const int cd = code[p];
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    for (int a = 0; a < 8; ++a) {
      if (!((cd >> a) & 1)) continue;
      f0 += arr->Wd[a][0] * bulk; f1 += arr->Wd[a][1] * bulk; f2 += arr->Wd[a][2] * bulk;
    }
    f[p] = f0; f[N + p] = f1; f[2 * N + p] = f2;
    s[0] += f0; s[1] += f1; s[2] += f2;
  }
  for (int c = 0; c < 3; ++c)
    if (fd_reduce<0>(s[c], part + c * kFdMaxBlocks, ticket + c, sc + FD_MEAN + c) && threadIdx.x == 0)
      sc[FD_MEAN + c] /= (double)N;
}

// R = F minus its means (in place), U = 0, ||R||^2
__global__ void __launch_bounds__(kFdThreads)
fd_start(double* __restrict__ r, double* __restrict__ u, long long N, double* __restrict__ part,
         unsigned* __restrict__ ticket, double* __restrict__ sc) {
  double s = 0.0;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N;
       p += (long long)gridDim.x * blockDim.x)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double v = r[c * N + p] - sc[FD_MEAN + c];
      r[c * N + p] = v;
      u[c * N + p] = 0.0;
      s = fma(v, v, s);
    }
  fd_reduce<0>(s, part, ticket, sc + FD_FF);
}

// S(k) of the averaged stencil (its six upper entries) over the half spectrum, k = 2 pi fftfreq per
// axis in grid units, component-major; the largest tr(S) / 3
__global__ void __launch_bounds__(kFdThreads)
fd_symbol(Grid3 g, int hz, const FdArrays* __restrict__ arr, double* __restrict__ tab,
          double* __restrict__ part, unsigned* __restrict__ ticket, double* __restrict__ sc) {
  const long long M = (long long)g.nx * g.ny * hz;
  const double frac = sc[FD_FRAC];
  double w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = arr->m.c[i] + frac * (arr->d.c[i] - arr->m.c[i]);
  double tmax = -INFINITY;
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < M;
       s += (long long)gridDim.x * blockDim.x) {
    const int t = (int)s / hz, iz = (int)s - t * hz, ix = t / g.ny, iy = t - ix * g.ny;
    double sx, cx, sy, cy, sz, cz;
    sincos(kcomp(ix, g.nx, 1.0), &sx, &cx);
    sincos(kcomp(iy, g.ny, 1.0), &sy, &cy);
    sincos(kcomp(iz, g.nz, 1.0), &sz, &cz);
    auto diag = [&](double a, double b, double c) {         // 2 cos of the own and the other axes
      return (w[0] + w[1] * (b + c) + w[2] * b * c) + a * (w[3] + w[4] * (b + c) + w[5] * b * c);
    };
    const double X = 2.0 * cx, Y = 2.0 * cy, Z = 2.0 * cz;
    const double xx = diag(X, Y, Z), yy = diag(Y, X, Z), zz = diag(Z, X, Y);
    tab[s] = xx;
    tab[M + s] = -4.0 * sx * sy * (w[6] + w[7] * Z);
    tab[2 * M + s] = -4.0 * sx * sz * (w[6] + w[7] * Y);
    tab[3 * M + s] = yy;
    tab[4 * M + s] = -4.0 * sy * sz * (w[6] + w[7] * X);
    tab[5 * M + s] = zz;
    tmax = fmax(tmax, (xx + yy + zz) / 3.0);
  }
  fd_reduce<1>(tmax, part, ticket, sc + FD_TRMAX);
}

// entries of the half spectrum that stand for two wavevectors
__device__ __forceinline__ bool fd_paired(long long s, int nz, int hz) {
  const int iz = (int)s % hz;
  return iz != 0 && 2 * iz != nz;
}

// S -> S^-1 / N in place, zero where singular; counts the dropped wavevectors of the full spectrum
__global__ void __launch_bounds__(kFdThreads)
fd_invert(double* __restrict__ tab, long long M, int nz, int hz, double invN, const double* __restrict__ sc,
          unsigned long long* __restrict__ count) {
  const double tmax = sc[FD_TRMAX];
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < M;
       s += (long long)gridDim.x * blockDim.x) {
    const double a = tab[s], b = tab[M + s], c = tab[2 * M + s], d = tab[3 * M + s], e = tab[4 * M + s];
    const double f = tab[5 * M + s];
    const double i00 = d * f - e * e, i01 = c * e - b * f, i02 = b * e - c * d;
    const double i11 = a * f - c * c, i12 = c * b - a * e, i22 = a * d - b * b;
    const double det = a * i00 + b * i01 + c * i02;
    const double tr = (a + d + f) / 3.0, t = fmax(tr, 0.0);
    const bool good = tr > 1e-12 * tmax && fabs(det) > 1e-9 * t * t * t;
    const double id = good ? invN / det : 0.0;
    tab[s] = i00 * id; tab[M + s] = i01 * id; tab[2 * M + s] = i02 * id;
    tab[3 * M + s] = i11 * id; tab[4 * M + s] = i12 * id; tab[5 * M + s] = i22 * id;
    if (!good) atomicAdd(count, fd_paired(s, nz, hz) ? 2ULL : 1ULL);
  }
}

// The spectra of r's three components (batch-major) times S^-1 / N, in place, and r.z = sum over the
// full spectrum of conj(R) Z
__global__ void __launch_bounds__(kFdThreads)
fd_precondition(double2* __restrict__ Rk, const double* __restrict__ tab, long long M, int nz, int hz,
                double* __restrict__ part, unsigned* __restrict__ ticket, double* __restrict__ rz) {
  double dot = 0.0;
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < M;
       s += (long long)gridDim.x * blockDim.x) {
    const double i00 = tab[s], i01 = tab[M + s], i02 = tab[2 * M + s];
    const double i11 = tab[3 * M + s], i12 = tab[4 * M + s], i22 = tab[5 * M + s];
    const double2 a = Rk[s], b = Rk[M + s], c = Rk[2 * M + s];
    const double2 x = make_double2(i00 * a.x + i01 * b.x + i02 * c.x, i00 * a.y + i01 * b.y + i02 * c.y);
    const double2 y = make_double2(i01 * a.x + i11 * b.x + i12 * c.x, i01 * a.y + i11 * b.y + i12 * c.y);
    const double2 z = make_double2(i02 * a.x + i12 * b.x + i22 * c.x, i02 * a.y + i12 * b.y + i22 * c.y);
    Rk[s] = x; Rk[M + s] = y; Rk[2 * M + s] = z;
    const double v = a.x * x.x + a.y * x.y + b.x * y.x + b.y * y.y + c.x * z.x + c.y * z.y;
    dot += fd_paired(s, nz, hz) ? 2.0 * v : v;
  }
  fd_reduce<0>(dot, part, ticket, rz);
}

// x += alpha p and r -= alpha q with alpha = rz / p.q, and ||r||^2; no step without positive rz and
// curvature (the host stops there)
__global__ void __launch_bounds__(kFdThreads)
fd_cg_step(double* __restrict__ x, const double* __restrict__ p, double* __restrict__ r,
           const double* __restrict__ q, const double* __restrict__ rz, long long n3,
           double* __restrict__ part, unsigned* __restrict__ ticket, double* __restrict__ sc) {
  const double num = *rz, den = sc[FD_PAP];
  const bool step = num > 0.0 && den > 0.0;
  const double alpha = step ? num / den : 0.0;
  double s = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3; i += stride) {
    double v = r[i];
    if (step) {
      x[i] = fma(alpha, p[i], x[i]);
      v = fma(-alpha, q[i], v);
      r[i] = v;
    }
    s = fma(v, v, s);
  }
  if (fd_reduce<0>(s, part, ticket, sc + FD_RR) && threadIdx.x == 0) sc[FD_RZ_USED] = num;
}

// p = z + (rz_new / rz_old) p; rz_old NULL: p = z
__global__ void __launch_bounds__(kFdThreads)
fd_direction(double* __restrict__ p, const double* __restrict__ z, const double* __restrict__ rz_new,
             const double* __restrict__ rz_old, long long n3) {
  const double beta = rz_old ? *rz_new / *rz_old : 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3; i += stride)
    p[i] = rz_old ? fma(beta, p[i], z[i]) : z[i];
}

// elastic strain at the element centres (u's mean drops out): grad_ij = sum_n G0[n, i] u_j[e + c_n]; the diagonal
// minus eps_T chi (elasticity_fd.py:343-362); out (6 x N): exx eyy ezz exy eyz ezx, and the
// total strain (optional) without the eigenstrain term
__global__ void fd_strain(const double* __restrict__ u, const unsigned char* __restrict__ chi, Grid3 g,
                          const FdArrays* __restrict__ arr, double eps_T, double* __restrict__ out,
                          double* __restrict__ total) {
  const long long N = (long long)g.nx * g.ny * g.nz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < N;
       e += (long long)gridDim.x * blockDim.x) {
    const int z = (int)(e % g.nz);
    const long long t = e / g.nz;
    const int y = (int)(t % g.ny), x = (int)(t / g.ny);
    double gr[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int n = 0; n < 8; ++n) {
      const long long q = ((long long)wrapi(x + (n >> 2), g.nx) * g.ny + wrapi(y + ((n >> 1) & 1), g.ny)) * g.nz
                          + wrapi(z + (n & 1), g.nz);
      const double uj[3] = {u[q], u[N + q], u[2 * N + q]};
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) gr[i][j] = fma(arr->G0[n][i], uj[j], gr[i][j]);
    }
    const double tot[6] = {gr[0][0], gr[1][1], gr[2][2], 0.5 * (gr[0][1] + gr[1][0]),
                           0.5 * (gr[1][2] + gr[2][1]), 0.5 * (gr[2][0] + gr[0][2])};
    const double off = chi[e] ? eps_T : 0.0;
    for (int c = 0; c < 6; ++c) {
      out[c * N + e] = tot[c] - (c < 3 ? off : 0.0);
      if (total) total[c * N + e] = tot[c];
    }
  }
}


// ---- host: element arrays (elasticity_fd.py:90-153) and the PCG driver (elasticity_fd.py:366-419)
// dN_n/dx_d at the local point xi of the cube [-1, 1]^3 of side h, N_n = prod (1 + s_nd xi_d) / 2
static void fd_shape_gradients(const double xi[3], double h, double G[8][3]) {
  for (int n = 0; n < 8; ++n) {
    const double sn[3] = {(n >> 2) ? 1.0 : -1.0, ((n >> 1) & 1) ? 1.0 : -1.0, (n & 1) ? 1.0 : -1.0};
    for (int d = 0; d < 3; ++d) {
      double v = 0.5 * sn[d];
      for (int e = 0; e < 3; ++e)
        if (e != d) v *= 0.5 * (1.0 + sn[e] * xi[e]);
      G[n][d] = v * (2.0 / h);
    }
  }
}

// K[a][b][j][l] = (h/2)^3 sum_gauss sum_ik C_ijkl G[a][i] G[b][k] for a cubic C, and W[a][j]
static void fd_element(double C11, double C12, double C44, double h, double K[8][8][3][3],
                       double W[8][3]) {
  // C_ijkl = C12 d_ij d_kl + C44 (d_ik d_jl + d_il d_jk) + Ca (all equal)
  const double w = (h / 2.0) * (h / 2.0) * (h / 2.0), Ca = C11 - C12 - 2.0 * C44;
  std::memset(K, 0, sizeof(double) * 576);
  std::memset(W, 0, sizeof(double) * 24);
  for (int gq = 0; gq < 8; ++gq) {
    const double r = 1.0 / std::sqrt(3.0);
    const double xi[3] = {(gq >> 2) ? r : -r, ((gq >> 1) & 1) ? r : -r, (gq & 1) ? r : -r};
    double G[8][3];
    fd_shape_gradients(xi, h, G);
    for (int a = 0; a < 8; ++a) {
      for (int j = 0; j < 3; ++j) W[a][j] += w * G[a][j];
      for (int b = 0; b < 8; ++b) {
        const double gg = G[a][0] * G[b][0] + G[a][1] * G[b][1] + G[a][2] * G[b][2];
        for (int j = 0; j < 3; ++j)
          for (int l = 0; l < 3; ++l) {
            double v = C12 * G[a][j] * G[b][l] + C44 * G[a][l] * G[b][j];
            if (j == l) v += C44 * gg + Ca * G[a][j] * G[b][j];
            K[a][b][j][l] += w * v;
          }
      }
    }
  }
}

// the eight weights of the stencil that the element arrays assemble to in one material
static void fd_stencil(const double K[8][8][3][3], FdStencil& S) {
  double k27[27][3][3] = {};
  for (int a = 0; a < 8; ++a)
    for (int b = 0; b < 8; ++b) {
      const int dx = (b >> 2) - (a >> 2), dy = ((b >> 1) & 1) - ((a >> 1) & 1), dz = (b & 1) - (a & 1);
      for (int j = 0; j < 3; ++j)
        for (int l = 0; l < 3; ++l) k27[(dx + 1) * 9 + (dy + 1) * 3 + (dz + 1)][j][l] += K[a][b][j][l];
    }
  auto at = [&](int dx, int dy, int dz) { return k27[(dx + 1) * 9 + (dy + 1) * 3 + (dz + 1)]; };
  for (int own = 0; own < 2; ++own)
    for (int others = 0; others < 3; ++others)
      S.c[3 * own + others] = at(own, others > 0, others > 1)[0][0];
  S.c[6] = at(1, 1, 0)[0][1];
  S.c[7] = at(1, 1, 1)[0][1];
}

static int fd_blocks(long long n) { return (int)std::min<long long>((n + kFdThreads - 1) / kFdThreads, kFdMaxBlocks); }

// a stream and an event for the host's reads beside the solve
struct FdSide {
  cudaStream_t st = nullptr;
  cudaEvent_t ev = nullptr;
  ~FdSide() {
    if (st) cudaStreamDestroy(st);
    if (ev) cudaEventDestroy(ev);
  }
};

}  // namespace qdkp

using namespace qdkp;

extern "C" {

size_t qdkp_fd_strain_workspace_size(int nx, int ny, int nz) {
  if (nx < 1 || ny < 1 || nz < 1) return 0;
  const long long N = (long long)nx * ny * nz, M = (long long)nx * ny * (nz / 2 + 1);
  int dev = 0;
  cudaGetDevice(&dev);
  const size_t fw = plan_work(dev, nx, ny, nz, 3, CUFFT_D2Z), bw = plan_work(dev, nx, ny, nz, 3, CUFFT_Z2D);
  return 5 * al(3 * N * sizeof(double)) + al(3 * M * sizeof(double2)) + al(6 * M * sizeof(double)) + al(N)
         + al(N * sizeof(int)) + al((kFdMaxBlocks + 1) * sizeof(int))
         + al(sizeof(FdArrays)) + al(3 * kFdMaxBlocks * sizeof(double)) + al(FD_SCALARS * sizeof(double))
         + al(sizeof(unsigned long long) + 4 * sizeof(unsigned)) + al(std::max(fw, bw)) + 256;
}

int qdkp_fd_strain(int nx, int ny, int nz, double h, const unsigned char* mask, double eps_star,
                   const double* C_dot, const double* C_matrix, double tol, int maxiter,
                   double* strain, double* total, qdkp_fd_info* info, void* ws, size_t ws_bytes,
                   void* stream) {
  QDKP_CHECK_ARG(nx >= 1 && ny >= 1 && nz >= 1 && h > 0.0, "grid extents must be >= 1, h > 0");
  QDKP_CHECK_ARG(mask && strain && C_dot && C_matrix && info, "NULL argument");
  QDKP_CHECK_ARG(tol > 0.0 && maxiter >= 1, "tol must be > 0 and maxiter >= 1");
  const long long N = (long long)nx * ny * nz;
  QDKP_CHECK_ARG(3 * N < (1LL << 31), "grid too large for one transform");
  const size_t need = qdkp_fd_strain_workspace_size(nx, ny, nz);
  if (!ws || ws_bytes < need || need == 0) {
    set_error("qdkp_fd_strain: workspace too small (see qdkp_fd_strain_workspace_size)");
    return QDKP_ERR_WORKSPACE;
  }
  int dev = 0;
  QDKP_CUDA_TRY(cudaGetDevice(&dev));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const Grid3 g{nx, ny, nz, h};
  const int hz = nz / 2 + 1;
  const long long n3 = 3 * N, M = (long long)nx * ny * hz;
  char* p = static_cast<char*>(ws);
  auto take = [&](size_t b) { char* r = p; p += al(b); return r; };
  double* U = reinterpret_cast<double*>(take(n3 * sizeof(double)));
  double* R = reinterpret_cast<double*>(take(n3 * sizeof(double)));
  double* Z = reinterpret_cast<double*>(take(n3 * sizeof(double)));
  double* P = reinterpret_cast<double*>(take(n3 * sizeof(double)));
  double* AP = reinterpret_cast<double*>(take(n3 * sizeof(double)));
  double2* Ck = reinterpret_cast<double2*>(take(3 * M * sizeof(double2)));
  double* tab = reinterpret_cast<double*>(take(6 * M * sizeof(double)));
  unsigned char* code = reinterpret_cast<unsigned char*>(take(N));
  int* list = reinterpret_cast<int*>(take(N * sizeof(int)));
  int* counts = reinterpret_cast<int*>(take((kFdMaxBlocks + 1) * sizeof(int)));
  int* nmixed = counts + kFdMaxBlocks;
  FdArrays* dArr = reinterpret_cast<FdArrays*>(take(sizeof(FdArrays)));
  double* part = reinterpret_cast<double*>(take(3 * kFdMaxBlocks * sizeof(double)));
  double* sc = reinterpret_cast<double*>(take(FD_SCALARS * sizeof(double)));
  unsigned long long* dropped = reinterpret_cast<unsigned long long*>(take(sizeof(unsigned long long) + 4 * sizeof(unsigned)));
  unsigned* ticket = reinterpret_cast<unsigned*>(dropped + 1);
  char* work = p;
  const size_t work_bytes = ws_bytes - (size_t)(p - static_cast<char*>(ws));
  const int B = fd_blocks(N), BM = fd_blocks(M), B3 = fd_blocks((n3 + 3) / 4);
  // the shortest march that leaves the blocks one wave: each march reads two planes more than it writes
  const long long columns = ((long long)ny * nz + kFdApplyThreads - 1) / kFdApplyThreads;
  int march = kFdMarchMin;
  while (march < kFdMarchMax && columns * ((nx + march - 1) / march) > kFdApplyBlocks) ++march;
  const int BA = (int)std::min<long long>(columns * ((nx + march - 1) / march), kFdMaxBlocks);
  FdSide side;
  QDKP_CUDA_TRY(cudaStreamCreateWithFlags(&side.st, cudaStreamNonBlocking));
  QDKP_CUDA_TRY(cudaEventCreateWithFlags(&side.ev, cudaEventDisableTiming));
  QDKP_CUDA_TRY(cudaMemsetAsync(dropped, 0, sizeof(unsigned long long) + 4 * sizeof(unsigned), st));
  fd_codes<<<B, kFdThreads, 0, st>>>(mask, g, code, counts, part, ticket, sc);
  fd_list<<<B, kFdThreads, 0, st>>>(code, (int)N, counts, list, nmixed);
  count_launch(2);
  // ---- element arrays
  FdArrays h_arr;
  double Wm[8][3];
  fd_element(C_matrix[0], C_matrix[1], C_matrix[2], h, h_arr.Km, Wm);
  fd_element(C_dot[0], C_dot[1], C_dot[2], h, h_arr.Kd, h_arr.Wd);
  fd_stencil(h_arr.Km, h_arr.m);
  fd_stencil(h_arr.Kd, h_arr.d);
  {
    const double xi0[3] = {0.0, 0.0, 0.0};
    fd_shape_gradients(xi0, h, h_arr.G0);
  }
  QDKP_CUDA_TRY(cudaMemcpyAsync(dArr, &h_arr, sizeof(FdArrays), cudaMemcpyHostToDevice, st));
  // ---- preconditioner: the materials averaged by the dot's volume fraction
  fd_symbol<<<BM, kFdThreads, 0, st>>>(g, hz, dArr, tab, part, ticket, sc);
  fd_invert<<<BM, kFdThreads, 0, st>>>(tab, M, nz, hz, 1.0 / (double)N, sc, dropped);
  // ---- load, projected: R = F, U = 0
  const double eps_T = -eps_star;
  fd_load<<<B, kFdThreads, 0, st>>>(code, N, dArr, eps_T * (C_dot[0] + 2.0 * C_dot[1]), R, part, ticket, sc);
  fd_start<<<B, kFdThreads, 0, st>>>(R, U, N, part, ticket, sc);
  count_launch(4);
  QDKP_CUDA_TRY(cudaGetLastError());
  int rc;
  // Z = M R and rz = R.Z, then the next direction P from rz_old's
  auto direction = [&](double* rz, const double* rz_old) -> int {
    int r2 = run_fft_d2z(dev, nx, ny, nz, R, Ck, work, work_bytes, st);
    if (r2 != QDKP_OK) return r2;
    fd_precondition<<<BM, kFdThreads, 0, st>>>(Ck, tab, M, nz, hz, part, ticket, rz);
    if ((r2 = run_fft_z2d(dev, nx, ny, nz, Ck, Z, work, work_bytes, st)) != QDKP_OK) return r2;
    fd_direction<<<B3, kFdThreads, 0, st>>>(P, Z, rz, rz_old, n3);
    count_launch(2);
    QDKP_CUDA_TRY(cudaGetLastError());
    return QDKP_OK;
  };
  if ((rc = direction(sc + FD_RZ, nullptr)) != QDKP_OK) return rc;
  double hs[FD_HOST], fnorm = 0.0, rel = 1.0;
  int it = 0, breakdown = 0;
  for (it = 1; it <= maxiter; ++it) {
    double* rz = sc + FD_RZ + (it + 1) % 2;                 // R.Z of the current direction
    double* rz_new = sc + FD_RZ + it % 2;
    fd_apply<<<BA, kFdApplyThreads, 0, st>>>(P, code, g, march, list, nmixed, dArr, AP, part, ticket, sc);
    fd_cg_step<<<B3, kFdThreads, 0, st>>>(U, P, R, AP, rz, n3, part, ticket, sc);
    count_launch(2);
    QDKP_CUDA_TRY(cudaEventRecord(side.ev, st));
    if ((rc = direction(rz_new, rz)) != QDKP_OK) return rc;
    // the step's scalars, read while the GPU forms the next direction
    QDKP_CUDA_TRY(cudaStreamWaitEvent(side.st, side.ev, 0));
    QDKP_CUDA_TRY(cudaMemcpyAsync(hs, sc, sizeof(hs), cudaMemcpyDeviceToHost, side.st));
    QDKP_CUDA_TRY(cudaStreamSynchronize(side.st));
    fnorm = std::sqrt(hs[FD_FF]);
    if (fnorm == 0.0) { it = 0; rel = 0.0; break; }
    if (!(hs[FD_RZ_USED] > 0.0)) {                          // preconditioner not positive definite
      breakdown = it == 1 ? 1 : 3;
      --it;
      break;
    }
    if (!(hs[FD_PAP] > 0.0)) { breakdown = 2; break; }      // non-positive curvature (step skipped)
    rel = std::sqrt(hs[FD_RR]) / fnorm;
    if (rel < tol) break;
  }
  if (it > maxiter) {
    it = maxiter;
    double rz_last;
    QDKP_CUDA_TRY(cudaMemcpyAsync(&rz_last, sc + FD_RZ + it % 2, sizeof(double), cudaMemcpyDeviceToHost, st));
    QDKP_CUDA_TRY(cudaStreamSynchronize(st));
    if (!(rz_last > 0.0)) breakdown = 3;
  }
  // ---- strain at the element centres
  fd_strain<<<grid_blocks(N), 256, 0, st>>>(U, mask, g, dArr, eps_T, strain, total);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  unsigned long long hdrop = 0;
  QDKP_CUDA_TRY(cudaMemcpyAsync(&hdrop, dropped, sizeof(hdrop), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  info->iterations = it;
  info->residual = rel;
  info->modes_dropped = (int)hdrop;
  info->breakdown = breakdown;
  info->converged = rel < tol && !breakdown && hdrop <= 1;
  return QDKP_OK;
}

}  // extern "C"

extern "C" {

size_t qdkp_fourier_strain_workspace_size(int nx, int ny, int nz) {
  if (nx < 1 || ny < 1 || nz < 1) return 0;
  const long long N = (long long)nx * ny * nz;
  int dev = 0;
  cudaGetDevice(&dev);
  const size_t w = std::max(plan_work(dev, nx, ny, nz, 1), plan_work(dev, nx, ny, nz, 6));
  const size_t w3 = plan_work(dev, nx, ny, nz, 3);
  return al(7 * N * sizeof(double2)) + al(std::max(w, w3)) + 256;
}

int qdkp_fourier_strain(int nx, int ny, int nz, double h, const unsigned char* mask,
                        double eps_star, double C11, double C12, double C44, double* strain,
                        void* ws, size_t ws_bytes, void* stream) {
  QDKP_CHECK_ARG(nx >= 1 && ny >= 1 && nz >= 1 && h > 0.0, "grid extents must be >= 1, h > 0");
  QDKP_CHECK_ARG(mask && strain, "NULL argument");
  const long long N = (long long)nx * ny * nz;
  QDKP_CHECK_ARG(N < (1LL << 31), "grid too large for one transform");
  const size_t need = qdkp_fourier_strain_workspace_size(nx, ny, nz);
  if (!ws || ws_bytes < need || need == 0) {
    set_error("qdkp_fourier_strain: workspace too small (see qdkp_fourier_strain_workspace_size)");
    return QDKP_ERR_WORKSPACE;
  }
  int dev = 0;
  QDKP_CUDA_TRY(cudaGetDevice(&dev));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double2* chi = static_cast<double2*>(ws);
  double2* spec = chi + N;                                     // 6 N
  char* work = reinterpret_cast<char*>(ws) + al(7 * N * sizeof(double2));
  const size_t work_bytes = ws_bytes - al(7 * N * sizeof(double2));
  const Grid3 g{nx, ny, nz, h};
  const double eps_T = -eps_star;
  const int B = grid_blocks(N);
  mask_to_complex<<<B, 256, 0, st>>>(mask, N, chi);
  count_launch();
  int rc = run_fft(dev, nx, ny, nz, 1, chi, CUFFT_FORWARD, work, work_bytes, st);
  if (rc != QDKP_OK) return rc;
  strain_spectra<<<B, 256, 0, st>>>(chi, N, g, C11, C12, C44, eps_T, spec);
  count_launch();
  rc = run_fft(dev, nx, ny, nz, 6, spec, CUFFT_INVERSE, work, work_bytes, st);
  if (rc != QDKP_OK) return rc;
  strain_real<<<grid_blocks(6 * N), 256, 0, st>>>(spec, mask, N, eps_T, strain);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

size_t qdkp_piezo_potential_workspace_size(int nx, int ny, int nz) {
  return qdkp_fourier_strain_workspace_size(nx, ny, nz);
}

int qdkp_piezo_potential(int nx, int ny, int nz, double h, const double* strain,
                         const double* e14, double eps_r, double sign, double* phi, void* ws,
                         size_t ws_bytes, void* stream) {
  QDKP_CHECK_ARG(nx >= 1 && ny >= 1 && nz >= 1 && h > 0.0, "grid extents must be >= 1, h > 0");
  QDKP_CHECK_ARG(strain && e14 && phi, "NULL argument");
  QDKP_CHECK_ARG(eps_r > 0.0, "eps_r must be positive");
  const long long N = (long long)nx * ny * nz;
  QDKP_CHECK_ARG(N < (1LL << 31), "grid too large for one transform");
  const size_t need = qdkp_piezo_potential_workspace_size(nx, ny, nz);
  if (!ws || ws_bytes < need || need == 0) {
    set_error("qdkp_piezo_potential: workspace too small (see qdkp_piezo_potential_workspace_size)");
    return QDKP_ERR_WORKSPACE;
  }
  int dev = 0;
  QDKP_CUDA_TRY(cudaGetDevice(&dev));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double2* P = static_cast<double2*>(ws);                      // 3 N
  double2* D = P + 3 * N;                                      // N
  char* work = reinterpret_cast<char*>(ws) + al(7 * N * sizeof(double2));
  const size_t work_bytes = ws_bytes - al(7 * N * sizeof(double2));
  const Grid3 g{nx, ny, nz, h};
  const int B = grid_blocks(N);
  polarization_k<<<B, 256, 0, st>>>(strain, e14, N, sign, P);
  count_launch();
  int rc = run_fft(dev, nx, ny, nz, 3, P, CUFFT_FORWARD, work, work_bytes, st);
  if (rc != QDKP_OK) return rc;
  divergence_k<<<B, 256, 0, st>>>(P, N, g, D);
  count_launch();
  if ((rc = run_fft(dev, nx, ny, nz, 1, D, CUFFT_INVERSE, work, work_bytes, st)) != QDKP_OK) return rc;
  charge_density<<<B, 256, 0, st>>>(D, N);
  count_launch();
  if ((rc = run_fft(dev, nx, ny, nz, 1, D, CUFFT_FORWARD, work, work_bytes, st)) != QDKP_OK) return rc;
  poisson_filter<<<B, 256, 0, st>>>(D, N, g, eps_r);
  count_launch();
  if ((rc = run_fft(dev, nx, ny, nz, 1, D, CUFFT_INVERSE, work, work_bytes, st)) != QDKP_OK) return rc;
  real_part<<<B, 256, 0, st>>>(D, N, phi);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

}  // extern "C"
