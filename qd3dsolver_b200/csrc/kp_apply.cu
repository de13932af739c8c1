// Matrix-free H.X for the discretised Pryor eight-band k.p operator (sm_100a).
//
// Replaces the CSR product `H @ X` of qd3Dsolver (H from kp_pryor.confined_hamiltonian,
// kp_pryor.py:363-466) with a fused 8x8-block, 19-point stencil. The operator is the sum of
//   * a local Hermitian 8x8 block per site (band edges, spin-orbit, Bir-Pikus Q/R/S strain
//     terms kp_pryor.py:111-113, and the diagonal of every second-derivative stencil),
//   * six face couplings: the three-point face-averaged k2_a stencils (kp_confined.py:88-143)
//     feeding A, P, Q and the real part of R, and the symmetrised first-derivative terms U, V
//     (kp_pryor.py:430-454, central differences kp_confined.py:58-85),
//   * twelve in-plane edge couplings: the symmetrised cross terms cross(g3, a, b)
//     (kp_confined.py:146-183) feeding the imaginary part of R and all of S.
//
// The uncoupled basis. Pryor's table (kp_pryor.py:244-301) is written in |J, m_J> states, in which
// every k.p term mixes up to six bands with square-root factors. One constant unitary per site
// takes them to |S>, |X>, |Y>, |Z> times spin (i |S>, so that the first-order terms are real):
//   X+ = (x4 + t) / sqrt2, Y+ = -i (x4 - t) / sqrt2, t = (x2 + sqrt2 x7) / sqrt3,
//   Z+ = -(sqrt2 x5 + x6) / sqrt3, S+ = i x0,
//   X- = (q + p) / sqrt2,  Y- = -i (q - p) / sqrt2,  q = (sqrt2 x6 - x5) / sqrt3, p = -x3,
//   Z- = (x7 - sqrt2 x2) / sqrt3, S- = i x1.
// There every difference operator is the same real 4x4 matrix for both spins: a face along axis a
// couples |a> with the weight -kp - 4 k2 and the other two with -kp + 2 k2, S with X, Y, Z by three
// first-order weights, and an in-plane edge couples just the two states of its plane. Only the
// spin-orbit term, local to the site, mixes the spins. A site and column takes 400 real
// multiply-adds instead of 1046.
//
// Kernels:
//   kp_record_kernel  once per operator (and per band-edge update): folds the 15 raw per-site
//                     fields into a per-site record of stencil weights in that basis and a
//                     neighbour mask; FP64 and FP32, the sign of the hole convention / negation
//                     folded in.
//   kp_march_kernel   a CTA owns a tile of (y, z) sites and a few columns and marches along x.
//   kp_apply_kernel   one thread per (site, column), neighbours through L1/L2: small blocks,
//                     four-band slices, and the batched engine.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "mbar_dev.cuh"     // CUtensorMap and its enums (the encoder is fetched from the runtime)

namespace qdkp {

// Record layout, site-major: entry k of site s at rec[s * rec_stride<T>() + k]. A site's record is a
// whole number of 16-byte words, and its pitch spreads the records of eight neighbouring sites over
// all shared-memory banks.
enum RecEntry {
  K_A = 0,        // sign (Ec + 6 G / h^2): S diagonal
  K_DX, K_DY, K_DZ,   // X, Y, Z diagonals
  K_XY, K_XZ, K_YZ,   // strain couplings of X, Y, Z
  K_SO,           // sign Delta / 3: spin-orbit couplings
  K_FYZ = 8,      // faces y+, y-, z+, z-: {along, across, cx, cy, cz} each
  K_EZY = 28,     // zy edges e: sz = e & 1 ? -1 : 1, sy = e & 2 ? -1 : 1
  // xy edges, stored with the plane they read: weight of x(ix, iy + s, iz) in the output of
  // (ix - 1, iy, iz) [s = +, -], then of (ix + 1, iy, iz) [s = +, -]
  K_PXY = 32,
  K_PZX = 36,     // zx edges: x(ix, iy, iz + s) in the same way
  K_FX = 40,      // faces x+, x-
  K_COUNT = 50
};
template <typename T> __host__ __device__ constexpr int rec_stride() { return sizeof(T) == 8 ? 54 : 52; }
// Words of a second, word-major copy, which single columns read: there every lane of a warp is another site,
// and the same word of 32 records lies on 32 lines. (Word-major records for all, with the words of four or of
// all sites together, cost the other blocks 3 to 12%; a warp's records staged in shared memory took
// 10 to 40% more than reading them in place, since L1 shrinks by what the stage takes.)
template <typename T> __host__ __device__ constexpr int rec_words() { return (K_COUNT * (int)sizeof(T) + 15) / 16; }

// ---------------------------------------------------------------------------------------------
// Record construction (FP64, once per operator)
// ---------------------------------------------------------------------------------------------
// first-order couplings of S with X, Y, Z of the derivative along each axis (P0 (1 - strain))
__device__ __forceinline__ void first_order_coefs(const double* __restrict__ F, long long N,
                                                  long long q, bool inter, double (&c)[3][3]) {
  const double P0 = F[F_P0 * N + q];
  double e[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  if (inter) {
    e[0][0] = F[F_EXX * N + q]; e[1][1] = F[F_EYY * N + q]; e[2][2] = F[F_EZZ * N + q];
    e[0][1] = e[1][0] = F[F_EXY * N + q];
    e[1][2] = e[2][1] = F[F_EYZ * N + q];
    e[0][2] = e[2][0] = F[F_EZX * N + q];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int j = 0; j < 3; ++j) c[a][j] = P0 * ((a == j ? 1.0 : 0.0) - e[a][j]);
}

// A thread per site; the records of a CTA's sites are put together in shared memory and written out
// as one contiguous run.
constexpr int kRecThreads = 64;
// Grids that get the copy for single columns. One column, complex128, site-major | word-major records (us):
// 48x48x36 8 bands 19.7 | 14.9, 6 bands 17.3 | 12.8, 4 bands 13.9 | 9.8; 64x64x48 47 | 38, 42 | 31, 34 | 24.
// Smaller grids (33x33x25: 7.4 | 6.6) are bound by the call, and eight complex64 bands lose there
// (18x18x15: 4.3 | 4.9).
constexpr int64_t kColumnSitesMin = 1 << 15, kColumnSitesMax = 1 << 19;
__global__ void __launch_bounds__(kRecThreads)
kp_record_kernel(const double* __restrict__ F, long long N, int nx, int ny,
                                 int nz, double h, int flags, int nb, double sign,
                                 double* __restrict__ rec64, float* __restrict__ rec32,
                                 double* __restrict__ col64, float* __restrict__ col32,
                                 unsigned* __restrict__ nbmask) {
  const double G = kG;
  const double ih2 = 1.0 / (h * h);
  const double i4h = 1.0 / (4.0 * h);
  // an edge's weight in the plane's X/Y/Z pair: -sqrt3 x 2 sqrt3 G x -(sa sb) / (8 h^2)
  const double ek = 6.0 * G / (8.0 * h * h);
  const double sq3 = 1.73205080756887729353;
  const bool strain = (flags & QDKP_STRAIN) != 0;
  const bool inter = nb == 8 && strain && (flags & QDKP_INTERBAND_STRAIN);
  __shared__ double sr[kRecThreads][rec_stride<double>() + 1];
  for (long long s0 = blockIdx.x * (long long)kRecThreads; s0 < N; s0 += (long long)gridDim.x * kRecThreads) {
    const int sites = (int)min((long long)kRecThreads, N - s0);
    const long long s = s0 + min((int)threadIdx.x, sites - 1);     // spare threads repeat the last site
    const int iz = (int)(s % nz);
    const long long t = s / nz;
    const int iy = (int)(t % ny);
    const int ix = (int)(t / ny);
    const int coord[3] = {ix, iy, iz};
    const int ext[3] = {nx, ny, nz};
    const long long str[3] = {(long long)ny * nz, (long long)nz, 1LL};
    double* r = sr[threadIdx.x];
    for (int k = 0; k < rec_stride<double>(); ++k) r[k] = 0.0;
    // neighbour mask: bit f (0..5) face x+, x-, y+, y-, z+, z-; bit 6 + 4 pl + e the in-plane
    // edge e of plane pl (xy, zx, zy) with signs sa = e & 1 ? -1 : 1, sb = e & 2 ? -1 : 1
    unsigned msk = 0;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      if (coord[ax] + 1 < ext[ax]) msk |= 1u << (2 * ax);
      if (coord[ax] > 0) msk |= 1u << (2 * ax + 1);
    }
    const double g1 = F[F_G1 * N + s], g2 = F[F_G2 * N + s];
    double c_p[3][3];
    if (nb == 8) first_order_coefs(F, N, s, inter, c_p);
    double dk1 = 0.0, dk2[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      double d1 = 0.0, d2 = 0.0;
#pragma unroll
      for (int dir = 0; dir < 2; ++dir) {
        const bool in = dir == 0 ? (coord[ax] + 1 < ext[ax]) : (coord[ax] > 0);
        const int kf = ax == 0 ? K_FX + 5 * dir : K_FYZ + 5 * (2 * (ax - 1) + dir);
        if (in) {
          const long long q = dir == 0 ? s + str[ax] : s - str[ax];
          const double t1 = (g1 + F[F_G1 * N + q]) * 0.5 * ih2;
          const double t2 = (g2 + F[F_G2 * N + q]) * 0.5 * ih2;
          d1 += t1; d2 += t2;
          // P carries -G t1, the gamma2 stencil -G t2
          r[kf + 0] = sign * G * (t1 + 4.0 * t2);
          r[kf + 1] = sign * G * (t1 - 2.0 * t2);
          if (nb == 8) {
            // symmetrised first derivative: (c_p + c_q) / 4h, signed by the face direction
            double c_q[3][3];
            first_order_coefs(F, N, q, inter, c_q);
            const double sg = dir == 0 ? i4h : -i4h;
#pragma unroll
            for (int j = 0; j < 3; ++j) r[kf + 2 + j] = sign * (c_p[ax][j] + c_q[ax][j]) * sg;
          }
        } else {  // hard wall: ghost term alpha_p / h^2 (kp_confined.py:133-137)
          d1 += g1 * ih2; d2 += g2 * ih2;
        }
      }
      dk1 += d1; dk2[ax] = d2;
    }
    double Q = G * (dk2[0] + dk2[1] - 2.0 * dk2[2]);
    double Rre = -sq3 * G * (dk2[0] - dk2[1]), Rim = 0.0, Sre = 0.0, Sim = 0.0;
    if (strain) {
      const double b = F[F_B * N + s], d = F[F_D * N + s];
      const double exx = F[F_EXX * N + s], eyy = F[F_EYY * N + s], ezz = F[F_EZZ * N + s];
      const double exy = F[F_EXY * N + s], eyz = F[F_EYZ * N + s], ezx = F[F_EZX * N + s];
      Q += -(b / 2.0) * (exx + eyy - 2.0 * ezz);
      Rre += (sq3 / 2.0) * b * (exx - eyy);
      Rim += -d * exy;
      Sre = -d * ezx;
      Sim = d * eyz;
    }
    const double P = -F[F_EV * N + s] + G * dk1;
    // a four-band slice has no split-off states: its vectors are zero there, Delta does not enter
    const double D3 = nb == 4 ? 0.0 : F[F_DSO * N + s] / 3.0;
    r[K_A] = sign * (F[F_EC * N + s] + 6.0 * G * ih2);
    r[K_DX] = sign * (-P - Q + sq3 * Rre - D3);
    r[K_DY] = sign * (-P - Q - sq3 * Rre - D3);
    r[K_DZ] = sign * (-P + 2.0 * Q - D3);
    r[K_XY] = sign * -sq3 * Rim;
    r[K_XZ] = sign * -sq3 * Sre;
    r[K_YZ] = sign * sq3 * Sim;
    r[K_SO] = sign * D3;
    // cross(g3, a, b): x(p + sa e_a + sb e_b) enters with the g3 of the two sites between
    auto g3 = [&](int dx, int dy, int dz) {
      return F[F_G3 * N + s + dx * str[0] + dy * str[1] + dz * str[2]];
    };
    const bool xp = ix + 1 < nx, xm = ix > 0, yp = iy + 1 < ny, ym = iy > 0, zp = iz + 1 < nz,
               zm = iz > 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int sa = (e & 1) ? -1 : 1, sb = (e & 2) ? -1 : 1;
      const double w = sign * ek * (double)(sa * sb);
      const bool xa = sa > 0 ? xp : xm, yb = sb > 0 ? yp : ym, za = sa > 0 ? zp : zm,
                 xb = sb > 0 ? xp : xm;
      if (xa && yb) msk |= 1u << (6 + e);
      if (za && xb) msk |= 1u << (10 + e);
      if (za && yb) { msk |= 1u << (14 + e); r[K_EZY + e] = w * (g3(0, 0, sa) + g3(0, sb, 0)); }
    }
    // the xy and zx edges of the outputs one plane down and up that read this plane
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int sx = (e & 2) ? 1 : -1, sb = (e & 1) ? -1 : 1;    // output at ix + sx
      const bool xo = sx > 0 ? xp : xm;
      const double w = sign * ek * (double)(-sx * sb);           // this plane lies at -sx of it
      if (xo && (sb > 0 ? yp : ym)) r[K_PXY + e] = w * (g3(0, 0, 0) + g3(sx, sb, 0));
      if (xo && (sb > 0 ? zp : zm)) r[K_PZX + e] = w * (g3(0, 0, 0) + g3(sx, 0, sb));
    }
    nbmask[s] = msk;
    if (col64) {
      for (int w = 0; w < rec_words<double>(); ++w)
        reinterpret_cast<double2*>(col64)[w * N + s] = make_double2(r[2 * w], r[2 * w + 1]);
      for (int w = 0; w < rec_words<float>(); ++w)
        reinterpret_cast<float4*>(col32)[w * N + s] =
            make_float4((float)r[4 * w], (float)r[4 * w + 1], (float)r[4 * w + 2], (float)r[4 * w + 3]);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < sites * rec_stride<double>(); e += kRecThreads)
      rec64[s0 * rec_stride<double>() + e] = sr[e / rec_stride<double>()][e % rec_stride<double>()];
    for (int e = threadIdx.x; e < sites * rec_stride<float>(); e += kRecThreads)
      rec32[s0 * rec_stride<float>() + e] = (float)sr[e / rec_stride<float>()][e % rec_stride<float>()];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// Values and weights. A value is one complex128 number, or C adjacent complex64 columns on packed
// f32x2 registers (sm_100 `fma.rn.f32x2`: a complex value is one 64-bit register pair and a real
// weight is broadcast to both halves); every stencil term is a real weight times a value.
// ---------------------------------------------------------------------------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2pk(float a, float b) {
  f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r;
}
__device__ __forceinline__ float2 f2up(f2 v) {
  float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d;
}

struct VD {                         // one complex128 value
  typedef double T;
  typedef double W;
  static constexpr int C = 1;
  double2 v;
};
template <int C_>
struct VF {                         // C complex64 columns
  typedef float T;
  typedef f2 W;
  static constexpr int C = C_;
  f2 c[C_];
};
__device__ __forceinline__ double wt(double w, VD*) { return w; }
template <int C> __device__ __forceinline__ f2 wt(float w, VF<C>*) { return f2pk(w, w); }
template <class V> __device__ __forceinline__ typename V::W W_(typename V::T w) { return wt(w, (V*)nullptr); }

__device__ __forceinline__ void vzero(VD& a) { a.v = make_double2(0.0, 0.0); }
template <int C> __device__ __forceinline__ void vzero(VF<C>& a) {
#pragma unroll
  for (int i = 0; i < C; ++i) a.c[i] = 0ull;
}
// a += w x
__device__ __forceinline__ void vfma(VD& a, double w, const VD& x) {
  a.v.x = fma(w, x.v.x, a.v.x); a.v.y = fma(w, x.v.y, a.v.y);
}
template <int C> __device__ __forceinline__ void vfma(VF<C>& a, f2 w, const VF<C>& x) {
#pragma unroll
  for (int i = 0; i < C; ++i) a.c[i] = fma2(w, x.c[i], a.c[i]);
}
// w x
__device__ __forceinline__ VD vmul(double w, const VD& x) {
  VD r; r.v = make_double2(w * x.v.x, w * x.v.y); return r;
}
template <int C> __device__ __forceinline__ VF<C> vmul(f2 w, const VF<C>& x) {
  VF<C> r;
#pragma unroll
  for (int i = 0; i < C; ++i) r.c[i] = mul2(w, x.c[i]);
  return r;
}
// i x
__device__ __forceinline__ VD vi(const VD& x) { VD r; r.v = make_double2(-x.v.y, x.v.x); return r; }
template <int C> __device__ __forceinline__ VF<C> vi(const VF<C>& x) {
  VF<C> r;
#pragma unroll
  for (int i = 0; i < C; ++i) { const float2 u = f2up(x.c[i]); r.c[i] = f2pk(-u.y, u.x); }
  return r;
}
// -i x
__device__ __forceinline__ VD vmi(const VD& x) { VD r; r.v = make_double2(x.v.y, -x.v.x); return r; }
template <int C> __device__ __forceinline__ VF<C> vmi(const VF<C>& x) {
  VF<C> r;
#pragma unroll
  for (int i = 0; i < C; ++i) { const float2 u = f2up(x.c[i]); r.c[i] = f2pk(u.y, -u.x); }
  return r;
}
__device__ __forceinline__ VD vload(const double2* p, VD*) { VD r; r.v = *p; return r; }
__device__ __forceinline__ VF<1> vload(const float2* p, VF<1>*) {
  VF<1> r; r.c[0] = *reinterpret_cast<const f2*>(p); return r;
}
__device__ __forceinline__ VF<2> vload(const float2* p, VF<2>*) {
  VF<2> r; const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  r.c[0] = v.x; r.c[1] = v.y; return r;
}
__device__ __forceinline__ VD vldg(const double2* p, VD*) { VD r; r.v = __ldg(p); return r; }
__device__ __forceinline__ VF<1> vldg(const float2* p, VF<1>*) {
  VF<1> r; r.c[0] = __ldg(reinterpret_cast<const f2*>(p)); return r;
}
__device__ __forceinline__ VF<2> vldg(const float2* p, VF<2>*) {
  VF<2> r; const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p));
  r.c[0] = v.x; r.c[1] = v.y; return r;
}
__device__ __forceinline__ void vstore(double2* p, const VD& a) { *p = a.v; }
__device__ __forceinline__ void vstore(float2* p, const VF<1>& a) { *reinterpret_cast<f2*>(p) = a.c[0]; }
__device__ __forceinline__ void vstore(float2* p, const VF<2>& a) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a.c[0], a.c[1]);
}

// Order of the eight values of a site in the uncoupled basis
enum { US = 0, UX, UY, UZ, DS, DX, DY, DZ };

// |J, m_J> values x (Pryor's band order) to the uncoupled basis u; six-band values leave S alone
template <class V, int NB>
__device__ __forceinline__ void to_uncoupled(const V (&x)[8], V (&u)[8]) {
  const auto c = [](double w) { return W_<V>((typename V::T)w); };
  const double i3 = 0.57735026918962576451, s23 = 0.81649658092772603273;   // 1/sqrt3, sqrt(2/3)
  const double i2 = 0.70710678118654752440, i6 = 0.40824829046386301637;    // 1/sqrt2, 1/sqrt6
  const auto one = c(1.0), none = c(-1.0);
  V t = vmul(c(i6), x[2]); vfma(t, c(i3), x[7]);                // t / sqrt2
  V a = vmul(c(i2), x[4]);
  u[UX] = a; vfma(u[UX], one, t);
  vfma(a, none, t);
  u[UY] = vmi(a);
  u[UZ] = vmul(c(-s23), x[5]); vfma(u[UZ], c(-i3), x[6]);
  V q = vmul(c(i3), x[6]); vfma(q, c(-i6), x[5]);               // q / sqrt2
  const V p = vmul(c(i2), x[3]);                                // -p / sqrt2
  u[DX] = q; vfma(u[DX], none, p);
  vfma(q, one, p);
  u[DY] = vmi(q);
  u[DZ] = vmul(c(i3), x[7]); vfma(u[DZ], c(-s23), x[2]);
  if (NB == 8) { u[US] = vi(x[0]); u[DS] = vi(x[1]); }
}

// the adjoint: uncoupled values u to |J, m_J>
template <class V, int NB>
__device__ __forceinline__ void from_uncoupled(const V (&u)[8], V (&x)[8]) {
  const auto c = [](double w) { return W_<V>((typename V::T)w); };
  const double i3 = 0.57735026918962576451, s23 = 0.81649658092772603273;
  const double i2 = 0.70710678118654752440, i6 = 0.40824829046386301637;
  const V iyu = vi(u[UY]), iyd = vi(u[DY]);
  x[4] = vmul(c(i2), u[UX]); vfma(x[4], c(i2), iyu);
  V t = u[UX]; vfma(t, c(-1.0), iyu);                           // sqrt2 t
  x[2] = vmul(c(i6), t); vfma(x[2], c(-s23), u[DZ]);
  x[7] = vmul(c(i3), t); vfma(x[7], c(i3), u[DZ]);
  V q = u[DX]; vfma(q, c(1.0), iyd);                            // sqrt2 q
  x[3] = vmul(c(-i2), u[DX]); vfma(x[3], c(i2), iyd);           // -p
  x[5] = vmul(c(-s23), u[UZ]); vfma(x[5], c(-i6), q);
  x[6] = vmul(c(-i3), u[UZ]); vfma(x[6], c(i3), q);
  if (NB == 8) { x[0] = vmi(u[US]); x[1] = vmi(u[DS]); }
}

// ---- stencil terms in the uncoupled basis ----------------------------------------------------
// the local block: y += (diagonal + shift) x, strain couplings, spin-orbit
template <class V, int NB>
__device__ __forceinline__ void local_term(V (&y)[8], const V (&x)[8], const typename V::T (&w)[8],
                                           typename V::T shift) {
  const auto dx = W_<V>(w[K_DX] + shift), dy = W_<V>(w[K_DY] + shift), dz = W_<V>(w[K_DZ] + shift);
  const auto xy = W_<V>(w[K_XY]), xz = W_<V>(w[K_XZ]), yz = W_<V>(w[K_YZ]);
  if (NB == 8) {
    const auto a = W_<V>(w[K_A] + shift);
    vfma(y[US], a, x[US]); vfma(y[DS], a, x[DS]);
  }
#pragma unroll
  for (int s = 0; s < 8; s += 4) {
    vfma(y[s + 1], dx, x[s + 1]); vfma(y[s + 2], dy, x[s + 2]); vfma(y[s + 3], dz, x[s + 3]);
    vfma(y[s + 1], xy, x[s + 2]); vfma(y[s + 2], xy, x[s + 1]); vfma(y[s + 3], xz, x[s + 1]);
    vfma(y[s + 1], xz, x[s + 3]); vfma(y[s + 2], yz, x[s + 3]); vfma(y[s + 3], yz, x[s + 2]);
  }
  const auto d = W_<V>(w[K_SO]), nd = W_<V>(-w[K_SO]);
  const V iyu = vi(x[UY]), iyd = vi(x[DY]), ixu = vi(x[UX]), ixd = vi(x[DX]);
  const V izu = vi(x[UZ]), izd = vi(x[DZ]);
  vfma(y[UX], d, iyu);  vfma(y[UX], nd, x[DZ]);
  vfma(y[UY], nd, ixu); vfma(y[UY], nd, izd);
  vfma(y[UZ], d, x[DX]); vfma(y[UZ], d, iyd);
  vfma(y[DX], nd, iyd); vfma(y[DX], d, x[UZ]);
  vfma(y[DY], d, ixd);  vfma(y[DY], nd, izu);
  vfma(y[DZ], nd, x[UX]); vfma(y[DZ], d, iyu);
}

// a face neighbour x along AX: w = {along, across, cx, cy, cz}; NEG: the first-order weights enter
// with the other sign (the same face seen from its other side); INIT: y is set, not added to
template <class V, int NB, int AX, bool NEG, bool INIT = false>
__device__ __forceinline__ void face_term(V (&y)[8], const V (&x)[8], const typename V::T* w,
                                          typename V::W cb) {
  const auto wl = W_<V>(w[0]), wm = W_<V>(w[1]);
  const auto add = [](V& a, typename V::W c, const V& v) {
    if (INIT) a = vmul(c, v);
    else vfma(a, c, v);
  };
#pragma unroll
  for (int s = 0; s < 8; s += 4) {
    add(y[s + 1], AX == 0 ? wl : wm, x[s + 1]);
    add(y[s + 2], AX == 1 ? wl : wm, x[s + 2]);
    add(y[s + 3], AX == 2 ? wl : wm, x[s + 3]);
  }
  if (NB == 8) {
    add(y[US], cb, x[US]); add(y[DS], cb, x[DS]);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const auto c = W_<V>(NEG ? -w[2 + j] : w[2 + j]), nc = W_<V>(NEG ? w[2 + j] : -w[2 + j]);
      vfma(y[US], c, x[UX + j]); vfma(y[DS], c, x[DX + j]);
      vfma(y[UX + j], nc, x[US]); vfma(y[DX + j], nc, x[DS]);
    }
  }
}

// an edge neighbour in the plane of the states A and B (1 X, 2 Y, 3 Z)
template <class V, int A, int B>
__device__ __forceinline__ void edge_term(V (&y)[8], const V (&x)[8], typename V::T w) {
  const auto c = W_<V>(w);
#pragma unroll
  for (int s = 0; s < 8; s += 4) { vfma(y[s + A], c, x[s + B]); vfma(y[s + B], c, x[s + A]); }
}

template <int NB> __device__ __forceinline__ constexpr bool has_band(int b) {
  return NB == 8 ? true : (NB == 6 ? b >= 2 : (b >= 2 && b <= 5));
}
template <int NB> __device__ __forceinline__ constexpr int band_off() { return NB == 8 ? 0 : 2; }

// ---------------------------------------------------------------------------------------------
// Direct kernel: one thread per (site, column), neighbours read through L1/L2. Bound by load latency
// and L1 wavefronts (128 16-byte loads per value). 48x48x36 x 12: complex128 119 us (185 in Pryor's
// basis with branches at the walls), complex64 59 us (116).
// ---------------------------------------------------------------------------------------------
template <typename T>
struct HXArgs {
  const T* __restrict__ rec;
  const unsigned* __restrict__ msk;
  const cplx<T>* __restrict__ X;
  cplx<T>* __restrict__ Y;
  int N, ldx, ldy, m, sx, sy;   // sites, leading dimensions, columns, site strides of x and y
  T shift;                      // -sigma for a shifted apply, else 0
  T cb;                         // conduction-band face weight sign (-G / h^2)
};

// Values of one column (or column pair) of the block in Pryor's band order at site offset `off`
// (in elements), xs = &X[0, s, j], bs = N ldx. Every offset fits 32 bits for the blocks this
// library accepts (n ldx < 2^31).
template <class V, int NB>
__device__ __forceinline__ void load_bands(const cplx<typename V::T>* __restrict__ xs, int bs,
                                           int off, bool vb_only, V (&x)[8]) {
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (!has_band<NB>(b) || (vb_only && b < 2)) { vzero(x[b]); continue; }
    x[b] = vldg(xs + ((b - band_off<NB>()) * bs + off), (V*)nullptr);
  }
}

// K entries of a record, in global (LDG) or shared memory
template <bool LDG, typename T, int K>
__device__ __forceinline__ void load_rec(const T* r, T (&w)[K]) {
  constexpr int E = 16 / (int)sizeof(T);
  static_assert(K % E == 0, "records are read in 16-byte words");
#pragma unroll
  for (int k = 0; k < K; k += E) {
    if constexpr (sizeof(T) == 8) {
      const double2* p = reinterpret_cast<const double2*>(r + k);
      const double2 v = LDG ? __ldg(p) : *p;
      w[k] = v.x; w[k + 1] = v.y;
    } else {
      const float4* p = reinterpret_cast<const float4*>(r + k);
      const float4 v = LDG ? __ldg(p) : *p;
      w[k] = v.x; w[k + 1] = v.y; w[k + 2] = v.z; w[k + 3] = v.w;
    }
  }
}

// Band order of the values in shared memory, and of a block in the uncoupled basis: Pryor's as copied (band b at word b - band_off),
// the uncoupled order after conversion: S+, X+, Y+, Z+, S-, X-, Y-, Z- (six bands: no S; RAW: the
// S values stay in words 0 and 1, the others follow).
template <int NB, bool RAW> __device__ __forceinline__ constexpr int uslot(int b) {
  return NB != 8 ? (b < 4 ? b - 1 : b - 2) : (RAW ? (b < 4 ? b + 1 : b) : b);
}

// One column's values at a site offset in the uncoupled basis; BASIS says which one X is in
template <class V, int NB, int BASIS>
__device__ __forceinline__ void load_uncoupled(const cplx<typename V::T>* __restrict__ xs, int bs, int off,
                                               V (&u)[8]) {
  if constexpr (BASIS & HX_X_UNCOUPLED) {
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (NB != 8 && (b & 3) == 0) { vzero(u[b]); continue; }
      u[b] = vldg(xs + (uslot<NB, false>(b) * bs + off), (V*)nullptr);
    }
  } else {
    V x[8];
    load_bands<V, NB>(xs, bs, off, false, x);
    to_uncoupled<V, NB>(x, u);
  }
}

// K entries of a record from entry FIRST on: COLUMN in the word-major copy, whose 16-byte word w of site s is at
// rec + (w N + s) words (rp: the site's first word, pitch N), else in the site's own run
template <bool COLUMN, int FIRST, typename T, int K>
__device__ __forceinline__ void load_site_rec(const T* rp, unsigned pitch, T (&w)[K]) {
  if constexpr (COLUMN) {
    constexpr int E = 16 / (int)sizeof(T);
#pragma unroll
    for (int k = 0; k < K; k += E) {
      T v[E];
      load_rec<true>(rp + pitch * (unsigned)(FIRST + k), v);
#pragma unroll
      for (int e = 0; e < E; ++e) w[k + e] = v[e];
    }
  } else {
    load_rec<true>(rp + FIRST, w);
  }
}

// Faces are taken to the uncoupled basis one by one; the four edge neighbours of a plane share
// one weight per band, so their weighted sum is formed first and taken there once. Nothing
// branches on the walls: a missing neighbour reads the site itself under a zero weight, so the
// loads of several neighbours can be in flight together.
// wall_self: the conduction bands' face weight, the one that is not zero at a wall, stays on there
// and multiplies the site itself. That is the operator complex64 engine slots of even width iterate
// on; it differs from the hard-wall operator only in rows next to a wall, and the complex128 finish
// of a mixed solve does not use it.
template <class V, int NB, int BASIS, bool COLUMN = false>
__device__ __forceinline__ void hx_item(const HXArgs<typename V::T>& a, int s, int j,
                                        bool wall_self = false) {
  typedef typename V::T T;
  const cplx<T>* xs = a.X + ((long long)s * a.ldx + j);
  const int bs = a.N * a.ldx;
  const int sx = a.sx * a.ldx, sy = a.sy * a.ldx, sz = a.ldx;
  constexpr int pitch = COLUMN ? 16 / (int)sizeof(T) : rec_stride<T>();     // of the sites
  const T* rp = a.rec + (long long)s * pitch;
  const long long rx = (long long)a.sx * pitch;                    // the x neighbours' records
  const unsigned msk = __ldg(a.msk + s);
  V y[8], x[8], u[8];
#pragma unroll
  for (int b = 0; b < 8; ++b) vzero(y[b]);
  {
    T w[8];
    load_site_rec<COLUMN, 0>(rp, a.N, w);
    load_uncoupled<V, NB, BASIS>(xs, bs, 0, u);
    local_term<V, NB>(y, u, w, a.shift);
  }
  const auto cbf = [&](int f) { return W_<V>(wall_self || (msk >> f & 1u) ? a.cb : T(0)); };
  const auto face_off = [&](int f, int d) { return (msk >> f & 1u) ? d : 0; };
  {
    T w[20];
    load_site_rec<COLUMN, K_FYZ>(rp, a.N, w);
#pragma unroll
    for (int f = 2; f < 6; ++f) {
      const int d = f < 4 ? sy : sz;
      load_uncoupled<V, NB, BASIS>(xs, bs, face_off(f, (f & 1) ? -d : d), u);
      if (f < 4) face_term<V, NB, 1, false>(y, u, w + 5 * (f - 2), cbf(f));
      else face_term<V, NB, 2, false>(y, u, w + 5 * (f - 2), cbf(f));
    }
  }
  {
    T w[sizeof(T) == 8 ? 10 : 12];
    load_site_rec<COLUMN, K_FX>(rp, a.N, w);
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      load_uncoupled<V, NB, BASIS>(xs, bs, face_off(f, f ? -sx : sx), u);
      face_term<V, NB, 0, false>(y, u, w + 5 * f, cbf(f));
    }
  }
#pragma unroll
  for (int pl = 0; pl < 3; ++pl) {
    const int sa = pl == 0 ? sx : sz, sb = pl == 1 ? sx : sy;
    // weights by e: an xy or zx edge's stands in the record of the x neighbour on its side
    T w[4];
    if (pl == 2) {
      load_site_rec<COLUMN, K_EZY>(rp, a.N, w);
    } else {
      T p[4];
      const bool up = msk & 1u, dn = msk & 2u;
      if (pl == 0) load_site_rec<COLUMN, K_PXY>(rp + (up ? rx : 0), a.N, p);
      else load_site_rec<COLUMN, K_PZX>(rp + (up ? rx : 0), a.N, p);
      w[0] = up ? p[0] : T(0); w[pl == 0 ? 2 : 1] = up ? p[1] : T(0);
      if (pl == 0) load_site_rec<COLUMN, K_PXY>(rp - (dn ? rx : 0), a.N, p);
      else load_site_rec<COLUMN, K_PZX>(rp - (dn ? rx : 0), a.N, p);
      w[pl == 0 ? 1 : 2] = dn ? p[2] : T(0); w[3] = dn ? p[3] : T(0);
    }
    V z[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) vzero(z[b]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int off = ((e & 1) ? -sa : sa) + ((e & 2) ? -sb : sb);
      const int o = (msk >> (6 + 4 * pl + e) & 1u) ? off : 0;
      const auto c = W_<V>(w[e]);
      if constexpr (BASIS & HX_X_UNCOUPLED) {
        // only the two states of the plane enter
        const int sa_ = pl == 2 ? 2 : 1, sb_ = pl == 0 ? 2 : 3;
#pragma unroll
        for (int sp = 0; sp < 8; sp += 4) {
          vfma(z[sp + sa_], c, vldg(xs + (uslot<NB, false>(sp + sa_) * bs + o), (V*)nullptr));
          vfma(z[sp + sb_], c, vldg(xs + (uslot<NB, false>(sp + sb_) * bs + o), (V*)nullptr));
        }
      } else {
        load_bands<V, NB>(xs, bs, o, true, x);
#pragma unroll
        for (int b = 2; b < 8; ++b) if (has_band<NB>(b)) vfma(z[b], c, x[b]);
      }
    }
    if constexpr (BASIS & HX_X_UNCOUPLED) {
#pragma unroll
      for (int b = 0; b < 8; ++b) u[b] = z[b];
    } else {
      to_uncoupled<V, 6>(z, u);
    }
    if (pl == 0) edge_term<V, 1, 2>(y, u, T(1));
    else if (pl == 1) edge_term<V, 1, 3>(y, u, T(1));
    else edge_term<V, 2, 3>(y, u, T(1));
  }
  cplx<T>* __restrict__ ys = a.Y + ((long long)s * a.ldy + j);
  const int ybs = a.N * a.ldy;
  if constexpr (BASIS & HX_Y_UNCOUPLED) {
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (NB != 8 && (b & 3) == 0) continue;
      vstore(ys + uslot<NB, false>(b) * ybs, y[b]);
    }
  } else {
    from_uncoupled<V, NB>(y, x);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (!has_band<NB>(b)) continue;
      vstore(ys + (b - band_off<NB>()) * ybs, x[b]);
    }
  }
}

constexpr int kApplyThreads = 256;
template <typename T> struct Column { typedef VF<1> V; };     // one column's value type
template <> struct Column<double> { typedef VD V; };
template <typename T> struct ApplyOcc;
template <> struct ApplyOcc<double> { static constexpr int kMinBlocks = 2; };
template <> struct ApplyOcc<float> { static constexpr int kMinBlocks = 3; };

template <typename T, int NB, int BASIS>
__global__ void __launch_bounds__(kApplyThreads, ApplyOcc<T>::kMinBlocks)
kp_apply_kernel(const HXArgs<T> a) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= a.N * a.m) return;
  const int s = it / a.m;
  hx_item<typename Column<T>::V, NB, BASIS>(a, s, it - s * a.m);
}

// ... of one column, with the records' word-major copy (kColumnSitesMin)
template <typename T, int NB, int BASIS>
__global__ void __launch_bounds__(kApplyThreads, ApplyOcc<T>::kMinBlocks)
kp_apply_column_kernel(const HXArgs<T> a) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < a.N) hx_item<typename Column<T>::V, NB, BASIS, true>(a, s, 0);
}

// Many operators and blocks in one launch (the batched engine): CTA b serves slot k with
// tile0[k] <= b < tile0[k+1]; the column count is read on the device (the slot's active width).
template <typename T, int BASIS, bool LOOP>
__global__ void __launch_bounds__(kApplyThreads, ApplyOcc<T>::kMinBlocks)
kp_apply_multi_kernel(const HXSlot* __restrict__ slots, int nslots, int tiles) {
  if (LOOP) {                                  // usually nothing to do
    bool any = false;
    for (int k = threadIdx.x; k < nslots; k += blockDim.x) any |= !(slots[k].skip && *slots[k].skip);
    if (!__syncthreads_or(any)) return;
  }
  for (int tile = blockIdx.x; tile < tiles; tile += LOOP ? (int)gridDim.x : tiles) {
    int k = 0;
    while (k + 1 < nslots && tile >= slots[k + 1].tile0) ++k;
    const HXSlot& d = slots[k];
    if ((d.skip && *d.skip) || (BASIS != 0) != (d.shifted != 0)) continue;
    const int m = d.m_dev ? *d.m_dev : d.m;
    const int it = (tile - d.tile0) * kApplyThreads + threadIdx.x;
    if (m <= 0 || it >= d.N * m) continue;
    HXArgs<T> a;
    a.rec = static_cast<const T*>(d.rec);
    a.msk = d.msk;
    a.X = static_cast<const cplx<T>*>(d.X);
    a.Y = static_cast<cplx<T>*>(d.Y);
    a.N = d.N; a.ldx = d.ld_same ? m : d.ldx; a.ldy = d.ld_same ? m : d.ldy;
    a.m = m; a.sx = d.sx; a.sy = d.sy;
    a.shift = d.shifted ? (T)(-d.sigma) : T(0);
    a.cb = (T)d.cb;
    const bool wall_self = std::is_same<T, float>::value && ((m | a.ldx | a.ldy) & 1) == 0 &&
                           ((reinterpret_cast<uintptr_t>(a.X) | reinterpret_cast<uintptr_t>(a.Y)) & 15) == 0;
    const int s = it / m;
    hx_item<typename Column<T>::V, 8, BASIS>(a, s, it - s * m, wall_self);
  }
}

// ---------------------------------------------------------------------------------------------
// Marching kernel: a CTA owns a TY x TZ tile of (y, z) sites and MC columns and marches along x.
// Plane x + 1 of the tile (a one-site halo in y and z, zero beyond the walls) and its records
// stream into shared memory with cp.async while plane x is worked on. The thread that copied a
// cell takes it to the uncoupled basis in place, so every value is converted once; then each
// thread reads the nine in-plane points of its site once and adds their contributions to the
// outputs of planes x - 1, x and x + 1, kept in registers: 56 shared loads per value where
// gathering the nineteen points takes 104, and one plane (not three) resident per stage. Bound by
// shared-memory wavefronts (complex128, 68% of the pipe) and, with eight warps of 200 registers on
// an SM, by fixed latencies; 128x128x96 x 24 columns, launches one after the other:
// complex128 2.77 ms, 3.6 TB/s (7.34 before, direct), complex64 1.42 ms, 3.5 TB/s (2.18 before, three resident
// planes in Pryor's basis); one launch after a pause, at full clocks, 2.42 and 1.22 ms.
// Smem of a stage: [band][y + 1][z + 1][column], then the records [site][kPitch].
// ---------------------------------------------------------------------------------------------
template <typename T_, int TY_, int TZ_, int MC_, int MINB_>
struct March {
  typedef T_ T;
  typedef typename std::conditional<std::is_same<T_, double>::value, VD, VF<2>>::type V;
  static constexpr int TY = TY_, TZ = TZ_, MC = MC_, MINB = MINB_;
  static constexpr int G = MC / V::C;                  // 16-byte column groups per cell
  static constexpr int PY = TY + 2, PZ = TZ + 2;
  static constexpr int BAND = PY * PZ * G;             // 16-byte words per band of a plane
  static constexpr int THREADS = TY * TZ * G;
  static constexpr int UNITS = PY * PZ * G;            // cell columns a plane copy is made of
  static constexpr int ROUNDS = (UNITS + THREADS - 1) / THREADS;
  static constexpr int kPitch = rec_stride<T>();
  static constexpr int RUNITS = kPitch * (int)sizeof(T) / 16;           // 16-byte words per site
  static_assert(MC % V::C == 0, "whole 16-byte groups");
  template <int NB> static constexpr size_t stage_bytes() {
    return (size_t)NB * BAND * 16 + (size_t)TY * TZ * kPitch * sizeof(T);
  }
  template <int NB> static constexpr size_t smem() { return 2 * stage_bytes<NB>(); }
};

template <typename T>
struct MarchArgs {
  const T* __restrict__ rec;
  const cplx<T>* __restrict__ X;
  cplx<T>* __restrict__ Y;
  long long bsx, bsy;           // band strides N ldx, N ldy
  int nx, ny, nz, ldx, ldy, m;
  int tiles_z, chunks, xsplit, xlen;
  int v16;                      // complex64: 16-byte column pairs in X
  int v16y;                     // ... and in Y
  T shift, cb;
  int* fault;                   // device_fault_flag
};

// cp.async of 16 (or 8) bytes of which the first `src_bytes` are read, the rest zero
__device__ __forceinline__ void cp16z(unsigned dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp8z(unsigned dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// raw_s: a converted cell keeps its two S values as copied (x0, x1 in slots 0 and 1) and the
// reader takes i times them, which complex128 folds into its multiply-adds; in complex64 the
// conversion does it.
template <class V> __device__ __forceinline__ constexpr bool raw_s() { return V::C == 1; }

template <class V, int NB, int BAND, bool RAW>
__device__ __forceinline__ void smem_cell(const cplx<typename V::T>* q, V (&x)[8]) {
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (NB != 8 && (b & 3) == 0) continue;
    if (RAW && (b & 3) == 0) { x[b] = vi(vload(q + (size_t)(b >> 2) * BAND * V::C, (V*)nullptr)); continue; }
    x[b] = vload(q + (size_t)uslot<NB, RAW>(b) * BAND * V::C, (V*)nullptr);
  }
}

// one cell column in shared memory from Pryor's basis to the uncoupled one, in place
template <class G, int NB>
__device__ __forceinline__ void convert_cell(cplx<typename G::T>* q) {
  typedef typename G::V V;
  constexpr bool RAW = raw_s<V>() && NB == 8;
  V x[8], u[8];
#pragma unroll
  for (int b = RAW ? 2 : 0; b < 8; ++b)
    if (has_band<NB>(b)) x[b] = vload(q + (size_t)(b - band_off<NB>()) * G::BAND * V::C, (V*)nullptr);
  to_uncoupled<V, RAW ? 6 : NB>(x, u);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if ((NB != 8 || RAW) && (b & 3) == 0) continue;
    vstore(q + (size_t)uslot<NB, RAW>(b) * G::BAND * V::C, u[b]);
  }
}

// the nine points of one plane added to the outputs of the plane below (lo) and its own (me), and
// the first part of the plane above's (up, set); a part that is not wanted is left out
template <class G, int NB, bool RAW, bool LO, bool ME, bool UP>
__device__ __forceinline__ void march_plane(const cplx<typename G::T>* cell,
                                            const typename G::T* r, typename G::T shift,
                                            typename G::V::W cb, typename G::V (&lo)[8],
                                            typename G::V (&me)[8], typename G::V (&up)[8]) {
  typedef typename G::V V;
  typedef typename G::T T;
  constexpr int DY_ = G::PZ * G::G * V::C, DZ_ = G::G * V::C;    // y and z strides (elements)
  V x[8];
  smem_cell<V, NB, G::BAND, RAW>(cell, x);
  if (ME) {
    T w[8];
    load_rec<false>(r, w);
    local_term<V, NB>(me, x, w, shift);
  }
  if (LO || UP) {
    T w[sizeof(T) == 8 ? 10 : 12];
    load_rec<false>(r + K_FX, w);
    // the face between this plane and the one above as the plane above sees it: same second-order
    // weights, opposite first-order ones
    if (UP) face_term<V, NB, 0, true, true>(up, x, w, cb);
    if (LO) face_term<V, NB, 0, true>(lo, x, w + 5, cb);
  }
  T wxy[4], wzx[4], wf[20];
  if (LO || UP) { load_rec<false>(r + K_PXY, wxy); load_rec<false>(r + K_PZX, wzx); }
  if (ME) load_rec<false>(r + K_FYZ, wf);
  smem_cell<V, NB, G::BAND, RAW>(cell + DY_, x);
  if (ME) face_term<V, NB, 1, false>(me, x, wf, cb);
  if (LO) edge_term<V, 1, 2>(lo, x, wxy[0]);
  if (UP) edge_term<V, 1, 2>(up, x, wxy[2]);
  smem_cell<V, NB, G::BAND, RAW>(cell - DY_, x);
  if (ME) face_term<V, NB, 1, false>(me, x, wf + 5, cb);
  if (LO) edge_term<V, 1, 2>(lo, x, wxy[1]);
  if (UP) edge_term<V, 1, 2>(up, x, wxy[3]);
  smem_cell<V, NB, G::BAND, RAW>(cell + DZ_, x);
  if (ME) face_term<V, NB, 2, false>(me, x, wf + 10, cb);
  if (LO) edge_term<V, 1, 3>(lo, x, wzx[0]);
  if (UP) edge_term<V, 1, 3>(up, x, wzx[2]);
  smem_cell<V, NB, G::BAND, RAW>(cell - DZ_, x);
  if (ME) face_term<V, NB, 2, false>(me, x, wf + 15, cb);
  if (LO) edge_term<V, 1, 3>(lo, x, wzx[1]);
  if (UP) edge_term<V, 1, 3>(up, x, wzx[3]);
  if (ME) {
    T w[4];
    load_rec<false>(r + K_EZY, w);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const cplx<T>* q = cell + ((e & 1) ? -DZ_ : DZ_) + ((e & 2) ? -DY_ : DY_);
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if ((b & 3) >= 2) x[b] = vload(q + (size_t)uslot<NB, RAW>(b) * G::BAND * V::C, (V*)nullptr);
      edge_term<V, 2, 3>(me, x, w[e]);
    }
  }
}

// a finished output column written in its basis
template <class G, int NB, int BASIS>
__device__ __forceinline__ void store_column(const typename G::V (&lo)[8], cplx<typename G::T>* ys, long long bsy,
                                             bool v16y, bool pair) {
  typedef typename G::V V;
  constexpr bool UNC = (BASIS & HX_Y_UNCOUPLED) != 0;
  V x[8];
  if (!UNC) from_uncoupled<V, NB>(lo, x);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (UNC ? (NB != 8 && (b & 3) == 0) : !has_band<NB>(b)) continue;
    const V v = UNC ? lo[b] : x[b];
    auto* yb = ys + (UNC ? uslot<NB, false>(b) : b - band_off<NB>()) * bsy;
    if constexpr (V::C == 1) {
      vstore(yb, v);
    } else if (v16y && pair) {
      vstore(yb, v);
    } else {
      const float2 e0 = f2up(v.c[0]), e1 = f2up(v.c[1]);
      yb[0] = e0;
      if (pair) yb[1] = e1;
    }
  }
}

template <class G, int NB, int BASIS>
__global__ void __launch_bounds__(G::THREADS, G::MINB)
kp_march_kernel(const MarchArgs<typename G::T> a) {
  typedef typename G::V V;
  typedef typename G::T T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool CONV = !(BASIS & HX_X_UNCOUPLED), RAW = CONV && raw_s<V>() && NB == 8;
  constexpr int STAGE = (int)G::template stage_bytes<NB>();
  int bid = blockIdx.x;
  const int xs = bid % a.xsplit; bid /= a.xsplit;
  const int ch = bid % a.chunks; bid /= a.chunks;
  const int tzi = bid % a.tiles_z;
  const int tyi = bid / a.tiles_z;
  const int c0 = ch * G::MC, y0 = tyi * G::TY, z0 = tzi * G::TZ;
  const int xa = xs * a.xlen, xb = min(a.nx, xa + a.xlen);
  if (c0 >= a.m || xa >= xb) return;          // uniform over the CTA
  const int t = threadIdx.x;
  const int g = t % G::G, tz = (t / G::G) % G::TZ, ty = t / (G::G * G::TZ);
  const int iy = y0 + ty, iz = z0 + tz, col = c0 + g * V::C;
  const bool active = iy < a.ny && iz < a.nz && col < a.m;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem_raw);
  // the cell columns this thread copies and converts: source of band 0 in plane 0, valid bytes
  const cplx<T>* src[G::ROUNDS];
  int bytes[G::ROUNDS];
#pragma unroll
  for (int k = 0; k < G::ROUNDS; ++k) {
    const int u = t + k * G::THREADS;
    const int cu = u % G::G, zz = (u / G::G) % G::PZ, yy = u / (G::G * G::PZ);
    const int gy = y0 - 1 + yy, gz = z0 - 1 + zz, gc = c0 + cu * V::C;
    const bool in = u < G::UNITS && gy >= 0 && gy < a.ny && gz >= 0 && gz < a.nz && gc < a.m;
    bytes[k] = in ? min(V::C, a.m - gc) * (int)sizeof(cplx<T>) : 0;
    src[k] = a.X + (in ? ((long long)gy * a.nz + gz) * a.ldx + gc : 0);
  }
  const long long xstr = (long long)a.ny * a.nz * a.ldx;
  auto copy_plane = [&](int p) {
    const unsigned st = sbase + (p & 1) * STAGE;
#pragma unroll
    for (int k = 0; k < G::ROUNDS; ++k) {
      const int u = t + k * G::THREADS;
      if (u < G::UNITS) {
        const unsigned dst = st + u * 16;
        const cplx<T>* s = src[k] + (bytes[k] ? p * xstr : 0);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const cplx<T>* sb = s + (bytes[k] ? b * a.bsx : 0);
          if (sizeof(T) == 8 || a.v16) {
            cp16z(dst + b * G::BAND * 16, sb, bytes[k]);
          } else {
            cp8z(dst + b * G::BAND * 16, sb, min(bytes[k], 8));
            cp8z(dst + b * G::BAND * 16 + 8, sb + (bytes[k] > 8 ? 1 : 0), max(bytes[k] - 8, 0));
          }
        }
      }
    }
    // records of the tile's sites
    const unsigned rt = st + NB * G::BAND * 16;
    for (int u = t; u < G::TY * G::TZ * G::RUNITS; u += G::THREADS) {
      const int w = u % G::RUNITS, site = u / G::RUNITS;
      const int gy = y0 + site / G::TZ, gz = z0 + site % G::TZ;
      if (gy < a.ny && gz < a.nz)
        cp16z(rt + site * (G::kPitch * (int)sizeof(T)) + w * 16,
              a.rec + (((long long)p * a.ny + gy) * a.nz + gz) * G::kPitch + w * (16 / (int)sizeof(T)), 16);
    }
    cp_async_commit();
  };
  auto convert_plane = [&](int p) {
    cplx<T>* st = reinterpret_cast<cplx<T>*>(smem_raw + (p & 1) * STAGE);
#pragma unroll
    for (int k = 0; k < G::ROUNDS; ++k) {
      if (bytes[k] == 0) continue;
      cplx<T>* q = st + (size_t)(t + k * G::THREADS) * V::C;
      convert_cell<G, NB>(q);
    }
  };
  V lo[8], me[8], up[8];
#pragma unroll
  for (int b = 0; b < 8; ++b) { vzero(lo[b]); vzero(me[b]); vzero(up[b]); }
  const int p0 = max(xa - 1, 0), p1 = min(xb, a.nx - 1);     // planes read
  const auto cb = W_<V>(a.cb);
  const int cell = ((ty + 1) * G::PZ + (tz + 1)) * G::G + g;
  cplx<T>* __restrict__ yout = a.Y + ((long long)iy * a.nz + iz) * a.ldy + col;
  const long long ystr = (long long)a.ny * a.nz * a.ldy;
  copy_plane(p0);
  for (int p = p0; p <= p1; ++p) {
    cp_async_wait_all();
    if (CONV) convert_plane(p);
    __syncthreads();          // plane p is complete; every thread is done with plane p - 1
    if (p < p1) copy_plane(p + 1);
    if (active) {
      const cplx<T>* c = reinterpret_cast<const cplx<T>*>(smem_raw + (p & 1) * STAGE) + (size_t)cell * V::C;
      const T* r = reinterpret_cast<const T*>(smem_raw + (p & 1) * STAGE + NB * G::BAND * 16) +
                   (ty * G::TZ + tz) * G::kPitch;
      if (p < xa) march_plane<G, NB, RAW, false, false, true>(c, r, a.shift, cb, lo, me, up);
      else if (p == xb) march_plane<G, NB, RAW, true, false, false>(c, r, a.shift, cb, lo, me, up);
      else march_plane<G, NB, RAW, true, true, true>(c, r, a.shift, cb, lo, me, up);
    }
    // output of plane q = p - 1 is complete; the last one also when no plane follows
#pragma unroll 1
    for (int q = p - 1; q <= p; ++q) {
      const bool write = q == p - 1 ? q >= xa : (p == p1 && p < xb);
      if (q == p && !write) break;
      if (write && active)
        store_column<G, NB, BASIS>(lo, yout + q * ystr, a.bsy, a.v16y, col + 1 < a.m);
#pragma unroll
      for (int b = 0; b < 8; ++b) { lo[b] = me[b]; me[b] = up[b]; }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The same march fed by the tensor-memory accelerator: one elected thread brings in a plane with
// one bulk tensor copy (coordinates beyond the walls read as zeros) and the tile's records with
// one bulk copy per tile row, completion on an mbarrier per stage, so no thread computes a copy
// address. NS stages of planes are in flight; a plane is converted (where X is in Pryor's basis) after the previous
// one's arithmetic, before the barrier that the two share. The launcher takes it where a tensor
// map can describe the block (tma_fits).
// ---------------------------------------------------------------------------------------------
template <class G, int NB, int NS, int BASIS>
__global__ void __launch_bounds__(G::THREADS, G::MINB)
kp_march_tma_kernel(const __grid_constant__ CUtensorMap tmx, const MarchArgs<typename G::T> a) {
  typedef typename G::V V;
  typedef typename G::T T;
  extern __shared__ unsigned char smem_raw[];
  constexpr bool CONV = !(BASIS & HX_X_UNCOUPLED), RAW = CONV && raw_s<V>() && NB == 8;
  constexpr int STAGE = (int)G::template stage_bytes<NB>();
  constexpr int XBYTES = NB * G::BAND * 16;
  static_assert(STAGE % 128 == 0 && XBYTES % 128 == 0, "stages stay 128-byte aligned");
  const unsigned raw = (unsigned)__cvta_generic_to_shared(smem_raw);
  const unsigned pad = ((raw + 127u) & ~127u) - raw;
  unsigned char* sm = smem_raw + pad;
  const unsigned sbase = raw + pad, bars = sbase + NS * STAGE;
  int bid = blockIdx.x;
  const int xs = bid % a.xsplit; bid /= a.xsplit;
  const int ch = bid % a.chunks; bid /= a.chunks;
  const int tzi = bid % a.tiles_z;
  const int tyi = bid / a.tiles_z;
  const int c0 = ch * G::MC, y0 = tyi * G::TY, z0 = tzi * G::TZ;
  const int xa = xs * a.xlen, xb = min(a.nx, xa + a.xlen);
  if (c0 >= a.m || xa >= xb) return;          // uniform over the CTA
  const int t = threadIdx.x;
  const int g = t % G::G, tz = (t / G::G) % G::TZ, ty = t / (G::G * G::TZ);
  const int iy = y0 + ty, iz = z0 + tz, col = c0 + g * V::C;
  const bool active = iy < a.ny && iz < a.nz && col < a.m;
  const int p0 = max(xa - 1, 0), p1 = min(xb, a.nx - 1);     // planes read
  const int rrows = min(G::TY, a.ny - y0), rsites = min(G::TZ, a.nz - z0);
  // plane p lives in stage (p - p0) % NS, whose barrier completes phase (p - p0) / NS
  auto issue = [&](int p) {
    const int q = (p - p0) % NS;
    const unsigned bar = bars + 8u * q, st = sbase + q * STAGE;
    const unsigned rb = (unsigned)(rsites * G::kPitch * (int)sizeof(T));
    mbar_expect_tx(bar, XBYTES + rrows * rb);
    tma_load_5d(st, &tmx, bar, c0 * (int)(sizeof(cplx<T>) / 8), z0 - 1, y0 - 1, p, 0);
    for (int r = 0; r < rrows; ++r)
      bulk_load(st + XBYTES + r * (G::TZ * G::kPitch * (int)sizeof(T)),
                a.rec + (((long long)p * a.ny + y0 + r) * a.nz + z0) * G::kPitch, rb, bar);
  };
  if (t == 0) {
    for (int i = 0; i < NS; ++i) mbar_init(bars + 8u * i, 1);
    mbar_init_fence();
    for (int p = p0; p < p0 + NS && p <= p1; ++p) issue(p);
  }
  __syncthreads();
  // the cells this thread converts (those of the halo beyond a wall hold zeros)
  auto convert = [&](unsigned char* st) {
#pragma unroll
    for (int k = 0; k < G::ROUNDS; ++k) {
      const int u = t + k * G::THREADS;
      if (u >= G::UNITS) break;
      cplx<T>* q = reinterpret_cast<cplx<T>*>(st) + (size_t)u * V::C;
      convert_cell<G, NB>(q);
    }
    // these stores are ordered before the copy that refills the stage
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  };
  V lo[8], me[8], up[8];
#pragma unroll
  for (int b = 0; b < 8; ++b) { vzero(lo[b]); vzero(me[b]); vzero(up[b]); }
  const auto cb = W_<V>(a.cb);
  const int cell = ((ty + 1) * G::PZ + (tz + 1)) * G::G + g;
  cplx<T>* __restrict__ yout = a.Y + ((long long)iy * a.nz + iz) * a.ldy + col;
  const long long ystr = (long long)a.ny * a.nz * a.ldy;
  bool ok = mbar_wait(bars, 0);
  if (CONV) {
    if (ok) convert(sm);
    ok = __syncthreads_and(ok) != 0;
  }
  int slot = 0;
  unsigned phase = 0;
  for (int p = p0; p <= p1; ++p) {
    unsigned char* st = sm + slot * STAGE;
    if (active && ok) {
      const cplx<T>* c = reinterpret_cast<const cplx<T>*>(st) + (size_t)cell * V::C;
      const T* r = reinterpret_cast<const T*>(st + XBYTES) + (ty * G::TZ + tz) * G::kPitch;
      if (p < xa) march_plane<G, NB, RAW, false, false, true>(c, r, a.shift, cb, lo, me, up);
      else if (p == xb) march_plane<G, NB, RAW, true, false, false>(c, r, a.shift, cb, lo, me, up);
      else march_plane<G, NB, RAW, true, true, true>(c, r, a.shift, cb, lo, me, up);
    }
    // output of plane q = p - 1 is complete; the last one also when no plane follows
#pragma unroll 1
    for (int q = p - 1; q <= p; ++q) {
      const bool write = q == p - 1 ? q >= xa : (p == p1 && p < xb);
      if (q == p && !write) break;
      if (write && active && ok)
        store_column<G, NB, BASIS>(lo, yout + q * ystr, a.bsy, a.v16y, col + 1 < a.m);
#pragma unroll
      for (int b = 0; b < 8; ++b) { lo[b] = me[b]; me[b] = up[b]; }
    }
    if (p == p1) break;
    const int next = slot + 1 == NS ? 0 : slot + 1;
    const unsigned nphase = next == 0 ? phase ^ 1u : phase;
    ok = ok && mbar_wait(bars + 8u * next, nphase);
    if (CONV && ok) convert(sm + next * STAGE);
    ok = __syncthreads_and(ok) != 0;       // plane p + 1 is complete, stage `slot` may be refilled
    if (!ok) break;
    if (t == 0 && p + NS <= p1) issue(p + NS);
    slot = next;
    phase = nphase;
  }
  if (!ok && t == 0) {
    // a copy never landed: flag it, then give the copies still in flight a bounded chance to
    // finish before the CTA's shared memory is released
    raise_device_fault(a.fault);
    for (int i = 0; i < NS; ++i) { mbar_wait(bars + 8u * i, 0); mbar_wait(bars + 8u * i, 1); }
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
// Tile shapes {TY, TZ, columns, CTAs per SM} of the TMA march, the shape of its cp.async form, and
// per shape the time of one plane of a CTA (us, measured at 128x128x96 with 24 columns: launch time
// over waves x planes), which pick_tile compares shapes by. Tile numbers 0..3 exist in both
// precisions, the others in complex64 only; a number past the built ones takes shape 0.
template <typename T> struct MarchCfgs;
template <> struct MarchCfgs<double> {
  using C0 = March<double, 8, 8, 4, 1>;
  using C1 = March<double, 4, 8, 4, 2>;
  using C2 = March<double, 8, 12, 4, 1>;
  using C3 = March<double, 8, 8, 2, 2>;
  using Any = C3;
  static constexpr int kShapes = 4;
};
template <> struct MarchCfgs<float> {
  using C0 = March<float, 8, 8, 8, 1>;
  using C1 = March<float, 4, 8, 8, 2>;
  using C2 = March<float, 8, 12, 8, 1>;
  using C3 = March<float, 8, 8, 4, 2>;
  using C4 = March<float, 4, 12, 8, 2>;
  using C5 = March<float, 4, 8, 4, 4>;
  using Any = C3;
  static constexpr int kShapes = 6;
};
constexpr int kBothCfgs = 4;               // tiles built for both precisions
constexpr int kDirect = QDKP_TILE_DIRECT;  // staged_cfg value selecting the direct kernel

// f(shape tag, plane time) over the shapes of a precision; f returns true to stop
template <class S> struct ShapeTag { using G = S; };
template <typename T, class F>
static void each_shape(F f) {
  using C = MarchCfgs<T>;
  if constexpr (std::is_same<T, double>::value) {
    if (f(0, ShapeTag<typename C::C0>(), 2.34)) return;
    if (f(1, ShapeTag<typename C::C1>(), 2.49)) return;
    if (f(2, ShapeTag<typename C::C2>(), 3.41)) return;
    f(3, ShapeTag<typename C::C3>(), 2.72);
  } else {
    if (f(0, ShapeTag<typename C::C0>(), 2.58)) return;
    if (f(1, ShapeTag<typename C::C1>(), 2.48)) return;
    if (f(2, ShapeTag<typename C::C2>(), 3.41)) return;
    if (f(3, ShapeTag<typename C::C3>(), 2.67)) return;
    if (f(4, ShapeTag<typename C::C4>(), 3.27)) return;
    f(5, ShapeTag<typename C::C5>(), 2.57);
  }
}

struct MarchGeom { int tiles_y, tiles_z, chunks, xsplit, xlen, ctas; double steps; };   // steps: waves x planes

// CTA decomposition for a grid: x is split so that the CTA count fills whole waves, trading the
// two extra planes that each x run reads.
static MarchGeom march_geom(int nx, int ny, int nz, int m, int MC, int TY, int TZ, int slots) {
  MarchGeom g;
  g.tiles_y = (ny + TY - 1) / TY;
  g.tiles_z = (nz + TZ - 1) / TZ;
  g.chunks = (m + MC - 1) / MC;
  const long long base = (long long)g.tiles_y * g.tiles_z * g.chunks;
  double best = 1e30;
  g.xsplit = 1;
  for (int xs = 1; xs <= nx; ++xs) {
    const int xlen = (nx + xs - 1) / xs;
    if ((long long)(xs - 1) * xlen >= nx) continue;
    const long long ctas = base * xs;
    const double cost = (double)((ctas + slots - 1) / slots) * (xlen + 2);
    if (cost < best - 1e-9) { best = cost; g.xsplit = xs; }
  }
  g.xlen = (nx + g.xsplit - 1) / g.xsplit;
  g.ctas = (int)(base * g.xsplit);
  g.steps = best;
  return g;
}

// A kernel's shared-memory limit, raised once per device.
template <class K>
static cudaError_t raise_smem(K kernel, size_t bytes, int device, std::atomic<unsigned long long>& done) {
  const unsigned long long bit = 1ull << (device & 63);
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && device < 64) done.fetch_or(bit, std::memory_order_release);
  return e;
}

template <class G, int NB, int BASIS>
static int launch_march_g(const qdkp_operator* op, const typename G::T* rec, const void* X, int ldx,
                          void* Y, int ldy, int m, typename G::T shift, typename G::T cb, int sms,
                          cudaStream_t st) {
  typedef typename G::T T;
  constexpr size_t smem = G::template smem<NB>();
  static_assert((smem + 1024) * G::MINB <= 233472, "over the shared memory of one SM");
  static std::atomic<unsigned long long> raised{0};
  QDKP_CUDA_TRY(raise_smem(kp_march_kernel<G, NB, BASIS>, smem, op->device, raised));
  const MarchGeom g = march_geom(op->nx, op->ny, op->nz, m, G::MC, G::TY, G::TZ, sms * G::MINB);
  MarchArgs<T> a;
  a.rec = rec;
  a.X = static_cast<const cplx<T>*>(X);
  a.Y = static_cast<cplx<T>*>(Y);
  a.bsx = (long long)op->n_sites * ldx; a.bsy = (long long)op->n_sites * ldy;
  a.nx = op->nx; a.ny = op->ny; a.nz = op->nz;
  a.ldx = ldx; a.ldy = ldy; a.m = m;
  a.tiles_z = g.tiles_z; a.chunks = g.chunks; a.xsplit = g.xsplit; a.xlen = g.xlen;
  a.v16 = ((uintptr_t)X & 15) == 0 && ldx % 2 == 0;
  a.v16y = ((uintptr_t)Y & 15) == 0 && ldy % 2 == 0;
  a.shift = shift; a.cb = cb;
  kp_march_kernel<G, NB, BASIS><<<g.ctas, G::THREADS, smem, st>>>(a);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda)
static EncodeTiledFn tensor_map_encoder() {
  static const EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                        cudaSuccess && q == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
  }();
  return fn;
}

// tensor-map rules: 16-byte aligned base and strides; every box no larger than its tensor
template <class G>
static bool tma_fits(const qdkp_operator* op, const void* X, int64_t ldx, int m) {
  return ((uintptr_t)X & 15) == 0 && (sizeof(typename G::T) == 8 || ldx % 2 == 0) && m >= G::MC &&
         op->ny >= G::PY && op->nz >= G::PZ && tensor_map_encoder() != nullptr;
}

template <class G, int NB, int NS, int BASIS>
static int launch_march_tma(const qdkp_operator* op, const typename G::T* rec, const void* X, int ldx,
                            void* Y, int ldy, int m, typename G::T shift, typename G::T cb, int sms,
                            cudaStream_t st) {
  typedef typename G::T T;
  constexpr size_t smem = 128 + NS * G::template stage_bytes<NB>() + 8 * NS;
  static_assert((smem + 1024) * G::MINB <= 233472, "over the shared memory of one SM");
  static std::atomic<unsigned long long> raised{0};
  QDKP_CUDA_TRY(raise_smem(kp_march_tma_kernel<G, NB, NS, BASIS>, smem, op->device, raised));
  // X as [band][x][y][z][column], in 8-byte elements with the column innermost
  constexpr int E = (int)sizeof(cplx<T>) / 8;
  const cuuint64_t ld = (cuuint64_t)ldx * sizeof(cplx<T>);
  const cuuint64_t dim[5] = {(cuuint64_t)m * E, (cuuint64_t)op->nz, (cuuint64_t)op->ny,
                             (cuuint64_t)op->nx, (cuuint64_t)NB};
  const cuuint64_t str[4] = {ld, (cuuint64_t)op->nz * ld, (cuuint64_t)op->ny * op->nz * ld,
                             (cuuint64_t)op->n_sites * ld};
  const cuuint32_t box[5] = {(cuuint32_t)(G::MC * E), (cuuint32_t)G::PZ, (cuuint32_t)G::PY, 1, (cuuint32_t)NB};
  const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
  CUtensorMap tmx;
  const CUresult r = tensor_map_encoder()(
      &tmx, CU_TENSOR_MAP_DATA_TYPE_INT64, 5, const_cast<void*>(X), dim, str, box, ones,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed for the X block (code " + std::to_string((int)r) + ")");
    return QDKP_ERR_CUDA;
  }
  const MarchGeom g = march_geom(op->nx, op->ny, op->nz, m, G::MC, G::TY, G::TZ, sms * G::MINB);
  MarchArgs<T> a{};
  a.rec = rec;
  a.Y = static_cast<cplx<T>*>(Y);
  a.bsy = (long long)op->n_sites * ldy;
  a.nx = op->nx; a.ny = op->ny; a.nz = op->nz;
  a.ldx = ldx; a.ldy = ldy; a.m = m;
  a.tiles_z = g.tiles_z; a.chunks = g.chunks; a.xsplit = g.xsplit; a.xlen = g.xlen;
  a.v16y = ((uintptr_t)Y & 15) == 0 && ldy % 2 == 0;
  a.shift = shift; a.cb = cb;
  a.fault = device_fault_flag(op->device);
  kp_march_tma_kernel<G, NB, NS, BASIS><<<g.ctas, G::THREADS, smem, st>>>(tmx, a);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

template <typename T, int NB, int BASIS>
static int launch_march(int cfg, const qdkp_operator* op, const T* rec, const void* X, int ldx,
                        void* Y, int ldy, int m, T shift, T cb, int sms, cudaStream_t st) {
  int rc = QDKP_OK;
  bool done = false;
  each_shape<T>([&](int i, auto tag, double) {
    using G = typename decltype(tag)::G;
    if (i != (cfg < MarchCfgs<T>::kShapes ? cfg : 0) || !tma_fits<G>(op, X, ldx, m)) return false;
    rc = launch_march_tma<G, NB, 2, BASIS>(op, rec, X, ldx, Y, ldy, m, shift, cb, sms, st);
    return done = true;
  });
  if (done) return rc;
  // a block no tensor map describes, or a grid or block smaller than the tile
  return launch_march_g<typename MarchCfgs<T>::Any, NB, BASIS>(op, rec, X, ldx, Y, ldy, m, shift, cb, sms, st);
}

int launch_apply_multi(const HXSlot* slots_dev, int nslots, int total_tiles, int precision, int basis,
                       int max_ctas, cudaStream_t st) {
  if (total_tiles <= 0) return QDKP_OK;
  const auto launch = [&](auto kernel, int ctas) {
    kernel<<<ctas, kApplyThreads, 0, st>>>(slots_dev, nslots, total_tiles);
  };
  const auto of_basis = [&](auto tag) {
    typedef decltype(tag) T;
    const int n = total_tiles;
    if (max_ctas < n) {
      if (basis == HX_X_UNCOUPLED) launch(kp_apply_multi_kernel<T, HX_X_UNCOUPLED, true>, max_ctas);
      else if (basis == HX_Y_UNCOUPLED) launch(kp_apply_multi_kernel<T, HX_Y_UNCOUPLED, true>, max_ctas);
      else launch(kp_apply_multi_kernel<T, 0, true>, max_ctas);
    } else {
      if (basis == HX_X_UNCOUPLED) launch(kp_apply_multi_kernel<T, HX_X_UNCOUPLED, false>, n);
      else if (basis == HX_Y_UNCOUPLED) launch(kp_apply_multi_kernel<T, HX_Y_UNCOUPLED, false>, n);
      else launch(kp_apply_multi_kernel<T, 0, false>, n);
    }
  };
  if (precision == QDKP_C128) of_basis(double());
  else of_basis(float());
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  return QDKP_OK;
}

int apply_tiles(int64_t n_sites, int m) {
  return (int)((n_sites * m + kApplyThreads - 1) / kApplyThreads);
}

// sign of the operator as applied: -1 for a hole-convention 6/4-band slice, flipped by NEGATE
static double op_sign(const qdkp_operator* op) {
  double sign = ((op->flags & QDKP_HOLE_CONVENTION) && op->n_bands != 8) ? -1.0 : 1.0;
  if (op->flags & QDKP_NEGATE) sign = -sign;
  return sign;
}

double apply_cb_weight(const qdkp_operator* op) { return op_sign(op) * (-kG / (op->h * op->h)); }

int build_records(qdkp_operator* op) {
  const long long N = op->n_sites;
  const int blocks = (int)std::min<long long>((N + kRecThreads - 1) / kRecThreads, 148 * 16);
  kp_record_kernel<<<blocks, kRecThreads>>>(op->fields64, N, op->nx, op->ny, op->nz, op->h, op->flags,
                                     op->n_bands, op_sign(op), op->rec64, op->rec32, op->col64, op->col32,
                                     op->nbmask);
  count_launch();
  QDKP_CUDA_TRY(cudaGetLastError());
  QDKP_CUDA_TRY(cudaDeviceSynchronize());
  return QDKP_OK;
}

size_t column_record_bytes(int64_t n_sites, int precision) {
  if (n_sites < kColumnSitesMin || n_sites > kColumnSitesMax) return 0;
  return (size_t)(precision == QDKP_C64 ? rec_words<float>() : rec_words<double>()) * 16 * n_sites;
}

size_t record_values(int64_t n_sites) { return (size_t)rec_stride<double>() * n_sites; }

static int num_sms(int device) {
  static int cached[64] = {0};
  if (device < 0 || device >= 64) return 148;
  if (!cached[device]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || v <= 0)
      v = 148;
    cached[device] = v;
  }
  return cached[device];
}

// Default kernel of a launch: the shape with the smallest waves x planes x plane time, against the
// direct kernel's time per (site, column). A block that no tensor map describes stays on the direct kernel:
// 91x91x76, complex64, 13 / 17 / 23 columns 479 / 625 / 846 us, the cp.async march 654 / 905 / 1162. Measured (us, direct / march): complex128 23x23x20 x 12
// 20 / 18, 48x48x36 x 12 119 / 82, 91x91x76 x 24 2111 / 1160; complex64 10 / 15, 59 / 51, 947 / 560.
// qdkp_operator_tune refines this per operator.
template <typename T>
static int pick_tile(const qdkp_operator* op, const void* X, int64_t ldx, int m, int sms) {
  if (op->n_bands == 4) return kDirect;
  const double items = (double)op->n_sites * m;
  double best = 3.0 + items * (sizeof(T) == 8 ? 1.18e-4 : 0.57e-4);
  int tile = kDirect;
  if (best <= 3.0 + 2.3) return tile;              // no march takes less than a plane: skip the models
  each_shape<T>([&](int i, auto tag, double plane) {
    using G = typename decltype(tag)::G;
    if (!tma_fits<G>(op, X, ldx, m)) return false;
    const MarchGeom g = march_geom(op->nx, op->ny, op->nz, m, G::MC, G::TY, G::TZ, sms * G::MINB);
    const double us = 3.0 + g.steps * plane;
    if (us < best) { best = us; tile = i; }
    return false;
  });
  return tile;
}

// The direct kernel; a block of few items is spread over the whole chip in small CTAs (23x23x20 x 1:
// 42 CTAs of 256 threads would leave 106 SMs idle; 8.0 -> 5.1 us with 64).
template <typename T, int NB, int BASIS>
static int launch_direct(const qdkp_operator* op, HXArgs<T> a, int sms, cudaStream_t st) {
  const int64_t items = op->n_sites * a.m;
  int threads = kApplyThreads;
  while (threads > 64 && items < (int64_t)threads * 2 * sms) threads /= 2;
  // a single column's call is bound by the host: one runtime call, which returns its own error
  const T* col = sizeof(T) == 8 ? (const T*)op->col64 : (const T*)op->col32;
  const bool column = a.m == 1 && col != nullptr;
  if (column) a.rec = col;
  void* args[] = {&a};
  QDKP_CUDA_TRY(cudaLaunchKernel(column ? reinterpret_cast<const void*>(&kp_apply_column_kernel<T, NB, BASIS>)
                                        : reinterpret_cast<const void*>(&kp_apply_kernel<T, NB, BASIS>),
                                 dim3((unsigned)((items + threads - 1) / threads)), dim3(threads), args, 0, st));
  count_launch();
  return QDKP_OK;
}

template <typename T, int BASIS>
static int launch_apply_t(const qdkp_operator* op, const T* rec, const void* X, int64_t ldx,
                          void* Y, int64_t ldy, int m, double sigma, int shifted, int precision,
                          cudaStream_t st) {
  if ((int64_t)op->n_bands * op->n_sites * std::max(ldx, ldy) >= (int64_t(1) << 31)) {
    set_error("H.X: n * leading dimension must stay below 2^31 elements");
    return QDKP_ERR_UNSUPPORTED;
  }
  const T shift = shifted ? (T)(-sigma) : T(0);
  const T cb = (T)apply_cb_weight(op);
  const int forced = op->staged_cfg[precision == QDKP_C64];
  const int sms = num_sms(op->device);
  const int cfg = forced == QDKP_TILE_AUTO ? pick_tile<T>(op, X, ldx, m, sms) : forced;
  if (cfg != kDirect && op->n_bands != 4 && ((uintptr_t)X % sizeof(cplx<T>)) == 0) {
    if (op->n_bands == 8)
      return launch_march<T, 8, BASIS>(cfg, op, rec, X, (int)ldx, Y, (int)ldy, m, shift, cb, sms, st);
    return launch_march<T, 6, BASIS>(cfg, op, rec, X, (int)ldx, Y, (int)ldy, m, shift, cb, sms, st);
  }
  HXArgs<T> a;
  a.rec = rec;
  a.msk = op->nbmask;
  a.X = static_cast<const cplx<T>*>(X);
  a.Y = static_cast<cplx<T>*>(Y);
  a.N = (int)op->n_sites; a.ldx = (int)ldx; a.ldy = (int)ldy; a.m = m;
  a.sx = op->ny * op->nz; a.sy = op->nz;
  a.shift = shift;
  a.cb = cb;
  switch (op->n_bands) {
    case 8: return launch_direct<T, 8, BASIS>(op, a, sms, st);
    case 6: return launch_direct<T, 6, BASIS>(op, a, sms, st);
    case 4: return launch_direct<T, 4, 0>(op, a, sms, st);
    default: set_error("n_bands must be 8, 6 or 4"); return QDKP_ERR_ARG;
  }
}

template <int BASIS>
static int launch_apply_b(const qdkp_operator* op, const void* X, int64_t ldx, void* Y, int64_t ldy,
                          int m, double sigma, int shifted, int precision, cudaStream_t st) {
  if (precision == QDKP_C128)
    return launch_apply_t<double, BASIS>(op, op->rec64, X, ldx, Y, ldy, m, sigma, shifted, precision, st);
  if (precision == QDKP_C64)
    return launch_apply_t<float, BASIS>(op, op->rec32, X, ldx, Y, ldy, m, sigma, shifted, precision, st);
  set_error("precision must be QDKP_C128 or QDKP_C64");
  return QDKP_ERR_ARG;
}

// Y = sign*H X (- sigma X if shifted) for one block in the given precision.
int launch_apply(const qdkp_operator* op, const void* X, int64_t ldx, void* Y, int64_t ldy,
                 int m, double sigma, int shifted, int precision, cudaStream_t st, int basis) {
  if (basis == HX_X_UNCOUPLED)
    return launch_apply_b<HX_X_UNCOUPLED>(op, X, ldx, Y, ldy, m, sigma, shifted, precision, st);
  if (basis == HX_Y_UNCOUPLED)
    return launch_apply_b<HX_Y_UNCOUPLED>(op, X, ldx, Y, ldy, m, sigma, shifted, precision, st);
  return launch_apply_b<0>(op, X, ldx, Y, ldy, m, sigma, shifted, precision, st);
}

int launch_folded(const qdkp_operator* op, const void* X, int64_t ldx, void* T, void* Y, int64_t ldy,
                  int m, double sigma, int precision, cudaStream_t st) {
  const int rc = launch_apply(op, X, ldx, T, m, m, sigma, 1, precision, st, HX_Y_UNCOUPLED);
  if (rc != QDKP_OK) return rc;
  return launch_apply(op, T, m, Y, ldy, m, sigma, 1, precision, st, HX_X_UNCOUPLED);
}

}  // namespace qdkp

using namespace qdkp;

extern "C" {

int qdkp_operator_set_tile(qdkp_operator* op, int precision, int tile) {
  QDKP_CHECK_ARG(op != nullptr, "operator must not be NULL");
  QDKP_CHECK_ARG(precision == QDKP_C128 || precision == QDKP_C64, "bad precision");
  QDKP_CHECK_ARG(tile >= QDKP_TILE_DIRECT && tile < QDKP_TILE_COUNT, "tile out of range");
  QDKP_CHECK_ARG(precision == QDKP_C64 || tile < kBothCfgs,
                 "the tile shapes from 4 on are built for complex64 only");
  op->staged_cfg[precision == QDKP_C64] = tile;
  return QDKP_OK;
}

int qdkp_operator_get_tile(const qdkp_operator* op, int precision, int* tile) {
  QDKP_CHECK_ARG(op != nullptr && tile != nullptr, "NULL argument");
  QDKP_CHECK_ARG(precision == QDKP_C128 || precision == QDKP_C64, "bad precision");
  *tile = op->staged_cfg[precision == QDKP_C64];
  return QDKP_OK;
}

int qdkp_operator_tune(qdkp_operator* op, const void* X, int64_t ldx, void* Y, int64_t ldy,
                       int m, int precision, int reps, double* seconds, void* stream) {
  QDKP_CHECK_ARG(op != nullptr && X != nullptr && Y != nullptr, "NULL argument");
  QDKP_CHECK_ARG(precision == QDKP_C128 || precision == QDKP_C64, "bad precision");
  QDKP_CHECK_ARG(m > 0 && ldx >= m && ldy >= m && reps > 0, "bad block or repetitions");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  QDKP_CUDA_TRY(cudaSetDevice(op->device));
  const int pi = precision == QDKP_C64;
  const int saved = op->staged_cfg[pi];
  cudaEvent_t e0, e1;
  QDKP_CUDA_TRY(cudaEventCreate(&e0));
  QDKP_CUDA_TRY(cudaEventCreate(&e1));
  int best = saved;
  float best_ms = 3.4e38f;
  int rc = QDKP_OK;
  // candidates: the built shapes, the direct kernel last; the seconds array has one entry per
  // tile number, -1 for one that does not apply
  for (int c = 0; c <= QDKP_TILE_COUNT && rc == QDKP_OK; ++c) {
    const int tile = c < QDKP_TILE_COUNT ? c : kDirect;
    if (seconds) seconds[c] = -1.0;
    if (op->n_bands == 4 && tile != kDirect) continue;                // four bands: direct only
    if (tile != kDirect && tile >= (precision == QDKP_C64 ? MarchCfgs<float>::kShapes : MarchCfgs<double>::kShapes)) continue;
    op->staged_cfg[pi] = tile;
    rc = launch_apply(op, X, ldx, Y, ldy, m, 0.0, 0, precision, st);      // warm-up
    if (rc != QDKP_OK) break;
    if (cudaEventRecord(e0, st) != cudaSuccess) { rc = QDKP_ERR_CUDA; break; }
    for (int r = 0; r < reps && rc == QDKP_OK; ++r)
      rc = launch_apply(op, X, ldx, Y, ldy, m, 0.0, 0, precision, st);
    if (rc != QDKP_OK) break;
    float ms = 0.f;
    if (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
        cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) { rc = QDKP_ERR_CUDA; break; }
    if (seconds) seconds[c] = ms * 1e-3 / reps;
    if (ms < best_ms) { best_ms = ms; best = tile; }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  op->staged_cfg[pi] = rc == QDKP_OK ? best : saved;
  if (rc == QDKP_ERR_CUDA) set_error("qdkp_operator_tune: CUDA event failure");
  return rc;
}

}  // extern "C"
