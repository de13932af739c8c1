// Device side of the batched LOBPCG engine: per-slot state, descriptors and the multi-slot
// kernels. One tick advances every running slot by one iteration of scipy's LOBPCG
// (lobpcg.py:688-973); the decisions scipy takes on host scalars are taken here by one-CTA
// kernels per slot, so a tick is a fixed sequence of launches with no host round trip.
#pragma once
#include "dense_dev.cuh"

namespace qdkp {

// Per-slot mutable state (device memory, written by the decision kernels).
struct EState {
  int running;          // 1 while the slot iterates
  int status;           // QDKP_LOBPCG_* once it stopped
  int iter;             // scipy's iterationNumber of the current tick (starts at -1)
  int idle;             // 1: this tick's kernels skip the slot (written by the decision kernel alone)
  int r_idle;           // idle, or R's orthonormalisation or the eigensolve failed: the kernels on R and
                        // those that follow the eigensolve skip the slot. (Those on P run beside R's.)
  int ma;               // active residual columns this tick
  int mp;               // P columns in this tick's Rayleigh-Ritz (0: restart)
  int restart, forced, explicit_gram;
  int best_iter;
  int copy_best;        // X of this tick is the new best iterate
  int skip_recompute;   // 0: forced restart recomputes A X this tick
  int skip_p;           // 1: no P block this tick (iteration 0 or idle)
  int skip_pnorm;       // 1: P orthonormalisation is not applied
  int resid_ready;      // 1: Ra holds the residuals of all m columns of X
  int skip_resid;       // 1: ... and this tick wants them all
  double smallest;
  int active[kMaxBlock];
  int idx[kMaxBlock];
  double lam[kMaxBlock];
  double norms[kMaxBlock];
};

// Per-slot constant descriptor (built on the host at admission, device resident).
// The tall blocks (X ... T) hold complex128 or, for a complex64 slot (prec = QDKP_C64), complex64
// values; they are declared double2 and reinterpreted through blk<T>(). Everything small (Gram
// matrices, Ritz coefficients, residual norms) is FP64 in both cases.
struct ESlot {
  long long n;          // rows (8 N)
  int m;                // block width
  int prec;             // QDKP_C128 or QDKP_C64: arithmetic of the tall blocks and of H.X
  double sqrt_eps;      // sqrt(machine epsilon) of that arithmetic (explicit Gram switch)
  int folded;
  double tol;
  int maxiter;
  int stall_iterations;  // > 0: stop once the best mean residual is this many iterations old
  int restart_control;
  double2 *X, *AX, *P, *AP, *best, *Ra, *ARa, *Pa, *APa, *T;
  double2 *W, *U, *Up, *gS, *gT, *gA, *gB, *E, *scr, *Cx, *Cr, *Cp;
  double* w;
  double* npart;        // [nparts][m] residual-norm partials of the current X
  double* gpart;        // Gram partials (real)
  double* ppart;        // ... of P^H P
  int nparts;           // their parts: CTAs of the row kernels
  int gparts;           // row parts (CTAs) of the Gram kernel
  int gram0, row0;      // first CTA of this slot in the Gram / row-kernel launches
  int utile0;           // complex64 slots: first 128-row tile in the group's tcgen05 update space
  int rows_per_cta;     // rows per CTA in the row kernels (gather, update, norms)
  EState* st;
  int* fault;           // device_fault_flag
  EState* snap;         // NULL, or where the decision kernel leaves a copy of st for the host
};

template <typename T>
__device__ __forceinline__ cplx<T>* blk(double2* p) { return reinterpret_cast<cplx<T>*>(p); }

__device__ __forceinline__ int slot_of(const ESlot* __restrict__ S, int ns, int b,
                                       int ESlot::*first) {
  int k = 0;
  while (k + 1 < ns && b >= S[k + 1].*first) ++k;
  return k;
}

}  // namespace qdkp
