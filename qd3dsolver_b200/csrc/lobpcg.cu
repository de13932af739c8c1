// LOBPCG on the device: the iteration of scipy.sparse.linalg.lobpcg (scipy 1.18.1,
// _eigen/lobpcg/lobpcg.py:688-1060) as qd3Dsolver calls it (eigensolvers.py:247-248, 352-353:
// B = None, M = None, Y = None, largest = False), with every block operation on the GPU.
//
// Per iteration (scipy line ranges in brackets):
//   R = A X - X diag(lambda), residual norms                       [688-700]
//   best-iterate bookkeeping, forced restart                       [702-718]
//   active mask                                                    [720-731]
//   R_act -= X (X^H R_act); Cholesky-orthonormalise R_act          [762-787]
//   A R_act                                                        [788]
//   Cholesky-orthonormalise P_act, A P_act (restart on failure)    [790-809]
//   explicit-Gram switch (sticky)                                  [815-824]
//   Gram blocks, generalized eigh of 3m x 3m (2m x 2m on restart)  [826-909]
//   Ritz update of X, A X, P, A P                                  [911-973]
// then the final Rayleigh-Ritz on the best iterate               [975-1060].
// The iteration is the batched engine's (engine.cu), run on a group of one slot: the decisions scipy
// takes on host scalars are taken on the device, and the host reads them once an iteration, on a
// second stream while R is being projected, to launch H.X with the active width. (Nine reads and
// host-side pencils an iteration took 9.6 ms for ten iterations of a 27 x 27 x 22 box, 12 columns;
// 7.4 ms so.)
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#include "engine_host.cuh"

namespace qdkp {

namespace {

constexpr int kNormParts = 296;
constexpr size_t kTables = 4096;       // the slot's descriptor on the device; the decisions' copy
static_assert(sizeof(ESlot) <= kTables && sizeof(EState) <= kTables, "tables");

BlockList<double> blist(std::initializer_list<std::pair<const double2*, int>> blocks, long long ld_default = -1) {
  BlockList<double> L;
  L.nblk = 0;
  for (auto& b : blocks) {
    L.p[L.nblk] = b.first;
    L.cols[L.nblk] = b.second;
    L.ld[L.nblk] = ld_default;
    ++L.nblk;
  }
  return L;
}

// the tall blocks of a solve: X AX P AP best Ra ARa Pa APa, and T for the folded operator
int n_blocks(const qdkp_lobpcg_params* prm) { return 9 + (prm->folded ? 1 : 0); }

struct Solver {
  const qdkp_operator* op;
  qdkp_lobpcg_params prm;
  cudaStream_t st;
  cudaStream_t side = nullptr;         // reads the decisions while st goes on
  cudaStream_t pst = nullptr;          // the work on P, beside that on R
  cudaEvent_t decided = nullptr, p_done = nullptr;
  int64_t n;
  int m;
  SlotLayout L;
  ESlot d{};
  int64_t applies = 0;
  int64_t hx_launches = 0;
  double hx_bytes = 0.0;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev;   // per-launch timing (time_hx)
  size_t ev_used = 0;

  int hx(const double2* V, int c, double2* out, double sigma, int shifted, int basis = 0) {
    ++hx_launches;
    hx_bytes += (double)op->n_sites * (15.0 * 8.0 + 2.0 * 8.0 * c * 16.0);
    if (!prm.time_hx) return launch_apply(op, V, c, out, c, c, sigma, shifted, QDKP_C128, st, basis);
    if (ev_used == ev.size()) {
      cudaEvent_t a, b2;
      QDKP_CUDA_TRY(cudaEventCreate(&a));
      QDKP_CUDA_TRY(cudaEventCreate(&b2));
      ev.emplace_back(a, b2);
    }
    auto& e = ev[ev_used++];
    QDKP_CUDA_TRY(cudaEventRecord(e.first, st));
    int rc = launch_apply(op, V, c, out, c, c, sigma, shifted, QDKP_C128, st, basis);
    QDKP_CUDA_TRY(cudaEventRecord(e.second, st));
    return rc;
  }

  // Sum the recorded launch durations (events are complete after the caller's sync).
  double hx_seconds() {
    double t = 0.0;
    for (size_t i = 0; i < ev_used; ++i) {
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, ev[i].first, ev[i].second) == cudaSuccess) t += ms * 1e-3;
    }
    return t;
  }

  ~Solver() {
    for (auto& e : ev) { cudaEventDestroy(e.first); cudaEventDestroy(e.second); }
    if (side) cudaStreamDestroy(side);
    if (pst) { cudaStreamSynchronize(pst); cudaStreamDestroy(pst); }
    if (decided) cudaEventDestroy(decided);
    if (p_done) cudaEventDestroy(p_done);
  }

  // A(V) for V (n x c, ld c) into out (ld c)
  int applyA(const double2* V, int c, double2* out) {
    applies += c;
    if (prm.folded) {
      int rc = hx(V, c, d.T, prm.sigma, 1, HX_Y_UNCOUPLED);
      if (rc) return rc;
      return hx(d.T, c, out, prm.sigma, 1, HX_X_UNCOUPLED);
    }
    return hx(V, c, out, 0.0, 0);
  }

  int gram(BlockList<double> A, BlockList<double> B, double2* out) {
    return launch_gram(A, B, n, reinterpret_cast<double2*>(d.gpart), L.gpart / sizeof(double2), out, st);
  }

  int sync_read(void* host, const void* dev, size_t bytes) {
    QDKP_CUDA_TRY(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st));
    QDKP_CUDA_TRY(cudaStreamSynchronize(st));
    return QDKP_OK;
  }

  // norms[j] = |A_j - lambda_j B_j|, through npart
  int col_norms(const double2* A, const double2* B, const double* lam, std::vector<double>& norms) {
    int rc = launch_colnorm2(A, m, B, m, lam, m, n, d.npart, d.nparts, d.gpart, st);
    if (rc) return rc;
    rc = sync_read(norms.data(), d.gpart, m * sizeof(double));
    if (rc) return rc;
    for (int j = 0; j < m; ++j) norms[j] = std::sqrt(std::fabs(norms[j]));
    return QDKP_OK;
  }

  int put(void* dev, const void* host, size_t bytes) {
    QDKP_CUDA_TRY(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st));
    return QDKP_OK;
  }
};

}  // namespace
}  // namespace qdkp

using namespace qdkp;

extern "C" {

size_t qdkp_lobpcg_workspace_size(const qdkp_operator* op, const qdkp_lobpcg_params* prm) {
  if (!op || !prm || prm->block < 1 || prm->block > kMaxBlock) return 0;
  const int64_t n = (int64_t)op->n_bands * op->n_sites;
  return slot_layout(n, prm->block, QDKP_C128, n_blocks(prm)).total + 2 * kTables;
}

int qdkp_lobpcg_solve(const qdkp_operator* op, const qdkp_lobpcg_params* prm, const void* X0,
                      double* lambda_out, void* V, double* resid_history,
                      qdkp_lobpcg_info* info, void* ws, size_t ws_bytes, void* stream) {
  QDKP_CHECK_ARG(op && prm && X0 && lambda_out && V && info, "NULL argument");
  QDKP_CHECK_ARG(prm->block >= 1 && prm->block <= kMaxBlock, "block must be in [1, 24]");
  QDKP_CHECK_ARG(prm->maxiter >= 0, "maxiter must be >= 0");
  if (prm->precision != QDKP_C128) {
    set_error("qdkp_lobpcg_solve: only QDKP_C128 is built for the single-solve form");
    return QDKP_ERR_UNSUPPORTED;
  }
  const auto t_start = std::chrono::steady_clock::now();
  Solver s;
  s.op = op;
  s.prm = *prm;
  s.st = static_cast<cudaStream_t>(stream);
  s.n = (int64_t)op->n_bands * op->n_sites;
  s.m = prm->block;
  const int m = s.m;
  const int64_t n = s.n;
  QDKP_CHECK_ARG(n >= 5 * m, "problem too small for LOBPCG (scipy switches to dense eigh)");
  s.L = slot_layout(n, m, QDKP_C128, n_blocks(prm));
  if (!ws || ws_bytes < s.L.total + 2 * kTables) {
    set_error("qdkp_lobpcg_solve: workspace too small (see qdkp_lobpcg_workspace_size)");
    return QDKP_ERR_WORKSPACE;
  }
  char* tables = static_cast<char*>(ws);
  ESlot& d = s.d;
  slot_carve(d, tables + 2 * kTables, s.L, n, m, QDKP_C128, n_blocks(prm));
  d.snap = reinterpret_cast<EState*>(tables + kTables);
  d.fault = device_fault_flag(op->device);
  cudaStream_t st = s.st;
  const int maxiter = prm->maxiter;
  const int hist_rows = maxiter + 3;
  std::vector<double> hist((size_t)hist_rows * m, 0.0);
  int rc;
#define TRY(x) do { rc = (x); if (rc != QDKP_OK) return rc; } while (0)

  // ---- X = orthonormalise(X0) ------------------------------------------------------------
  TRY(launch_copy((const double2*)X0, m, m, n, d.Ra, m, st));
  TRY(s.gram(blist({{d.Ra, m}}, m), blist({{d.Ra, m}}, m), d.gS));
  TRY(launch_chol_inv(d.gS, m, d.U, (int*)d.Up, st));
  int hstat;
  TRY(s.sync_read(&hstat, d.Up, sizeof(int)));
  if (hstat) { set_error("Linearly dependent initial approximations"); return QDKP_ERR_NUMERIC; }
  {
    const double2* C[1] = {d.U};
    TRY(launch_update(blist({{d.Ra, m}}, m), C, m, n, d.X, m, 0, st));
  }
  // ---- initial Ritz vectors ------------------------------------------------------------------
  TRY(s.applyA(d.X, m, d.AX));
  TRY(s.gram(blist({{d.X, m}}, m), blist({{d.AX, m}}, m), d.gT));
  TRY(launch_eigh(d.gT, nullptr, m, d.w, d.E, d.scr, (int*)d.Up, st));
  {
    const double2* C[1] = {d.E};
    TRY(launch_update(blist({{d.X, m}}, m), C, m, n, d.X, m, 0, st));
    TRY(launch_update(blist({{d.AX, m}}, m), C, m, n, d.AX, m, 0, st));
  }
  // the first decisions read the partials that this leaves in npart
  TRY(launch_colnorm2(d.AX, m, d.X, m, d.w, m, n, d.npart, d.nparts, d.gpart, st));
  std::vector<double> lam(m);
  TRY(s.sync_read(lam.data(), d.w, m * sizeof(double)));

  // ---- iterations ------------------------------------------------------------------------------
  EState es;
  slot_params(d, es, prm, lam.data());
  d.stall_iterations = 0;
  TRY(s.put(d.st, &es, sizeof(es)));
  TRY(s.put(tables, &d, sizeof(d)));
  QDKP_CUDA_TRY(cudaStreamCreateWithFlags(&s.side, cudaStreamNonBlocking));
  QDKP_CUDA_TRY(cudaStreamCreateWithFlags(&s.pst, cudaStreamNonBlocking));
  QDKP_CUDA_TRY(cudaEventCreateWithFlags(&s.decided, cudaEventDisableTiming));
  QDKP_CUDA_TRY(cudaEventCreateWithFlags(&s.p_done, cudaEventDisableTiming));
  set_slot_kernel_limits();
  EGroup G;
  G.d_slots = reinterpret_cast<ESlot*>(tables);
  G.ns = 1; G.gram_ctas = d.gparts; G.row_ctas = d.nparts; G.hx_ns[0] = 1; G.m_max = m;
  G.widths = {m};
  std::vector<double> norms(m);
  bool have_best = false;
  int it = -1;
  for (;;) {
    TRY(launch_decide(G, st));
    QDKP_CUDA_TRY(cudaEventRecord(s.decided, st));
    // H.X launches are timed alone
    const cudaStream_t ps = prm->time_hx ? st : s.pst;
    if (ps != st) QDKP_CUDA_TRY(cudaStreamWaitEvent(ps, s.decided, 0));
    TRY(launch_p_chain(G, ps));
    QDKP_CUDA_TRY(cudaEventRecord(s.p_done, ps));
    TRY(launch_r_chain(G, st));
    // none of this needs the host: it runs while the host reads the decisions
    QDKP_CUDA_TRY(cudaStreamWaitEvent(s.side, s.decided, 0));
    QDKP_CUDA_TRY(cudaMemcpyAsync(&es, d.snap, sizeof(es), cudaMemcpyDeviceToHost, s.side));
    QDKP_CUDA_TRY(cudaStreamSynchronize(s.side));
    TRY(check_device_fault(op->device));
    if (es.iter != it) {
      it = es.iter;
      std::memcpy(&hist[(size_t)it * m], es.norms, m * sizeof(double));
    }
    have_best = have_best || es.copy_best;
    if (!es.running) {
      QDKP_CUDA_TRY(cudaStreamWaitEvent(st, s.p_done, 0));      // the best iterate's copy
      break;
    }
    // scipy recomputes A X on a forced restart but keeps the residuals of the old A X
    if (!es.skip_recompute) TRY(s.applyA(d.X, m, d.AX));
    TRY(s.applyA(d.Ra, es.ma, d.ARa));
    QDKP_CUDA_TRY(cudaStreamWaitEvent(st, s.p_done, 0));
    TRY(launch_ritz_step(G, st));
    if (prm->verbosity > 1)
      fprintf(stderr, "lobpcg it %d active %d restart %d explicit %d\n", it, es.ma, es.restart,
              es.explicit_gram);
  }
  TRY(s.sync_read(&es, d.st, sizeof(es)));
  int status = es.status;
  const bool explicit_gram = es.explicit_gram;
  double smallest = es.smallest;
  int best_iter = es.best_iter;
  lam.assign(es.lam, es.lam + m);
  // ---- final residuals of the last iterate -------------------------------------------------
  if (status != QDKP_LOBPCG_NONFINITE) {
    TRY(s.col_norms(d.AX, d.X, d.st->lam, norms));
    double mean = 0.0;
    for (int j = 0; j < m; ++j) mean += norms[j];
    mean /= m;
    if (it + 1 < hist_rows) std::memcpy(&hist[(size_t)(it + 1) * m], norms.data(), m * sizeof(double));
    if (mean < smallest) {
      smallest = mean;
      best_iter = it + 1;
      TRY(launch_copy(d.X, m, m, n, d.best, m, st));
      have_best = true;
    }
  }
  if (!have_best) TRY(launch_copy(d.X, m, m, n, d.best, m, st));
  if (status == QDKP_LOBPCG_NONFINITE) {
    // a non-finite residual: nothing to refine; the iterate is returned as it is, Ritz values NaN
    TRY(launch_copy(d.best, m, m, n, (double2*)V, m, st));
    for (int j = 0; j < m; ++j) lambda_out[j] = std::numeric_limits<double>::quiet_NaN();
    const int rows = std::min(it + 1, hist_rows);
    if (resid_history) std::memcpy(resid_history, hist.data(), (size_t)rows * m * sizeof(double));
    info->iterations = rows;
    info->best_iteration = have_best ? best_iter : -1;
    info->status = status;
    info->explicit_gram = explicit_gram;
    info->best_mean_residual = smallest;
    info->hx_applications = s.applies * (prm->folded ? 2 : 1);
    info->hx_launches = s.hx_launches;
    info->hx_bytes = s.hx_bytes;
    QDKP_CUDA_TRY(cudaStreamSynchronize(st));
    info->hx_seconds = prm->time_hx ? s.hx_seconds() : 0.0;
    info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
    return check_device_fault(op->device);
  }
  // ---- final Rayleigh-Ritz on the best iterate (scipy lobpcg.py:1009-1060) -----------------
  TRY(s.applyA(d.best, m, d.AX));
  TRY(s.gram(blist({{d.best, m}}, m), blist({{d.AX, m}}, m), d.gT));
  TRY(s.gram(blist({{d.best, m}}, m), blist({{d.best, m}}, m), d.gS));
  {
    std::vector<double2> t((size_t)m * m), s2((size_t)m * m), a((size_t)m * m), bb((size_t)m * m);
    TRY(s.sync_read(t.data(), d.gT, t.size() * sizeof(double2)));
    TRY(s.sync_read(s2.data(), d.gS, s2.size() * sizeof(double2)));
    for (int i = 0; i < m; ++i)
      for (int j = 0; j < m; ++j) {
        const double2 x = t[(size_t)i * m + j], y = t[(size_t)j * m + i];
        a[(size_t)i * m + j] = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
        const double2 u = s2[(size_t)i * m + j], v = s2[(size_t)j * m + i];
        bb[(size_t)i * m + j] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
      }
    TRY(s.put(d.gA, a.data(), a.size() * sizeof(double2)));
    TRY(s.put(d.gB, bb.data(), bb.size() * sizeof(double2)));
  }
  TRY(launch_eigh(d.gA, d.gB, m, d.w, d.E, d.scr, (int*)d.Up, st));
  TRY(s.sync_read(&hstat, d.Up, sizeof(int)));
  if (hstat) { set_error("eigh has failed in lobpcg postprocessing"); return QDKP_ERR_NUMERIC; }
  TRY(s.sync_read(lam.data(), d.w, m * sizeof(double)));
  {
    const double2* C[1] = {d.E};
    TRY(launch_update(blist({{d.best, m}}, m), C, m, n, (double2*)V, m, 0, st));
    TRY(launch_update(blist({{d.AX, m}}, m), C, m, n, d.AX, m, 0, st));
  }
  TRY(s.col_norms(d.AX, (const double2*)V, d.w, norms));
  if (best_iter + 1 < hist_rows)
    std::memcpy(&hist[(size_t)(best_iter + 1) * m], norms.data(), m * sizeof(double));
  std::memcpy(lambda_out, lam.data(), m * sizeof(double));
  const int rows = std::min(best_iter + 2, hist_rows);
  if (resid_history) std::memcpy(resid_history, hist.data(), (size_t)rows * m * sizeof(double));
  if (status == QDKP_LOBPCG_MAXITER) {
    bool all = true;
    for (int j = 0; j < m; ++j) all = all && norms[j] <= d.tol;
    if (all) status = QDKP_LOBPCG_CONVERGED;
  }
  info->iterations = rows;
  info->best_iteration = best_iter;
  info->status = status;
  info->explicit_gram = explicit_gram;
  info->best_mean_residual = smallest;
  info->hx_applications = s.applies * (prm->folded ? 2 : 1);
  info->hx_launches = s.hx_launches;
  info->hx_bytes = s.hx_bytes;
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  info->hx_seconds = prm->time_hx ? s.hx_seconds() : 0.0;
  info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
#undef TRY
  return check_device_fault(op->device);
}

size_t qdkp_residuals_workspace_size(const qdkp_operator* op, int k) {
  if (!op || k < 1 || k > kMaxBlock) return 0;
  const size_t blk = ((size_t)op->n_bands * op->n_sites * k * sizeof(double2) + 255) / 256 * 256;
  return blk + (size_t)kNormParts * k * sizeof(double) + 4096 + gram_partial_elems(k, k) * sizeof(double2)
         + (size_t)k * k * sizeof(double2) * 2 + 4096;
}

int qdkp_residuals(const qdkp_operator* op, const void* V, int64_t ldv, int k, const double* E_in,
                   double* rq, double* res, void* ws, size_t ws_bytes, void* stream) {
  QDKP_CHECK_ARG(op && V && rq && res, "NULL argument");
  QDKP_CHECK_ARG(k >= 1 && k <= kMaxBlock && ldv >= k, "k must be in [1, 24] and ldv >= k");
  const size_t need = qdkp_residuals_workspace_size(op, k);
  if (!ws || ws_bytes < need) { set_error("qdkp_residuals: workspace too small"); return QDKP_ERR_WORKSPACE; }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t n = (int64_t)op->n_bands * op->n_sites;
  char* p = static_cast<char*>(ws);
  const size_t blk = ((size_t)n * k * sizeof(double2) + 255) / 256 * 256;
  double2* HV = (double2*)p; p += blk;
  double* part = (double*)p; p += ((size_t)kNormParts * k * sizeof(double) + 255) / 256 * 256;
  double* out = (double*)p; p += 2048;
  double* lam = (double*)p; p += 2048;
  double2* gpart = (double2*)p; p += gram_partial_elems(k, k) * sizeof(double2);
  double2* g1 = (double2*)p; p += (size_t)k * k * sizeof(double2);
  double2* g2 = (double2*)p;
  int rc = launch_apply(op, V, ldv, HV, k, k, 0.0, 0, QDKP_C128, st);
  if (rc) return rc;
  // Rayleigh quotients: diag(V^H H V) / diag(V^H V)
  BlockList<double> Lv = blist({{(const double2*)V, k}}, ldv);
  BlockList<double> Lh = blist({{HV, k}}, k);
  rc = launch_gram(Lv, Lh, n, gpart, gram_partial_elems(k, k), g1, st); if (rc) return rc;
  rc = launch_gram(Lv, Lv, n, gpart, gram_partial_elems(k, k), g2, st); if (rc) return rc;
  std::vector<double2> a((size_t)k * k), bb((size_t)k * k);
  QDKP_CUDA_TRY(cudaMemcpyAsync(a.data(), g1, a.size() * sizeof(double2), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaMemcpyAsync(bb.data(), g2, bb.size() * sizeof(double2), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  std::vector<double> E(k), nrm(k);
  for (int j = 0; j < k; ++j) {
    rq[j] = a[(size_t)j * k + j].x / bb[(size_t)j * k + j].x;
    nrm[j] = std::sqrt(bb[(size_t)j * k + j].x);
    E[j] = E_in ? E_in[j] : rq[j];
  }
  QDKP_CUDA_TRY(cudaMemcpyAsync(lam, E.data(), k * sizeof(double), cudaMemcpyHostToDevice, st));
  rc = launch_colnorm2(HV, k, (const double2*)V, ldv, lam, k, n, part, kNormParts, out, st);
  if (rc) return rc;
  std::vector<double> r2(k);
  QDKP_CUDA_TRY(cudaMemcpyAsync(r2.data(), out, k * sizeof(double), cudaMemcpyDeviceToHost, st));
  QDKP_CUDA_TRY(cudaStreamSynchronize(st));
  for (int j = 0; j < k; ++j) res[j] = std::sqrt(std::fabs(r2[j])) / nrm[j];
  return check_device_fault(op->device);
}

}  // extern "C"
