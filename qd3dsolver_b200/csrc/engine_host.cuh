// Host side shared by the batched engine (engine.cu) and the single-solve driver (lobpcg.cu): a
// solve's device workspace, and the launches of an iteration over a group of slots. The single
// solve is a group of one slot.
#pragma once
#include <vector>

#include "engine_dev.cuh"

namespace qdkp {

enum RowWhich { RW_COPYBEST = 0, RW_RESID, RW_GATHERP };

// bytes of a slot's pieces; `total` with n_blocks tall blocks
struct SlotLayout {
  size_t blk, small, npart, gpart, ppart, total;
  int nparts, gparts, rows_per_cta;
};
SlotLayout slot_layout(int64_t n, int m, int prec, int n_blocks);
// cuts ws into d's pieces (d.T only where n_blocks says so) and sets d.n .. d.rows_per_cta
void slot_carve(ESlot& d, void* ws, const SlotLayout& L, int64_t n, int m, int prec, int n_blocks);
// the solve's constants and its state before the first iteration (lam: initial Ritz values)
void slot_params(ESlot& d, EState& s, const qdkp_lobpcg_params* prm, const double* lam);

struct EGroup {
  ESlot* d_slots = nullptr;            // this group's run of the compact slot array
  HXSlot* d_hx = nullptr;              // [precision][phase][slot]: 2 x 4 x max_slots descriptors
  int ns = 0, gram_ctas = 0, row_ctas = 0;
  int utiles = 0;                      // 128-row tiles of the complex64 slots (tcgen05 updates)
  int nsm = 148;
  // per precision (QDKP_C128, QDKP_C64): slots, the folded ones among them, H.X tiles
  int hx_ns[2] = {0, 0}, hx_folded[2] = {0, 0}, hx_tiles[2] = {0, 0};
  int m_max = 1;
  std::vector<int> widths;             // distinct block widths among the group's slots
};

// dynamic shared memory limits of the iteration's kernels, on the current device
void set_slot_kernel_limits();

// complex64 slots of the group are updated by the tcgen05 kernels
bool group_umma(const EGroup& G);

// An iteration: the decisions; the best iterate's copy and P's orthonormalisation beside R's residual
// block, projection and orthonormalisation and (the caller's) A R, a recomputed A X not before
// the residual block; then pencil, eigensolve and Ritz update.
int launch_decide(const EGroup& G, cudaStream_t st);
int launch_p_chain(const EGroup& G, cudaStream_t st);
int launch_r_chain(const EGroup& G, cudaStream_t st);
int launch_ritz_step(const EGroup& G, cudaStream_t st);

}  // namespace qdkp
