// sweep_wave.hpp — lock-step triangular sweeps: host-side interface.
//
// A sweep of a block triangular factor (ILU0: unit-L forward, U backward with
// the inverted diagonal; IChol0: L forward with L_ii^-1, L^T backward with
// L_ii^-T) computes, in the reference's natural row order,
//     x_r = D_r (rhs_r - sum_e B_e x_{j_e})
// (blocksp_preconditioners.hpp:294-349 ILU0::invmul, :432-489 IChol0::invmul),
// with D_r the identity for the unit-L sweep.  wave_plan.h lays every block
// the sweep reads out once, in the order the device consumes it (the blocks
// transposed where the sweep reads B^T, each premultiplied by its row's D:
// x_r = D_r rhs_r - sum_e (D_r B_e) x_{j_e}, the same operator).  What a row
// computes is unchanged; only when it runs and where its inputs come from
// differ from the reference's loop.
#pragma once
#include <memory>
#include <vector>
#include "internal.hpp"
#include "wave_shape.h"

namespace bsp {

// Symbolic part of one sweep (depends on the matrix pattern only).
struct WaveSym {
  int n = 0, bs = 0, n_super = 0, n_levels = 0, ne = 0;
  int64_t n_blk = 0;   // stored blocks
  int64_t n_item = 0;
  bool to_items = false;  // its result goes to the item order of the sweep that follows
  bool trans_blocks = false, has_d = false, trans_d = false;
  DevBuf<int> super_step, super_group, item_row, ext_row, blk_row;
  DevBuf<int> item_of;  // per row: the item that reads its right-hand side
  DevBuf<int2> step;
  DevBuf<int4> rec;
  DevBuf<int64_t> blk_src;
};

// Uploads a plan (wave_plan.h).  A sweep reads its right-hand side in item
// order; one that is followed by another writes its result in that one's item
// order: row_item is, per row, the item that reads it (null: natural order),
// and item_of receives that of this sweep.
int wave_upload(WavePlan&& P, int bs, bool trans_blocks, bool has_d, bool trans_d, const std::vector<int>* row_item,
                std::vector<int>* item_of, WaveSym& S);
// Values of a vector of one value set per item (1 right-hand side).
size_t wave_item_values(const WaveSym& S, int nrhs);

// The stream's values in one precision.
struct WaveVals {
  DevBuf<unsigned char> vals;
  bool valid = false;
};
size_t wave_val_bytes(const WaveSym& S, int prec);

// Gathers the stream's values (into a buffer of at least wave_val_bytes) from
// the factor (FP64, factor entry order) and the D blocks from dinv (FP64, row
// order), converted to the precision `prec` (BSP_PREC_F64 / F32 / BF16).  premul:
// the blocks of a sweep without D blocks are w D_r B_e all the same.
int wave_gather(bsp_handle_s* h, const WaveSym& S, int prec, const double* fvals, const double* dinv, WaveVals& out,
                bool premul = false, double w = 1.0);

// Start of z = M^-1 r through the sweeps lo, then up (z may alias r): rp = r in
// lo's item order, w (up's item order) and z filled with the sentinel.
int wave_prepare(bsp_handle_s* h, const WaveSym& lo, const WaveSym& up, const double* r, double* rp, double* w,
                 double* z);

// Start of one SOR sweep (blocksp_preconditioners.hpp:116-240): the part of
//   x_i = (1 - w) xold_i + w D_i (b_i - sum_j A_ij x_j)
// that does not depend on the sweep, in S's item order (the sums over rows that
// the sweep visits later, from xold; null: 0), and x filled with the sentinel (x
// may be b).  A's rows in the precision of the solve, D = inverted diagonals.
int wave_sor_prepare(bsp_handle_s* h, const WaveSym& S, int prec, bool forward, const int* row_ptr, const int* col,
                     const void* avals, const void* dinv, double w, const double* b, const double* xold, double* rp,
                     double* x);

// x = sweep(rhs) on h's stream, one right-hand side, FP64 vectors.  x must hold
// the sentinel on entry; the ticket must be 0 and is 0 again afterwards.
int wave_sweep(bsp_handle_s* h, const WaveSym& S, int prec, const WaveVals& V, const double* rhs, double* x,
               unsigned* ticket);

// The same with nrhs (1, 2 or 4) right-hand sides interleaved per row, FP64, a
// sweep with D blocks, 4 x 4, 8 x 8 or 16 x 16 blocks, on a stream of its own
// (it may be capturing).  Rows of a group whose group_active is 0 are skipped.
int wave_sweep_multi(bsp_handle_s* h, const WaveSym& S, const WaveVals& V, int nrhs, const double* rhs, double* x,
                     unsigned* ticket, const int* group_active, cudaStream_t stream);

}  // namespace bsp
