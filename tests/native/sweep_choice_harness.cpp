// The shapes of the lock-step sweep and the choice of a sweep's kernel
// (csrc/wave_shape.h, csrc/sweep_cost.h) on the host.
#include "../../blocksp_b200/csrc/sweep_cost.h"
#include "../../blocksp_b200/csrc/wave_shape.h"

using namespace bsp;

// W, external rows, ring, slots, item-major, fetch warps of a block size.
extern "C" void sweep_shape(int bs, int nrhs, int* out) {
  const WaveShape s = wave_shape(bs, nrhs);
  const int v[6] = {s.W, s.ecap, s.ring, s.slots, s.item_major, s.fetch};
  std::copy(v, v + 6, out);
}

// 1 when the lock-step sweep is taken; out: its estimate, the other kernel's,
// super-tasks, their levels and steps planned before it was given up.  Rows of
// different groups (n_group + 1 first rows) are independent systems.  The other
// kernel: 0 level-ordered, 1 streamed, 2 the batched solver's.
extern "C" int sweep_choice(int n, int ascending, int bs, int nrhs, int other_kernel, int limited, const int* ptr,
                            const int* col, int n_group, const int* group_beg, double* out) {
  SweepEntries E;
  E.ptr.assign(ptr, ptr + n + 1);
  E.col.assign(col, col + ptr[n]);
  for (int t = 0; t < ptr[n]; ++t) E.blk.push_back(t);
  const double other =
      other_kernel == 2
          ? batch_sweep_cost_us(bs, nrhs, n, ascending != 0, E)
          : sweep_cost_us(other_kernel ? SweepKernel::kStreamed : SweepKernel::kPolled, bs, n, ascending != 0, E);
  WavePlan P;
  const std::vector<int> gb(group_beg, group_beg + (n_group ? n_group + 1 : 0));
  const double limit = kWaveShare * other;
  const bool ok = limited ? wave_plan(n, ascending != 0, wave_shape(bs, nrhs), true, E, gb, P, limit)
                          : wave_plan(n, ascending != 0, wave_shape(bs, nrhs), true, E, gb, P) && P.est_us <= limit;
  const double v[5] = {P.est_us, other, (double)P.n_super, (double)P.n_levels, (double)P.step.size()};
  std::copy(v, v + 5, out);
  return ok;
}
