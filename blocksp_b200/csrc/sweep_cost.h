// sweep_cost.h — which kernel runs a triangular sweep (no CUDA).
//
// The lock-step kernel (sweep_wave.cuh) is far ahead where its super-tasks
// overlap (grids in grid order, bands, red-black rows) and far behind where
// they follow one another: its plan cuts the rows in their natural order, and
// with rows in another order (reverse Cuthill-McKee of a 3D grid, nested
// dissection, random) a super-task's first steps need the last rows of the one
// before.  Times of an application in us, lock-step | the kernel it replaced
// (streamed for 8 x 8 and 16 x 16 blocks, level-ordered polling otherwise):
//   64^3 in grid order, 4x4      227 |  1364     8x8     295 |  366
//   64^3 RCM, 4x4               4963 |  1605     8x8    6450 |  850
//   64^3 random, 4x4           24919 |   262     8x8   33005 | 1091
//   64^3 red-black, 4x4          317 |   243     8x8     460 |  998
//   300 x 257 RCM, 4x4          1449 |  2227     8x8    3557 |  968
//   40^3 27-point, 4x4         23621 |  6979     8x8   19861 | 3741
//   Delaunay mesh, 1e5 rows    10291 |   143     8x8   13691 |  477
// So both are estimated on the host when a pattern is first seen and the faster
// one is built: the lock-step sweep by WaveClock on its own plan, the others
// from the pattern by the model below.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>
#include "wave_plan.h"

namespace bsp {

enum class SweepKernel { kPolled, kStreamed };

// Time of a sweep that waits row by row: the longest dependency path, where an
// entry costs `all` and one more `late` when it reads a row of the level
// before (it is awaited), or the rows and entries over the whole GPU, whichever
// is longer.  us and ns, fitted to measured applications of 23 patterns of 4,000
// to 260,000 rows (grids, RCM, red-black, nested dissection, random, meshes,
// bands); rms of the logarithm 0.15 to 0.35.
struct SweepCost {
  double late, all, row_ns, entry_ns;
};
inline SweepCost sweep_cost_of(SweepKernel k, int bs) {
  if (k == SweepKernel::kStreamed) return bs == 8 ? SweepCost{0.25, 0.15, 0.8, 0.4} : SweepCost{0.15, 0.4, 2.7, 1.4};
  switch (bs) {
    case 1: return {0.7, 0.2, 0.9, 0.0};
    case 2: return {0.6, 0.75, 0.12, 0.0};
    case 3: return {1.0, 0.3, 1.0, 0.0};
    case 4: return {0.6, 0.5, 0.04, 0.14};
    case 5: return {1.3, 0.4, 1.1, 0.0};
    case 6: return {1.4, 0.45, 1.2, 0.0};
    case 8: return {0.2, 0.45, 1.3, 0.15};
    default: return {0.55, 0.6, 1.6, 0.3};
  }
}

// The model's time of a sweep over the rows of E in their natural order.
inline double sweep_cost_us(SweepKernel k, int bs, int n, bool ascending, const SweepEntries& E) {
  const SweepCost c = sweep_cost_of(k, bs);
  std::vector<int> level(n, 0);
  // entries along the longest path of levels that ends in a row: late ones, all
  struct Path {
    int late = 0, all = 0;
  };
  std::vector<Path> path(n);
  int late = 0, all = 0;
  for (int idx = 0; idx < n; ++idx) {
    const int i = ascending ? idx : n - 1 - idx;
    int lv = 0;
    for (int t = E.ptr[i]; t < E.ptr[i + 1]; ++t) lv = std::max(lv, level[E.col[t]] + 1);
    level[i] = lv;
    Path p;
    int here = 0;
    for (int t = E.ptr[i]; t < E.ptr[i + 1]; ++t) {
      const int j = E.col[t];
      if (level[j] != lv - 1) continue;
      ++here;
      p.late = std::max(p.late, path[j].late);
      p.all = std::max(p.all, path[j].all);
    }
    p.late += here;
    p.all += E.ptr[i + 1] - E.ptr[i];
    path[i] = p;
    late = std::max(late, p.late);
    all = std::max(all, p.all);
  }
  const double chain = c.late * late + c.all * all + 5.0;
  const double bulk = (c.row_ns * n + c.entry_ns * (double)E.col.size()) * 1e-3;
  return std::sqrt(chain * chain + bulk * bulk);
}

// The batched solver's level-ordered sweep (batch_sweep.cuh) with nrhs
// right-hand sides: a block is read once for all of them, the waits are longer.
inline double batch_sweep_cost_us(int bs, int nrhs, int n, bool ascending, const SweepEntries& E) {
  const double f = bs == 4 ? (nrhs == 1 ? 1.1 : 1.8) : bs == 8 ? (nrhs == 1 ? 1.2 : 1.9) : (nrhs == 1 ? 1.4 : 3.3);
  return f * sweep_cost_us(SweepKernel::kPolled, bs, n, ascending, E);
}

// The lock-step sweep is taken when it is estimated at less than this share of
// the other.  Over those patterns and eight block sizes it is then taken nowhere
// where it was measured slower by more than 1.2, but for one chain of 8 x 8 rows
// that also read far back (1.26); it is left where it was faster by at most 1.7
// (1 x 1 blocks of a renumbered mesh, SOR of 4 x 4 on a renumbered 27-point grid).
constexpr double kWaveShare = 0.9;

}  // namespace bsp
