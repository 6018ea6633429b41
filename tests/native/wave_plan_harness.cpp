// Runs a lock-step sweep plan (csrc/wave_plan.h) on the host the way the
// kernel does: super-tasks in ticket order, steps in order, every operand a
// row of the CTA's vector memory, every limit checked.
#include <limits>
#include "../../blocksp_b200/csrc/wave_plan.h"

using namespace bsp;

// Returns 0, or a positive code for the first rule that the plan breaks.
// x (n * bs) receives the sweep's result; stats: super-tasks, steps, items,
// external rows, levels, entries of an item.
extern "C" int wave_plan_run(int n, int ascending, int bs, int W, int ecap, int ring, int slots, int has_d, int item_major,
                             const int* ptr, const int* col, const double* vals, const double* dinv,
                             const double* rhs, int n_group, const int* group_beg, double* x, int* stats) {
  SweepEntries E;
  E.ptr.assign(ptr, ptr + n + 1);
  E.col.assign(col, col + ptr[n]);
  for (int t = 0; t < ptr[n]; ++t) E.blk.push_back(t);
  WaveShape S;
  S.W = W;
  S.ecap = ecap;
  S.ring = ring;
  S.slots = slots;
  S.item_major = item_major != 0;
  WavePlan P;
  std::vector<int> gb(group_beg, group_beg + n_group);
  if (!wave_plan(n, ascending != 0, S, has_d != 0, E, gb, P)) return 1;
  const int b2 = bs * bs, NE = P.ne, NB = NE + (has_d ? 1 : 0);
  const double nan = std::numeric_limits<double>::quiet_NaN();
  std::vector<char> done(n, 0), rhs_used(n, 0);
  std::vector<double> mem((size_t)S.n_rows() * bs);
  if (P.super_step.front() != 0 || P.super_step.back() + 1 != (int)P.step.size()) return 2;
  if (P.blk_src.size() != P.rec.size() * NB || P.blk_row.size() != P.blk_src.size()) return 17;
  for (int task = 0; task < P.n_super; ++task) {
    const int t0 = P.super_step[task], T = P.super_step[task + 1] - t0;
    std::fill(mem.begin(), mem.end(), nan);
    std::fill(mem.begin() + (size_t)S.zero() * bs, mem.begin() + (size_t)(S.zero() + 1) * bs, 0.0);
    // the copies of step t: into its own slot, while later slots hold later steps
    auto stage = [&](int t) -> int {
      const WaveStep a = P.step[t0 + t], b = P.step[t0 + t + 1];
      const int cnt = b.item0 - a.item0, next = b.ext0 - a.ext0;
      if (cnt < 0 || cnt > W || next < 0 || next > ecap) return 3;
      for (int k = 0; k < cnt; ++k) {
        const int r = P.item_row[a.item0 + k];
        if (r >= 0) std::copy(rhs + (size_t)r * bs, rhs + (size_t)(r + 1) * bs, mem.begin() + (size_t)S.rhs(t, k) * bs);
      }
      return 0;
    };
    for (int t = 0; t < std::min(T, slots - 1); ++t)
      if (int e = stage(t)) return e;
    for (int t = 0; t < T; ++t) {
      // slot t - 1 is free once step t has begun: one step ahead of it is filled
      if (t + slots - 1 < T)
        if (int e = stage(t + slots - 1)) return e;
      const WaveStep a = P.step[t0 + t], b = P.step[t0 + t + 1];
      const int cnt = b.item0 - a.item0, next = b.ext0 - a.ext0;
      for (int e = 0; e < next; ++e) {
        const int r = P.ext_row[a.ext0 + e];
        if (!done[r]) return 4;  // would wait on a row that is not published yet
        std::copy(x + (size_t)r * bs, x + (size_t)(r + 1) * bs, mem.begin() + (size_t)S.ext(t, e) * bs);
      }
      std::vector<double> out((size_t)cnt * bs);
      for (int k = 0; k < cnt; ++k) {
        const WaveRec& rc = P.rec[a.item0 + k];
        const unsigned code[4] = {rc.base_c0 & 0xffffu, rc.base_c0 >> 16, rc.c1_c2 & 0xffffu, rc.c1_c2 >> 16};
        const int hr = P.item_row[a.item0 + k];
        auto block = [&](int b) { return (size_t)a.item0 * NB + (item_major ? (size_t)k * NB + b : (size_t)b * cnt + k); };
        const int row = P.blk_row[block(0)];
        if (row < 0 || row >= n || (rc.row != -1 && rc.row != row) || (hr != -1 && hr != row)) return 5;
        if (hr >= 0 && (rhs_used[row]++ || (int)code[0] != S.rhs(t, k))) return 6;
        std::vector<double> v(bs, 0.0);
        for (int u = 0; u <= NE; ++u) {
          const int c = (int)code[u];
          if (c >= S.n_rows()) return 7;
          if (c < ring * W && c / W == t % ring) return 8;  // this step's results replace that row
          const double* xv = mem.data() + (size_t)c * bs;
          int64_t src = kWaveOne;
          if (u > 0 || has_d) {
            const size_t at = block(has_d ? u : u - 1);
            if (P.blk_row[at] != row) return 9;
            src = P.blk_src[at];
          }
          if (u == 0 && has_d && src != (hr >= 0 ? kWaveD : kWaveOne)) return 10;
          if (u > 0 && !(src >= 0 || (src == kWaveZero && c == S.zero()))) return 11;
          for (int r = 0; r < bs; ++r)
            for (int q = 0; q < bs; ++q) {
              double m = r == q ? 1.0 : 0.0;
              if (src == kWaveD) {
                m = dinv[(size_t)row * b2 + r * bs + q];
              } else if (src == kWaveZero) {
                m = 0.0;
              } else if (src >= 0) {
                m = 0.0;
                if (has_d)
                  for (int z = 0; z < bs; ++z) m -= dinv[(size_t)row * b2 + r * bs + z] * vals[src * b2 + z * bs + q];
                else
                  m = -vals[src * b2 + r * bs + q];
              }
              v[r] += m * xv[q];
            }
        }
        std::copy(v.begin(), v.end(), out.begin() + (size_t)k * bs);
      }
      for (int k = 0; k < cnt; ++k) {
        const WaveRec& rc = P.rec[a.item0 + k];
        std::copy(out.begin() + (size_t)k * bs, out.begin() + (size_t)(k + 1) * bs,
                  mem.begin() + (size_t)S.result(t, k) * bs);
        if (rc.row >= 0) {
          if (done[rc.row]++) return 15;
          std::copy(out.begin() + (size_t)k * bs, out.begin() + (size_t)(k + 1) * bs, x + (size_t)rc.row * bs);
        }
      }
    }
  }
  for (int i = 0; i < n; ++i)
    if (!done[i] || !rhs_used[i]) return 16;
  const int s[6] = {P.n_super, (int)P.step.size() - 1, (int)P.rec.size(), (int)P.ext_row.size(), P.n_levels, P.ne};
  std::copy(s, s + 6, stats);
  return 0;
}
