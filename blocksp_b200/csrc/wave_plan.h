// wave_plan.h — the host layout of a lock-step triangular sweep (no CUDA).
//
// A sweep of a block triangular factor computes, in natural row order,
//     x_r = D_r rhs_r - sum_e (D_r B_e) x_{j_e}      (D = I for a unit factor)
// The plan cuts the rows into super-tasks (one CTA each) and every super-task
// into steps: the rows of a step depend only on rows of earlier steps of the
// same super-task and on rows of other super-tasks.  Inside a CTA the steps
// are separated by a barrier, so no row of the CTA is ever polled; only rows
// of other super-tasks ("external") are awaited, through global memory.
//   * chains are maximal runs of consecutive rows in which each row depends
//     on the one before; a super-task is a tile of wy consecutive chains by
//     wz chains one dominant chain stride apart (the neighbouring plane of a
//     grid), or consecutive chains when no stride links half of the chains;
//   * a step holds at most W items and ecap external rows.  An item is a row
//     with ne entries (2 when no row has more, else 3; absent ones are zero
//     blocks times the zero row); a longer row is cut into segments, each but
//     the last leaving its partial result in shared memory for the next;
//   * every operand of an item is a vector row in shared memory: one of the
//     results of the last `ring` steps, or of the `slots` steps staged ahead a
//     right-hand side or an external row.  An entry that reads a row of the
//     same super-task further back than the ring goes through global memory
//     like an external one (it was published before, so it never waits on its
//     own CTA's future);
//   * super-tasks are ordered by dependency level (the ticket order), so a
//     CTA waits only on tickets that were taken before its own.
// Rows of different groups (independent systems of a block-diagonal matrix)
// never share a super-task.
#pragma once
#include <algorithm>
#include <cstdint>
#include <functional>
#include <limits>
#include <map>
#include <numeric>
#include <queue>
#include <vector>

namespace bsp {

constexpr int kWaveMinRows = 1024;  // rows of a super-task of short chains
constexpr int kWaveHop = 4;         // steps that a hand-off between super-tasks takes

// The entries of a sweep in CSR form: row i reads rows col[t] through the
// factor blocks blk[t], t in [ptr[i], ptr[i+1]).
struct SweepEntries {
  std::vector<int> ptr, col;
  std::vector<int64_t> blk;
};

struct WaveShape {
  int W = 0;      // items per step
  int ecap = 0;   // external rows per step
  int ring = 0;   // steps whose results stay in shared memory
  int slots = 0;  // steps whose right-hand sides and external rows are staged
  bool item_major = false;  // order of a step's blocks, see WaveStep
  int fetch = 2;            // warps that bring in external rows, a step each in turn
  double step_us = 0.3;     // time of a step that waits for nothing
  // vector rows in shared memory, in this order
  int n_rows() const { return ring * W + 1 + slots * (W + ecap); }
  int result(int step, int item) const { return step % ring * W + item; }
  int zero() const { return ring * W; }
  int rhs(int step, int item) const { return ring * W + 1 + step % slots * W + item; }
  int ext(int step, int e) const { return ring * W + 1 + slots * W + step % slots * ecap + e; }
};

// One item: the vector rows of its base operand (its right-hand side, or the
// partial result it continues) and of its entries, and the row it completes
// (-1: a partial result).
struct WaveRec {
  uint32_t base_c0, c1_c2;
  int32_t row;
  uint32_t pad;
};

// Step t covers items [item0, next.item0) and external rows [ext0, next.ext0).
// Its values start at block item0 * (ne + has_d): item by item, the D block
// (when has_d) and the entries (item_major: a block is at least 128 bytes), or
// first the D blocks of all its items, then their first entries, and so on
// (small blocks: lanes of neighbouring items read neighbouring blocks).
struct WaveStep {
  int32_t item0, ext0;
};

// What a stored block holds: a factor block (>= 0), or
constexpr int64_t kWaveD = -1;     // the row's D block
constexpr int64_t kWaveZero = -2;  // zeros (an absent entry)
constexpr int64_t kWaveOne = -3;   // the identity (D of a continued row)

struct WavePlan {
  int n = 0, n_super = 0, n_levels = 0;
  int ne = 0;                    // entries of an item
  bool over_limit = false;       // given up: its estimate passed the caller's limit
  double est_us = 0.0;           // estimated time of the sweep, see WaveClock
  std::vector<int> super_step;   // n_super + 1
  std::vector<int> super_group;  // group of each super-task
  std::vector<WaveStep> step;    // all steps + 1
  std::vector<WaveRec> rec;      // per item
  std::vector<int> item_row;     // per item: the row of its right-hand side (-1: continued)
  std::vector<int> ext_row;
  std::vector<int64_t> blk_src;  // per stored block
  std::vector<int> blk_row;
};

namespace wave_detail {

constexpr int kMaxEnt = 3;

struct Item {
  int row;
  bool cont, last;
  int base, c[kMaxEnt];
  int64_t blk[kMaxEnt];
};

// Super-tasks of rows [r0, r1): lists of rows in sweep order, with levels.
struct Supers {
  std::vector<std::vector<int>> rows;
  std::vector<int> level;
};

inline bool group_rows(int r0, int r1, bool ascending, const WaveShape& S, const SweepEntries& E,
                       std::vector<int>& sup_of, int sup_base, Supers& out) {
  const int n = r1 - r0, dir = ascending ? 1 : -1;
  std::vector<int> chain_of(n), first, clen;
  for (int idx = 0; idx < n; ++idx) {
    const int r = ascending ? r0 + idx : r1 - 1 - idx;
    const int pr = r - dir;
    bool cont = false;
    if (idx > 0)
      for (int t = E.ptr[r]; t < E.ptr[r + 1]; ++t) cont |= (E.col[t] == pr);
    if (cont) {
      chain_of[r - r0] = chain_of[pr - r0];
      clen[chain_of[pr - r0]]++;
    } else {
      chain_of[r - r0] = (int)first.size();
      first.push_back(r);
      clen.push_back(1);
    }
  }
  const int nc = (int)first.size();
  // distinct predecessor chains of every chain, and their strides
  std::vector<std::vector<int>> cdeps(nc);
  std::vector<int> stride_count(nc + 1, 0);
  for (int c = 0; c < nc; ++c) {
    auto& dc = cdeps[c];
    for (int k = 0; k < clen[c]; ++k) {
      const int r = first[c] + k * dir;
      for (int t = E.ptr[r]; t < E.ptr[r + 1]; ++t)
        if (chain_of[E.col[t] - r0] != c) dc.push_back(chain_of[E.col[t] - r0]);
    }
    std::sort(dc.begin(), dc.end());
    dc.erase(std::unique(dc.begin(), dc.end()), dc.end());
    for (int cj : dc)
      if (c - cj >= 2) stride_count[c - cj]++;
  }
  std::vector<int> sup(nc), lvl;
  std::vector<std::vector<int>> members;
  int nsup = 0;
  // super-tasks from a key per chain; false when their graph has a cycle
  auto build = [&](auto key_of) {
    std::map<int64_t, int> ids;
    for (int c = 0; c < nc; ++c) {
      auto it = ids.find(key_of(c));
      if (it == ids.end()) it = ids.emplace(key_of(c), (int)ids.size()).first;
      sup[c] = it->second;
    }
    nsup = (int)ids.size();
    members.assign(nsup, {});
    for (int c = 0; c < nc; ++c) members[sup[c]].push_back(c);
    std::vector<std::vector<int>> succ(nsup);
    std::vector<int> indeg(nsup, 0), queue;
    for (int c = 0; c < nc; ++c)
      for (int cj : cdeps[c])
        if (sup[cj] != sup[c]) succ[sup[cj]].push_back(sup[c]);
    for (auto& v : succ) {
      std::sort(v.begin(), v.end());
      v.erase(std::unique(v.begin(), v.end()), v.end());
      for (int b : v) indeg[b]++;
    }
    lvl.assign(nsup, 0);
    for (int a = 0; a < nsup; ++a)
      if (!indeg[a]) queue.push_back(a);
    for (size_t h = 0; h < queue.size(); ++h) {
      const int a = queue[h];
      for (int b : succ[a]) {
        lvl[b] = std::max(lvl[b], lvl[a] + 1);
        if (--indeg[b] == 0) queue.push_back(b);
      }
    }
    return (int)queue.size() == nsup;
  };
  int dom = 0, dom_n = 0;
  for (int d = 2; d <= nc; ++d)
    if (stride_count[d] > dom_n) {
      dom = d;
      dom_n = stride_count[d];
    }
  int wz = 1;
  while (wz * wz * 4 <= S.W) wz *= 2;  // 16 -> 4 x 4, 8 -> 4 x 2, 64 -> 8 x 8
  const int wy = S.W / wz;
  bool ok = false;
  if (wz > 1 && dom >= 2 && dom_n * 2 >= nc) {
    const int cols = (dom + wy - 1) / wy;
    ok = build([&](int c) { return (int64_t)(c / (wz * dom)) * cols + (c % dom) / wy; });
  }
  if (!ok) {
    // consecutive chains (a chain never depends on a later one): W, whose
    // super-tasks follow one another a few steps apart, or with short chains
    // enough for kWaveMinRows rows, W at a time and one super-task after the
    // other.  Whichever takes fewer steps (80 x 80 rows of 16 x 16 blocks, W = 8:
    // 13 chains to a super-task took 605 us an application, 8 take 190)
    const int64_t most = std::max<int64_t>(S.W, ((int64_t)kWaveMinRows * nc + n - 1) / std::max(n, 1));
    const double len = (double)n / std::max(nc, 1), turns = (double)nc / S.W;
    const double steps_w = len + nc + kWaveHop * turns, steps_most = turns * len + S.W + kWaveHop * nc / most;
    const int64_t per = steps_w < steps_most ? S.W : most;
    ok = build([&](int c) { return (int64_t)c / per; });
  }
  if (!ok) return false;
  out.rows.assign(nsup, {});
  for (int idx = 0; idx < n; ++idx) {  // sweep order: dependencies first
    const int r = ascending ? r0 + idx : r1 - 1 - idx;
    const int s = sup[chain_of[r - r0]];
    sup_of[r] = sup_base + s;
    out.rows[s].push_back(r);
  }
  out.level = std::move(lvl);
  return true;
}

// Estimated time of a sweep: the CTAs take super-tasks in ticket order; a step
// starts when the one before is over and its external rows are there, which a
// fetch warp reads in about kFetchUs when they are published already and
// kHopUs after they are published otherwise.  Fitted to measured applications
// (step times per block size in wave_shape.h): within 20 % on most of 23
// patterns and 8 block sizes, grids and random orders alike; grids bound by
// bandwidth are up to 40 % slower than it says.
constexpr int kClockCtas = 148;
constexpr double kStartUs = 1.5, kHopUs = 1.2, kFetchUs = 0.8;
class WaveClock {
  std::vector<double> done_, fetch_;
  std::priority_queue<double, std::vector<double>, std::greater<double>> cta_;

 public:
  double end = 0.0;
  WaveClock(int n, const WaveShape& S) : done_(n, 0.0), fetch_(S.fetch, 0.0) {
    for (int i = 0; i < kClockCtas; ++i) cta_.push(0.0);
  }
  // the last super-task of P, its steps from `first` on
  void super_task(const WavePlan& P, const WaveShape& S, size_t first) {
    double now = cta_.top() + kStartUs;
    cta_.pop();
    std::fill(fetch_.begin(), fetch_.end(), now);
    for (size_t s = first; s < P.step.size(); ++s) {
      const bool last = s + 1 == P.step.size();
      const size_t i1 = last ? P.rec.size() : P.step[s + 1].item0, e1 = last ? P.ext_row.size() : P.step[s + 1].ext0;
      if ((size_t)P.step[s].ext0 < e1) {
        double there = 0.0;
        for (size_t e = P.step[s].ext0; e < e1; ++e) there = std::max(there, done_[P.ext_row[e]]);
        double& f = fetch_[(s - first) % fetch_.size()];
        f = std::max(f + kFetchUs, there + kHopUs);
        now = std::max(now, f);
      }
      now += S.step_us;
      for (size_t i = P.step[s].item0; i < i1; ++i)
        if (P.rec[i].row >= 0) done_[P.rec[i].row] = now;
    }
    cta_.push(now);
    end = std::max(end, now);
  }
};

}  // namespace wave_detail

// The layout of a sweep over n rows; ascending: forward (dependencies j < i),
// else backward.  has_d: rows carry a D block.  group_beg: first row of every
// independent group, then n (empty: one group).  False when the dependencies
// are not triangular, the stream is too long, or the sweep would take more than
// limit_us (over_limit; planning stops there).
inline bool wave_plan(int n, bool ascending, const WaveShape& S, bool has_d, const SweepEntries& E,
                      const std::vector<int>& group_beg, WavePlan& P,
                      double limit_us = std::numeric_limits<double>::infinity()) {
  using namespace wave_detail;
  P = WavePlan{};
  P.n = n;
  P.ne = 2;
  std::vector<int> gb = group_beg;
  if (gb.empty()) gb = {0, n};
  for (int i = 0; i < n; ++i) {
    if (E.ptr[i + 1] - E.ptr[i] > 2) P.ne = 3;
    for (int t = E.ptr[i]; t < E.ptr[i + 1]; ++t)
      if (ascending ? E.col[t] >= i : E.col[t] <= i) return false;
  }
  const int NE = P.ne;
  std::vector<int> sup_of(n, -1);
  struct Sup {
    std::vector<int> rows;
    int level, group;
  };
  std::vector<Sup> sups;
  for (size_t g = 0; g + 1 < gb.size(); ++g) {
    Supers one;
    if (gb[g] == gb[g + 1]) continue;
    if (!group_rows(gb[g], gb[g + 1], ascending, S, E, sup_of, (int)sups.size(), one)) return false;
    for (size_t k = 0; k < one.rows.size(); ++k) sups.push_back({std::move(one.rows[k]), one.level[k], (int)g});
  }
  std::vector<int> order(sups.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return sups[a].level < sups[b].level; });
  P.n_super = (int)sups.size();
  P.super_step.push_back(0);
  const int lag = S.ring - 1;  // furthest step a result in shared memory may lie back
  std::vector<int> r_step(n, -1), r_item(n, -1);  // step and item that complete a row
  std::vector<std::vector<Item>> st;
  std::vector<std::vector<int>> ext;
  std::vector<std::pair<int, int>> ord, seg;  // (step of the dependency or -1, entry); (first, count)
  std::vector<int> at;
  WaveClock clock(n, S);
  for (int sid : order) {
    const Sup& sp = sups[sid];
    P.n_levels = std::max(P.n_levels, sp.level + 1);
    size_t used = 0;  // steps of this super-task: their lists keep what they held room for
    // steps before room[k] are full, or have no room for k external rows (both
    // only fill up): without it a row of external rows passes over every step
    size_t room[kMaxEnt + 1] = {};
    for (int r : sp.rows) {
      ord.clear();
      int lo = 0;
      for (int t = E.ptr[r]; t < E.ptr[r + 1]; ++t) {
        const int j = E.col[t];
        const int s = sup_of[j] == sid ? r_step[j] : -1;
        ord.emplace_back(s, t);
        lo = std::max(lo, s + 1);
      }
      // few entries: by insertion (a stable sort would allocate for every row)
      for (size_t a = 1; a < ord.size(); ++a)
        for (size_t b = a; b > 0 && ord[b].first < ord[b - 1].first; --b) std::swap(ord[b], ord[b - 1]);
      const int ne = (int)ord.size();
      seg.clear();
      for (int f = 0; f == 0 || f < ne; f += NE) seg.emplace_back(f, std::min(ne - f, NE));
      const int ns = (int)seg.size();
      // whether the external rows of a segment at step s fit
      auto ext_fit = [&](int s, const std::pair<int, int>& sg) {
        const int have = s < (int)used ? (int)ext[s].size() : 0;
        int need = 0;
        for (int u = 0; u < sg.second; ++u) {
          const auto& o = ord[sg.first + u];
          if (o.first < 0 || s - o.first > lag) ++need;
        }
        return need == 0 || have + need <= S.ecap;
      };
      // external rows of the first segment wherever it goes
      int far = 0;
      while (far < seg[0].second && ord[far].first < 0) ++far;
      size_t& hint = room[far];
      while (hint < used && ((int)st[hint].size() >= S.W || (far > 0 && (int)ext[hint].size() + far > S.ecap))) ++hint;
      at.assign(ns, 0);
      for (int base = std::max({lo - ns + 1, 0, (int)hint});; ++base) {
        bool good = true;
        int s = base;
        for (int k = 0; k < ns && good; ++k) {
          for (int u = 0; u < seg[k].second; ++u) s = std::max(s, ord[seg[k].first + u].first + 1);
          while ((s < (int)used && (int)st[s].size() >= S.W) || !ext_fit(s, seg[k])) ++s;
          if (k > 0 && s - at[k - 1] > lag) good = false;
          at[k] = s++;
        }
        if (good) break;
      }
      for (; (int)used <= at[ns - 1]; ++used) {
        if (used == st.size()) {
          st.emplace_back();
          ext.emplace_back();
        }
        st[used].clear();
        ext[used].clear();
      }
      int prev_item = 0;
      for (int k = 0; k < ns; ++k) {
        const int s = at[k], item = (int)st[s].size();
        Item it;
        it.row = r;
        it.cont = k > 0;
        it.last = k == ns - 1;
        it.base = k > 0 ? S.result(at[k - 1], prev_item) : S.rhs(s, item);
        for (int u = 0; u < kMaxEnt; ++u) {
          it.c[u] = S.zero();
          it.blk[u] = kWaveZero;
        }
        for (int u = 0; u < seg[k].second; ++u) {
          const auto& o = ord[seg[k].first + u];
          const int j = E.col[o.second];
          it.blk[u] = E.blk[o.second];
          if (o.first >= 0 && s - o.first <= lag) {
            it.c[u] = S.result(o.first, r_item[j]);
          } else {
            auto& x = ext[s];
            const int p = (int)(std::find(x.begin(), x.end(), j) - x.begin());
            if (p == (int)x.size()) x.push_back(j);
            it.c[u] = S.ext(s, p);
          }
        }
        prev_item = item;
        st[s].push_back(it);
      }
      r_step[r] = at[ns - 1];
      r_item[r] = prev_item;
    }
    // flatten
    const size_t first_step = P.step.size();
    for (size_t s = 0; s < used; ++s) {
      P.step.push_back({(int32_t)P.rec.size(), (int32_t)P.ext_row.size()});
      for (const Item& it : st[s]) {
        P.rec.push_back({(uint32_t)it.base | (uint32_t)it.c[0] << 16, (uint32_t)it.c[1] | (uint32_t)it.c[2] << 16,
                         it.last ? it.row : -1, 0u});
        P.item_row.push_back(it.cont ? -1 : it.row);
      }
      auto put = [&](const Item& it, int u) {
        P.blk_src.push_back(u >= 0 ? it.blk[u] : it.cont ? kWaveOne : kWaveD);
        P.blk_row.push_back(it.row);
      };
      const int u0 = has_d ? -1 : 0;
      if (S.item_major) {
        for (const Item& it : st[s])
          for (int u = u0; u < NE; ++u) put(it, u);
      } else {
        for (int u = u0; u < NE; ++u)
          for (const Item& it : st[s]) put(it, u);
      }
      P.ext_row.insert(P.ext_row.end(), ext[s].begin(), ext[s].end());
    }
    P.super_step.push_back((int)P.step.size());
    P.super_group.push_back(sp.group);
    if (P.blk_src.size() >= (size_t)INT32_MAX || P.ext_row.size() >= (size_t)INT32_MAX) return false;
    clock.super_task(P, S, first_step);
    P.est_us = clock.end;
    if (clock.end > limit_us) {
      P.over_limit = true;
      return false;
    }
  }
  P.step.push_back({(int32_t)P.rec.size(), (int32_t)P.ext_row.size()});
  return S.n_rows() <= 0xffff;
}

}  // namespace bsp
