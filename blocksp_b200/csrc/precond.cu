// precond.cu — block Diag / SOR / ILU0 / IChol0 preconditioners on sm_100a.
//
// Reference: blocksp_preconditioners.hpp (BlockSp v1.0).
//   makeADInv            :22-63   -> k_factor mode DIAG (inverted diagonal blocks)
//   Diag                 :75-111  -> sweep with no off-diagonal entries, POST_D
//   SOR                  :116-240 -> nu sync-free forward / backward sweeps from x = 0
//   ILU0::factor         :274-291 -> k_factor mode ILU0 (row-wise, level scheduled)
//   ILU0::invmul         :294-349 -> unit-L forward sweep + U backward sweep
//                                    (sweep_wave.cu, sweep_stream.cu or here, by
//                                    the pattern: sweep_cost.h)
//   IChol0::factor       :393-429 -> k_factor mode ICHOL0
//   IChol0::invmul       :432-489 -> L forward sweep + L^T backward sweep
//
// Method preservation: every sweep and factorisation runs in the reference's
// natural row order.  Rows are only *scheduled* by dependency level (a row
// starts once every row it reads is final), which changes when a row is
// computed but not what it computes, so the preconditioner is the same
// operator as the reference's (no recolouring, no reordering).
//
// Sync-free execution: a sweep launch is persistent; each group of lanes
// claims the next task (a chain of consecutive dependent rows, in chain-level
// order) with an atomic ticket.  The output vector is pre-filled with a
// signalling-NaN sentinel and a row is published by its values: a consumer
// polls the words it needs (bounded spin) until they differ from the
// sentinel, so no flag or fence is involved.  A task only waits on rows of
// tasks with smaller tickets, which were claimed by groups that are already
// running, so the launch always progresses without any co-residency
// requirement.  The factorisation uses per-row ready flags that hold the
// epoch of the launch that last wrote them, so they never need clearing.
//
// A row's own inputs are staged ahead of it, so only the cross-chain values
// remain on the dependency path: each group keeps a shared-memory ring with
// the chain's next D rows (matrix blocks, inverted diagonal, right-hand side,
// old iterate), filled by per-lane cp.async copies; the chain's structure
// (entry ranges, column and block indices) is loaded one window of G rows
// ahead, one row per lane, and handed out by shuffles; the chain's previous
// row is passed on in registers.
//
// The factorisation is row-oriented (IKJ): row k applies the eliminations of
// rows i < k in increasing i, exactly the sequence of updates the reference's
// right-looking loop applies to each block (k, j), so the factors are the same.
#include <algorithm>
#include <atomic>
#include <numeric>
#include "blockops.cuh"
#include "per_device.h"
#include "precond.hpp"
#include "reduce.cuh"
#include "sentinel.cuh"
#include "stage.cuh"
#include "sweep_plan.hpp"

namespace bsp {

// ----------------------------------------------------------------- device wait
__device__ __forceinline__ void wait_flag(const int* f, int epoch, DevStatus* st, int who, unsigned limit) {
  if (ld_acquire(f) == epoch) return;
  unsigned spins = 0;
  while (ld_acquire(f) != epoch) {
    if (++spins > limit) {
      set_status(st, BSP_TIMEOUT, who);
      return;
    }
    if ((spins & 255u) == 0u && *reinterpret_cast<volatile int*>(&st->code) != 0) return;  // already failed
    poll_pause(spins);
  }
}

__global__ void k_fill_sentinel64(int64_t n, unsigned long long* __restrict__ x) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = kSentinel64;
}
__global__ void k_fill_sentinel32(int64_t n, unsigned* __restrict__ x) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = kSentinel32;
}

// ----------------------------------------------------------------- sweeps
enum { RANGE_LOWER = 0, RANGE_UPPER = 1, RANGE_SPLIT = 2, RANGE_ALL = 3, RANGE_NONE = 4 };
enum { POST_NONE = 0, POST_D = 1, POST_DT = 2, POST_SOR = 3 };

template <typename VT, typename AT> struct SweepP {
  int n;
  const int* order;     // processing order (null: identity)
  const int* ptr;       // row pointer of the structure swept
  const int* idx;       // column (transposed structure: source row) of each entry
  const int64_t* blk;   // block index of each entry (null: the entry index)
  const int* diag;      // position of the diagonal entry of each row
  int range;            // RANGE_*
  int dep_dir;          // RANGE_SPLIT: -1 deps are j < i (forward), +1 deps are j > i
  const VT* vals;
  const VT* dinv;
  const AT* rhs;
  const AT* xold;       // POST_SOR / RANGE_SPLIT: iterate before the sweep (null: zero)
  AT* x;
  AT w;
  int* flags;
  int epoch;
  unsigned* ticket;
  DevStatus* st;
  unsigned spin_limit;  // polls before a wait gives up with BSP_TIMEOUT
  // Chains: task t covers rows task_row[t], task_row[t] + task_dir, ... (task_len[t]
  // rows), each depending on the one before it; the group keeps the previous
  // row's result in shared memory instead of waiting for its flag.  Null
  // task_row: one row per task, taken from `order`.
  const int* task_row;
  const int* task_len;
  int task_dir;
  int n_tasks;
  int stage_vec;  // rhs and xold are 16-byte aligned: staged with the blocks (set at launch)
};

template <typename VT, typename AT>
__device__ __forceinline__ void row_range(const SweepP<VT, AT>& p, int i, int& beg, int& end) {
  switch (p.range) {
    case RANGE_LOWER: beg = __ldg(p.ptr + i); end = __ldg(p.diag + i); break;
    case RANGE_UPPER: beg = __ldg(p.diag + i) + 1; end = __ldg(p.ptr + i + 1); break;
    case RANGE_NONE: beg = end = 0; break;
    default: beg = __ldg(p.ptr + i); end = __ldg(p.ptr + i + 1); break;
  }
}

constexpr int kSweepThreads = 256;
constexpr int kSlotBudget = 12288;  // staging bytes per group of lanes

// Shared-memory ring of one group of lanes: D slots, each holding one row's
// first NPF blocks, its inverted diagonal block, right-hand side and old
// iterate, filled by per-lane asynchronous copies D rows ahead of their use.
// Every lane copies exactly the 16-byte chunks (and vector values) it reads
// later, so a lane only ever waits for its own copies.
template <int BS, typename VT, typename AT, bool TRANS, int POST> struct SweepCfg {
  using M = BlockMap<BS, VT>;
  static constexpr int G = M::G, P = M::P, CPB = M::CPB;
  static constexpr int GPC = kSweepThreads / G;
  static constexpr int NPF = (P == 1) ? 4 : (P == 2 ? 2 : 1);  // entries staged per row
  static constexpr bool kUseD = POST != POST_NONE;
  static constexpr int XR = TRANS ? M::V : P;          // rhs values a lane reads per row
  static constexpr int BB = CPB * 16;                  // bytes of one block
  static constexpr int LRB = XR * (int)sizeof(AT);     // rhs bytes of one lane
  static_assert(!TRANS || LRB % 16 == 0, "transposed rhs pieces are whole 16-byte chunks");
  static constexpr int OFF_D = NPF * BB;
  static constexpr int OFF_R = OFF_D + (kUseD ? BB : 0);
  static constexpr int OFF_O = OFF_R + (G * LRB + 15) / 16 * 16;
  static constexpr int SB = OFF_O + (POST == POST_SOR ? (G * P * (int)sizeof(AT) + 15) / 16 * 16 : 0);
  static constexpr int D0 = (4 * SB <= kSlotBudget) ? 4 : (3 * SB <= kSlotBudget ? 3 : 2);
  static constexpr int D = D0 < G ? D0 : G;  // lookahead stays within the next structure window
  static constexpr size_t kSmem = (size_t)GPC * D * SB;
};

template <int BS, typename VT, typename AT, bool TRANS, int POST>
__global__ void __launch_bounds__(kSweepThreads) k_sweep(const SweepP<VT, AT> p) {
  // Launch parameters used on the per-row path, held in registers.
  const int* __restrict__ const idx_ = p.idx;
  const int64_t* __restrict__ const blk_ = p.blk;
  const int range_ = p.range, dep_dir_ = p.dep_dir, task_dir_ = p.task_dir;
  const VT* __restrict__ const dinv_ = p.dinv;
  const AT* __restrict__ const rhs_ = p.rhs;
  const AT* __restrict__ const xold_ = p.xold;
  AT* const x_ = p.x;
  const AT w_ = p.w;
  DevStatus* const st_ = p.st;
  using M = BlockMap<BS, VT>;
  using C = SweepCfg<BS, VT, AT, TRANS, POST>;
  using CV = typename Chunk<VT>::vec;
  constexpr int V = M::V, G = M::G, P = M::P, CPR = M::CPR, RPP = M::RPP, CPB = M::CPB;
  constexpr int GPC = C::GPC, NPF = C::NPF, D = C::D, SB = C::SB, BB = C::BB;
  constexpr bool kUseD = C::kUseD;
  constexpr int XV = TRANS ? P : V;  // x values a lane reads per entry
  constexpr int XR = TRANS ? V : P;  // rhs values a lane reads per row
  extern __shared__ __align__(128) unsigned char sweep_smem[];
  __shared__ AT sm_s[GPC][BS];
  __shared__ AT sm_x[GPC][BS];  // the group's previous row of its chain
  const int gl = threadIdx.x % G;
  const int gid = threadIdx.x / G;
  const int lane = threadIdx.x & 31;
  const int gbase = lane - gl;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << gbase);
  const int c0 = (gl % CPR) * V;
  const CV* vb = reinterpret_cast<const CV*>(p.vals);
  AT* s = sm_s[gid];
  AT* xs = sm_x[gid];
  unsigned char* ring = sweep_smem + (size_t)gid * D * SB;
  const int n_tasks = p.task_row ? p.n_tasks : p.n;
  const bool stage_vec = p.stage_vec != 0;

  // Fill slot `slot` with row r, whose first entries are b0.. (block indices
  // bx) of the range [b0, b1): one commit group per row and lane.
  auto issue = [&](int r, int slot, int b0, int b1, const int64_t (&bx)[NPF]) {
    unsigned char* dst = ring + slot * SB;
#pragma unroll
    for (int u = 0; u < NPF; ++u)
      if (b0 + u < b1) {
#pragma unroll
        for (int q = 0; q < P; ++q) cp_async16(dst + u * BB + (q * G + gl) * 16, vb + bx[u] * CPB + q * G + gl);
      }
    if constexpr (kUseD) {
      const CV* db = reinterpret_cast<const CV*>(dinv_) + (int64_t)r * CPB;
#pragma unroll
      for (int q = 0; q < P; ++q) cp_async16(dst + C::OFF_D + (q * G + gl) * 16, db + q * G + gl);
    }
    if (stage_vec) {
      unsigned char* rd = dst + C::OFF_R + gl * C::LRB;
      if constexpr (!TRANS) {
#pragma unroll
        for (int q = 0; q < P; ++q)
          cp_async_small<sizeof(AT)>(rd + q * sizeof(AT), rhs_ + (int64_t)r * BS + q * RPP + gl / CPR);
      } else {
#pragma unroll
        for (int k = 0; k < C::LRB / 16; ++k)
          cp_async16(rd + 16 * k, reinterpret_cast<const unsigned char*>(rhs_ + (int64_t)r * BS + c0) + 16 * k);
      }
      if constexpr (POST == POST_SOR) {
        if (xold_) {
          unsigned char* od = dst + C::OFF_O + gl * P * sizeof(AT);
#pragma unroll
          for (int q = 0; q < P; ++q)
            cp_async_small<sizeof(AT)>(od + q * sizeof(AT), xold_ + (int64_t)r * BS + q * RPP + gl / CPR);
        }
      }
    }
    cp_async_commit();
  };
  // Entry classes: 0 skip, 1 the chain's previous row (shared memory),
  // 2 a row of this sweep (polled until it is no longer the sentinel),
  // 3 the previous iterate (SOR, final values).
  auto classify_j = [&](int j, int r, int pv) -> int {
    if (range_ == RANGE_SPLIT) {
      if (j == r) return 0;
      const bool dep = (dep_dir_ < 0) ? (j < r) : (j > r);
      if (!dep) return xold_ ? 3 : 0;
    }
    return j == pv ? 1 : 2;
  };
  auto classify = [&](int e, int r, int pv, int& j) -> int {
    j = __ldg(idx_ + e);
    return classify_j(j, r, pv);
  };
  // The chain's previous row, as this lane reads it (kind 1 entries).
  AT xp[XV];
  auto load_x = [&](int kind, int j, AT (&xv)[XV]) {
    const AT* src = kind == 3 ? xold_ : x_;
    if (kind == 1) {
#pragma unroll
      for (int v = 0; v < XV; ++v) xv[v] = xp[v];
    } else if constexpr (!TRANS) {
      ld_vec_cg<V>(src + (int64_t)j * BS + c0, xv);
    } else {
#pragma unroll
      for (int q = 0; q < P; ++q) xv[q] = __ldcg(src + (int64_t)j * BS + q * RPP + gl / CPR);
    }
  };
  auto poll_x = [&](int j, AT (&xv)[XV], int who) {
    bool pending = false;
#pragma unroll
    for (int v = 0; v < XV; ++v) pending |= is_sentinel(xv[v]);
    unsigned spins = 0;
    while (pending) {
      poll_pause(spins);
      if constexpr (!TRANS) {
#pragma unroll
        for (int v = 0; v < V; ++v) xv[v] = ld_poll(x_ + (int64_t)j * BS + c0 + v);
      } else {
#pragma unroll
        for (int q = 0; q < P; ++q) xv[q] = ld_poll(x_ + (int64_t)j * BS + q * RPP + gl / CPR);
      }
      pending = false;
#pragma unroll
      for (int v = 0; v < XV; ++v) pending |= is_sentinel(xv[v]);
      if (pending) {
        if (++spins > p.spin_limit) {
          set_status(st_, BSP_TIMEOUT, who);
          break;
        }
        if ((spins & 255u) == 0u && *reinterpret_cast<volatile int*>(&st_->code) != 0) break;  // already failed
      }
    }
  };

  unsigned cons = 0;  // rows consumed from this group's ring
  while (true) {
    int t = 0;
    if (gl == 0) t = (int)atomicAdd(p.ticket, 1u);
    t = __shfl_sync(gmask, t, gbase);
    if (t >= n_tasks) break;
    int i0, len;
    if (p.task_row) {
      i0 = __ldg(p.task_row + t);
      len = __ldg(p.task_len + t);
    } else {
      i0 = p.order ? __ldg(p.order + t) : t;
      len = 1;
    }
    // Row structure of the chain (entry range, first column and block
    // indices), one row per lane in windows of G rows, loaded a window ahead
    // and handed out by shuffles: no structure load sits on a row's path.
    struct Win {
      int b0, b1;
      int jx[NPF];
      int64_t bx[NPF];
    };
    auto load_window = [&](int w, Win& o) {
      const int k = w * G + gl;
      o.b0 = o.b1 = 0;
      if (k < len) row_range(p, i0 + k * task_dir_, o.b0, o.b1);
#pragma unroll
      for (int u = 0; u < NPF; ++u) {
        const bool in = o.b0 + u < o.b1;
        o.jx[u] = in ? __ldg(idx_ + o.b0 + u) : -1;
        o.bx[u] = in ? (blk_ ? __ldg(blk_ + o.b0 + u) : (int64_t)(o.b0 + u)) : 0;
      }
    };
    // Row k of window w: entry range, and (with_j) the first column indices.
    // Block indices are shuffled only for indirect structures; contiguous
    // ones use b0 + u.
    auto row_of = [&](const Win& w, int k, bool with_j, int& b0, int& b1, int (&jx)[NPF],
                      int64_t (&bx)[NPF]) {
      const int src = gbase + k % G;
      b0 = __shfl_sync(gmask, w.b0, src);
      b1 = __shfl_sync(gmask, w.b1, src);
#pragma unroll
      for (int u = 0; u < NPF; ++u) {
        if (with_j) jx[u] = __shfl_sync(gmask, w.jx[u], src);
        bx[u] = blk_ ? __shfl_sync(gmask, w.bx[u], src) : (int64_t)(b0 + u);
      }
    };
    Win cur, nxt;
    load_window(0, cur);
    if (len > G) load_window(1, nxt);
    // Matrix blocks, inverted diagonals, right-hand sides and old iterates do
    // not depend on the sweep: the ring holds the chain's next D rows.
    // (every lane commits exactly one copy group per ring position, empty
    // past the chain's end, so row s is complete once D - 1 groups remain)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      if (k < len) {  // uniform over the group (the shuffles need every lane)
        int b0, b1, jx[NPF];
        int64_t bx[NPF];
        row_of(cur, k, false, b0, b1, jx, bx);
        issue(i0 + k * task_dir_, (int)((cons + k) % D), b0, b1, bx);
      } else {
        cp_async_commit();
      }
    }
   for (int step = 0; step < len; ++step) {
    if (step > 0 && step % G == 0) {  // next structure window
      cur = nxt;
      if ((step / G + 1) * G < len) load_window(step / G + 1, nxt);
    }
    const int i = i0 + step * task_dir_;
    const int prev = step > 0 ? i - task_dir_ : -1;
    int beg, end, jr[NPF];
    int64_t br[NPF];
    row_of(cur, step, true, beg, end, jr, br);
    const int slot = (int)(cons % D);
    cp_async_wait<D - 1>();
    ++cons;
    const unsigned char* sl = ring + slot * SB;
    const CV* sblk = reinterpret_cast<const CV*>(sl);
    CV pf[NPF][P], pd[P];
    AT rh[XR], xo[P];
#pragma unroll
    for (int u = 0; u < NPF; ++u)
      if (beg + u < end) {
#pragma unroll
        for (int q = 0; q < P; ++q) pf[u][q] = sblk[u * CPB + q * G + gl];
      }
    if constexpr (kUseD) {
      const CV* sd = reinterpret_cast<const CV*>(sl + C::OFF_D);
#pragma unroll
      for (int q = 0; q < P; ++q) pd[q] = sd[q * G + gl];
    }
    if (stage_vec) {
      const AT* rl = reinterpret_cast<const AT*>(sl + C::OFF_R) + gl * C::XR;
#pragma unroll
      for (int v = 0; v < XR; ++v) rh[v] = rl[v];
    } else if constexpr (!TRANS) {
#pragma unroll
      for (int q = 0; q < P; ++q) rh[q] = __ldcg(rhs_ + (int64_t)i * BS + q * RPP + gl / CPR);
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) rh[v] = __ldcg(rhs_ + (int64_t)i * BS + c0 + v);
    }
    if constexpr (POST == POST_SOR) {
      const AT* ol = reinterpret_cast<const AT*>(sl + C::OFF_O) + gl * P;
#pragma unroll
      for (int q = 0; q < P; ++q)
        xo[q] = !xold_ ? AT(0) : stage_vec ? ol[q] : __ldcg(xold_ + (int64_t)i * BS + q * RPP + gl / CPR);
    }
    AT acc[P];
    AT tac[V];
#pragma unroll
    for (int q = 0; q < P; ++q) acc[q] = AT(0);
#pragma unroll
    for (int v = 0; v < V; ++v) tac[v] = AT(0);
    auto fma_entry = [&](const CV (&a)[P], const AT (&xv)[XV]) {
      if constexpr (!TRANS) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          AT av[V];
          unpack(a[q], av);
#pragma unroll
          for (int v = 0; v < V; ++v) acc[q] = fma(av[v], xv[v], acc[q]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          AT av[V];
          unpack(a[q], av);
#pragma unroll
          for (int v = 0; v < V; ++v) tac[v] = fma(av[v], xv[q], tac[v]);
        }
      }
    };
    // first NPF entries: issue every dependency load, then poll the ones
    // that are not final yet, so their round trips overlap
    {
      AT xv[NPF][XV];
      int kind[NPF], jj[NPF];
#pragma unroll
      for (int u = 0; u < NPF; ++u) {
        jj[u] = jr[u];
        kind[u] = (beg + u < end) ? classify_j(jj[u], i, prev) : 0;
        if (kind[u]) load_x(kind[u], jj[u], xv[u]);
      }
#pragma unroll
      for (int u = 0; u < NPF; ++u) {
        if (kind[u] == 2) poll_x(jj[u], xv[u], i);
        if (kind[u]) fma_entry(pf[u], xv[u]);
      }
    }
    for (int e = beg + NPF; e < end; ++e) {
      int j;
      const int kind = classify(e, i, prev, j);
      if (!kind) continue;
      const int64_t b = blk_ ? __ldg(blk_ + e) : (int64_t)e;
      CV a[P];
#pragma unroll
      for (int q = 0; q < P; ++q) a[q] = ld_stream(vb + b * CPB + q * G + gl);
      AT xe[XV];
      load_x(kind, j, xe);
      if (kind == 2) poll_x(j, xe, i);
      fma_entry(a, xe);
    }
    // s = rhs_i - sum  (in shared memory, BS values per group)
    if constexpr (!TRANS) {
#pragma unroll
      for (int q = 0; q < P; ++q) acc[q] = row_reduce<CPR>(acc[q], gmask);
      if (gl % CPR == 0) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const int r = q * RPP + gl / CPR;
          s[r] = rh[q] - acc[q];
        }
      }
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int o = CPR; o < G; o <<= 1) tac[v] += __shfl_xor_sync(gmask, tac[v], o);
      if (gl < CPR) {
#pragma unroll
        for (int v = 0; v < V; ++v) s[c0 + v] = rh[v] - tac[v];
      }
    }
    __syncwarp(gmask);
    // post-operation and write-back of row i
    if constexpr (POST == POST_NONE) {
      for (int r = gl; r < BS; r += G) {
        x_[(int64_t)i * BS + r] = s[r];
        xs[r] = s[r];
      }
    } else if constexpr (POST == POST_D || POST == POST_SOR) {
      AT sv[V];
#pragma unroll
      for (int v = 0; v < V; ++v) sv[v] = s[c0 + v];
      AT o[P];
#pragma unroll
      for (int q = 0; q < P; ++q) {
        AT av[V];
        unpack(pd[q], av);
        o[q] = AT(0);
#pragma unroll
        for (int v = 0; v < V; ++v) o[q] = fma(av[v], sv[v], o[q]);
        o[q] = row_reduce<CPR>(o[q], gmask);
      }
      if (gl % CPR == 0) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const int r = q * RPP + gl / CPR;
          AT val = o[q];
          if constexpr (POST == POST_SOR) {
            // x(im) += -w * x(im) + w * ph   (preconditioners.hpp:161-165)
            val = xo[q] + (-w_ * xo[q] + w_ * val);
          }
          x_[(int64_t)i * BS + r] = val;
          xs[r] = val;
        }
      }
    } else {  // POST_DT: x = D^T s
      AT o[V];
#pragma unroll
      for (int v = 0; v < V; ++v) o[v] = AT(0);
#pragma unroll
      for (int q = 0; q < P; ++q) {
        const int r = q * RPP + gl / CPR;
        const AT sr = s[r];
        AT av[V];
        unpack(pd[q], av);
#pragma unroll
        for (int v = 0; v < V; ++v) o[v] = fma(av[v], sr, o[v]);
      }
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int off = CPR; off < G; off <<= 1) o[v] += __shfl_xor_sync(gmask, o[v], off);
      if (gl < CPR) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          x_[(int64_t)i * BS + c0 + v] = o[v];
          xs[c0 + v] = o[v];
        }
      }
    }
    // Row i is published by its values themselves: readers poll the 8-byte
    // words until they are no longer the sentinel, so no flag or fence is
    // needed.  The barrier keeps shared memory consistent for the next row,
    // which takes row i from registers (read here, before the refill copies
    // are issued).
    __syncwarp(gmask);
    if constexpr (!TRANS) {
#pragma unroll
      for (int v = 0; v < V; ++v) xp[v] = xs[c0 + v];
    } else {
#pragma unroll
      for (int q = 0; q < P; ++q) xp[q] = xs[q * RPP + gl / CPR];
    }
    // Every value taken from the slot has been consumed: refill it with row
    // step + D of the chain.
    {
      const int s2 = step + D;
      if (s2 < len) {  // uniform over the group
        int b0, b1, jx[NPF];
        int64_t bx[NPF];
        row_of((s2 / G == step / G) ? cur : nxt, s2, false, b0, b1, jx, bx);
        issue(i + D * task_dir_, slot, b0, b1, bx);
      } else {
        cp_async_commit();
      }
    }
   }
  }
}

// Any block size (bs <= 32): one warp per row, lane r computes component r.
template <typename VT, typename AT, bool TRANS, int POST>
__global__ void __launch_bounds__(kSweepThreads) k_sweep_generic(const SweepP<VT, AT> p, int bs) {
  __shared__ AT sm_s[kSweepThreads / 32][32];
  const int lane = threadIdx.x & 31;
  AT* s = sm_s[threadIdx.x >> 5];
  const int b2 = bs * bs;
  while (true) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(p.ticket, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= p.n) break;
    const int i = p.order ? __ldg(p.order + t) : t;
    int beg, end;
    row_range(p, i, beg, end);
    AT acc = AT(0);
    for (int e = beg; e < end; ++e) {
      const int j = __ldg(p.idx + e);
      const AT* src;
      bool poll = true;
      if (p.range == RANGE_SPLIT) {
        if (j == i) continue;
        const bool dep = (p.dep_dir < 0) ? (j < i) : (j > i);
        if (dep) {
          src = p.x;
        } else {
          if (!p.xold) continue;
          src = p.xold;
          poll = false;
        }
      } else {
        src = p.x;
      }
      const int64_t b = p.blk ? __ldg(p.blk + e) : (int64_t)e;
      if (lane < bs) {
        const VT* a = p.vals + b * b2;
        for (int c = 0; c < bs; ++c) {
          const AT m = TRANS ? AT(a[c * bs + lane]) : AT(a[lane * bs + c]);
          AT xc = __ldcg(src + (int64_t)j * bs + c);
          if (poll) {
            unsigned spins = 0;
            while (is_sentinel(xc)) {  // row j of this sweep not final yet
              poll_pause(spins);
              xc = ld_poll(src + (int64_t)j * bs + c);
              if (++spins > p.spin_limit) {
                set_status(p.st, BSP_TIMEOUT, i);
                break;
              }
              if ((spins & 255u) == 0u && *reinterpret_cast<volatile int*>(&p.st->code) != 0) break;
            }
          }
          acc = fma(m, xc, acc);
        }
      }
    }
    if (lane < bs) s[lane] = __ldcg(p.rhs + (int64_t)i * bs + lane) - acc;
    __syncwarp();
    if (lane < bs) {
      AT val = s[lane];
      if constexpr (POST != POST_NONE) {
        const VT* d = p.dinv + (int64_t)i * b2;
        val = AT(0);
        for (int c = 0; c < bs; ++c) {
          const AT m = (POST == POST_DT) ? AT(d[c * bs + lane]) : AT(d[lane * bs + c]);
          val = fma(m, s[c], val);
        }
      }
      if constexpr (POST == POST_SOR) {
        const AT xo = p.xold ? __ldcg(p.xold + (int64_t)i * bs + lane) : AT(0);
        val = xo + (-p.w * xo + p.w * val);
      }
      p.x[(int64_t)i * bs + lane] = val;
    }
    __syncwarp();
  }
}

// ----------------------------------------------------------------- factorisation
enum { FACT_ILU0 = 0, FACT_ICHOL0 = 1, FACT_DIAG = 2 };

struct FactorP {
  int n, bs, mode;
  const int* order;
  const int* ptr;
  const int* col;
  const int* diag;
  double* vals;
  double* dinv;
  int* flags;
  int epoch;
  unsigned* ticket;
  DevStatus* st;
  unsigned spin_limit;
};

constexpr int kFactorWarps = 4;
constexpr size_t kFactorRowsSmem = 96 * 1024;  // staging of the row-resident kernel per CTA

__global__ void __launch_bounds__(kFactorWarps * 32) k_factor(const FactorP p) {
  extern __shared__ double smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bs = p.bs, b2 = bs * bs;
  double* sA = smem + (size_t)warp * 5 * b2;
  double* sB = sA + b2;
  double* sC = sB + b2;
  double* aug = sC + b2;  // 2*b2
  while (true) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(p.ticket, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= p.n) break;
    const int k = p.order ? __ldg(p.order + t) : t;
    const int beg = __ldg(p.ptr + k), dg = __ldg(p.diag + k), end = __ldg(p.ptr + k + 1);
    if (p.mode != FACT_DIAG) {
      for (int e = beg; e < dg; ++e) wait_flag(p.flags + __ldg(p.col + e), p.epoch, p.st, k, p.spin_limit);
      for (int e = beg; e < dg; ++e) {
        const int i = __ldg(p.col + e);
        warp_copy_in(sA, p.vals + (int64_t)e * b2, b2);
        warp_copy_in(sB, p.dinv + (int64_t)i * b2, b2);
        // ILU0: L_ki = A_ki U_ii^{-1};  IChol0: L_ki = A_ki L_ii^{-T}
        warp_gemm(sC, sA, sB, bs, p.mode == FACT_ICHOL0);
        warp_copy_out(p.vals + (int64_t)e * b2, sC, b2);
        if (p.mode == FACT_ILU0) {
          // A_kj -= L_ki U_ij for every j > i present in both rows
          const int ui0 = __ldg(p.diag + i) + 1, ui1 = __ldg(p.ptr + i + 1);
          for (int e2 = e + 1; e2 < end; ++e2) {
            const int pos = warp_find(p.col, ui0, ui1, __ldg(p.col + e2));
            if (pos >= 0) {
              warp_copy_in(sB, p.vals + (int64_t)pos * b2, b2);
              warp_gemm_sub_global(p.vals + (int64_t)e2 * b2, sC, sB, bs, false);
            }
          }
        } else {
          // A_kj -= L_ki L_ji^T for i < j <= k with (j, i) in the pattern
          for (int e2 = e + 1; e2 <= dg; ++e2) {
            const int j = __ldg(p.col + e2);
            if (j == k) {
              warp_gemm_sub_global(p.vals + (int64_t)e2 * b2, sC, sC, bs, true);
            } else {
              const int pos = warp_find(p.col, __ldg(p.ptr + j), __ldg(p.diag + j), i);
              if (pos >= 0) {
                warp_copy_in(sB, p.vals + (int64_t)pos * b2, b2);
                warp_gemm_sub_global(p.vals + (int64_t)e2 * b2, sC, sB, bs, true);
              }
            }
          }
        }
      }
    }
    warp_copy_in(sA, p.vals + (int64_t)dg * b2, b2);
    if (p.mode == FACT_ICHOL0) {
      const bool ok = warp_cholesky(sA, bs);
      if (!ok && lane == 0) set_status(p.st, BSP_NOT_SPD, k);
      warp_copy_out(p.vals + (int64_t)dg * b2, sA, b2);
      warp_lower_inverse(sB, sA, bs);
      warp_copy_out(p.dinv + (int64_t)k * b2, sB, b2);
    } else {
      const bool ok = warp_inverse(sB, sA, aug, bs);
      if (!ok && lane == 0) set_status(p.st, BSP_ZERO_PIVOT, k);
      warp_copy_out(p.dinv + (int64_t)k * b2, sB, b2);
    }
    __threadfence();
    __syncwarp();
    if (lane == 0 && p.flags) st_release(p.flags + k, p.epoch);
    __syncwarp();
  }
}

// Row-resident factorisation (ILU0 / IChol0, bs <= 16): one warp per block
// row k, rows claimed in level order.  The row's blocks are copied to shared
// memory before the warp waits for the rows it depends on, every dependency
// block (inverse diagonals U_ii^-1 / L_ii^-1 and the update sources of the
// elimination plan) is then fetched in one batch, and the whole elimination
// runs in shared memory: per lower entry (increasing i) L_ki = A_ki U_ii^-1
// (ILU0) or A_ki L_ii^-T (IChol0), then the planned updates of the later
// blocks; finally the diagonal block is inverted (ILU0) or factored and its
// triangular inverse formed (IChol0), and the row is written back.  The same
// operations in the same order as k_factor (bit-identical factors); only the
// memory traffic on the dependency path changes.
template <int BS = 0>
__device__ inline void warp_gemm_sub_smem(double* T, const double* A, const double* B, int bs_rt, bool trB) {
  const int bs = BS > 0 ? BS : bs_rt;
  const int lane = threadIdx.x & 31;
  for (int e = lane; e < bs * bs; e += 32) {
    const int r = e / bs, c = e % bs;
    double acc = 0.0;
    if (trB) {
#pragma unroll
      for (int t = 0; t < (BS > 0 ? BS : bs); ++t) acc = fma(A[r * bs + t], B[c * bs + t], acc);
    } else {
#pragma unroll
      for (int t = 0; t < (BS > 0 ? BS : bs); ++t) acc = fma(A[r * bs + t], B[t * bs + c], acc);
    }
    T[e] = T[e] - acc;
  }
  __syncwarp();
}

struct FactorRowsP {
  int n, bs, mode;
  const int* order;
  const int* ptr;
  const int* col;
  const int* diag;
  const int* pp;
  const int2* pairs;
  double* vals;
  double* dinv;
  int* flags;
  int epoch;
  unsigned* ticket;
  DevStatus* st;
  unsigned spin_limit;
  int nbmax, depmax;  // row blocks and dependency blocks staged per warp
};

// Per warp, after the blocks: the row's elimination plan staged from global
// memory before the dependency waits (at most kFrEnts lower entries and
// kFrPairs update pairs; longer rows read the plan from global memory).
constexpr int kFrEnts = 31, kFrPairs = 96;
constexpr size_t kFrPlanBytes = kFrPairs * sizeof(int2) + 2 * (kFrEnts + 1) * sizeof(int);

template <int BS>
__global__ void __launch_bounds__(256, 1) k_factor_rows(const FactorRowsP p) {
  extern __shared__ double fr_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bs = BS > 0 ? BS : p.bs, b2 = bs * bs;
  const size_t warp_bytes = (size_t)(p.nbmax + p.depmax + 3) * b2 * sizeof(double) + kFrPlanBytes;
  unsigned char* wbase = reinterpret_cast<unsigned char*>(fr_smem) + (size_t)warp * warp_bytes;
  double* rowb = reinterpret_cast<double*>(wbase);
  double* dep = rowb + (size_t)p.nbmax * b2;
  double* Lb = dep + (size_t)p.depmax * b2;
  double* aug = Lb + b2;
  int2* prw = reinterpret_cast<int2*>(aug + 2 * b2);
  int* ppw = reinterpret_cast<int*>(prw + kFrPairs);
  int* colw = ppw + kFrEnts + 1;
  const bool chol = p.mode == FACT_ICHOL0;
  while (true) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(p.ticket, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= p.n) break;
    const int k = __ldg(p.order + t);
    const int beg = __ldg(p.ptr + k), dg = __ldg(p.diag + k), end = __ldg(p.ptr + k + 1);
    // the row's own blocks, in flight while the warp waits for its dependencies
    for (int x = lane; x < (end - beg) * b2; x += 32)
      cp_async_small<8>(rowb + x, p.vals + (int64_t)beg * b2 + x);
    cp_async_commit();
    // and its elimination plan (entry offsets, columns, update pairs)
    const int nl = dg - beg;
    bool staged = nl <= kFrEnts;
    if (staged) {
      if (lane <= nl) ppw[lane] = __ldg(p.pp + beg + lane);
      if (lane < nl) colw[lane] = __ldg(p.col + beg + lane);
    }
    __syncwarp();
    const int q0 = staged ? ppw[0] : 0;
    staged = staged && ppw[nl] - q0 <= kFrPairs;
    if (staged)
      for (int y = lane; y < ppw[nl] - q0; y += 32) prw[y] = p.pairs[q0 + y];
    __syncwarp();
    auto PP = [&](int x) { return staged ? ppw[x - beg] : __ldg(p.pp + x); };
    auto PR = [&](int q) { return staged ? prw[q - q0] : p.pairs[q]; };
    auto COL = [&](int x) { return staged ? colw[x - beg] : __ldg(p.col + x); };
    for (int e = beg; e < dg; ++e) wait_flag(p.flags + COL(e), p.epoch, p.st, k, p.spin_limit);
    int e = beg;
    while (e < dg) {
      // a batch of consecutive lower entries whose dependency blocks fit
      int used = 0, eb = e;
      while (eb < dg) {
        int need = 1;
        for (int q = PP(eb); q < PP(eb + 1); ++q) need += PR(q).y >= 0;
        if (eb > e && used + need > p.depmax) break;
        used += need;
        ++eb;
      }
      int slot = 0;
      for (int x = e; x < eb; ++x) {
        const double* src = p.dinv + (int64_t)COL(x) * b2;
        for (int y = lane; y < b2; y += 32) cp_async_small<8>(dep + (size_t)slot * b2 + y, src + y);
        ++slot;
        for (int q = PP(x); q < PP(x + 1); ++q) {
          const int s = PR(q).y;
          if (s < 0) continue;
          for (int y = lane; y < b2; y += 32) cp_async_small<8>(dep + (size_t)slot * b2 + y, p.vals + (int64_t)s * b2 + y);
          ++slot;
        }
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncwarp();
      slot = 0;
      for (int x = e; x < eb; ++x) {
        double* Ak = rowb + (size_t)(x - beg) * b2;
        // ILU0: L_ki = A_ki U_ii^{-1};  IChol0: L_ki = A_ki L_ii^{-T}
        warp_gemm<BS>(Lb, Ak, dep + (size_t)slot * b2, bs, chol);
        ++slot;
        for (int y = lane; y < b2; y += 32) Ak[y] = Lb[y];
        __syncwarp();
        for (int q = PP(x); q < PP(x + 1); ++q) {
          const int2 pr = PR(q);
          const double* S;
          if (pr.y >= 0) {
            S = dep + (size_t)slot * b2;
            ++slot;
          } else {
            S = rowb + (size_t)(-1 - pr.y - beg) * b2;
          }
          warp_gemm_sub_smem<BS>(rowb + (size_t)(pr.x - beg) * b2, Lb, S, bs, chol);
        }
      }
      e = eb;
    }
    cp_async_wait<0>();
    __syncwarp();
    double* Dk = rowb + (size_t)(dg - beg) * b2;
    if (chol) {
      const bool ok = warp_cholesky<BS>(Dk, bs);
      if (!ok && lane == 0) set_status(p.st, BSP_NOT_SPD, k);
      warp_lower_inverse<BS>(Lb, Dk, bs);
    } else {
      const bool ok = warp_inverse<BS>(Lb, Dk, aug, bs);  // aug: bs x 2bs scratch
      if (!ok && lane == 0) set_status(p.st, BSP_ZERO_PIVOT, k);
    }
    for (int x = lane; x < (end - beg) * b2; x += 32) p.vals[(int64_t)beg * b2 + x] = rowb[x];
    for (int y = lane; y < b2; y += 32) p.dinv[(int64_t)k * b2 + y] = Lb[y];
    __threadfence();
    __syncwarp();
    if (lane == 0) st_release(p.flags + k, p.epoch);
    __syncwarp();
  }
}

// Gather blocks: dst[e] = src[perm[e]] (bs*bs values each).
__global__ void k_gather_blocks(int64_t nblk, int b2, const int64_t* __restrict__ perm,
                                const double* __restrict__ src, double* __restrict__ dst) {
  const int64_t total = nblk * b2;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = t / b2;
    dst[t] = src[perm[e] * b2 + (t % b2)];
  }
}
__global__ void k_scatter_blocks(int64_t nblk, int b2, const int64_t* __restrict__ perm,
                                 const double* __restrict__ src, double* __restrict__ dst) {
  const int64_t total = nblk * b2;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = t / b2;
    dst[perm[e] * b2 + (t % b2)] = src[t];
  }
}
template <typename T>
__global__ void k_convert(int64_t n, const double* __restrict__ a, T* __restrict__ b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if constexpr (std::is_same<T, float>::value) b[i] = (float)a[i];
    else b[i] = __float2bfloat16_rn((float)a[i]);
  }
}

int grid_for(const bsp_handle_s* h, int64_t n, int threads);

}  // namespace bsp

// ================================================================= host side
using namespace bsp;



namespace bsp {

// Level of each row when row i depends on the rows listed in deps(i).
template <class Deps>
static int level_order(int n, bool ascending, Deps deps, std::vector<int>& order) {
  std::vector<int> lvl(n, 0);
  int maxl = -1;
  if (ascending) {
    for (int i = 0; i < n; ++i) {
      int l = 0;
      deps(i, [&](int j) { l = std::max(l, lvl[j] + 1); });
      lvl[i] = l;
      maxl = std::max(maxl, l);
    }
  } else {
    for (int i = n - 1; i >= 0; --i) {
      int l = 0;
      deps(i, [&](int j) { l = std::max(l, lvl[j] + 1); });
      lvl[i] = l;
      maxl = std::max(maxl, l);
    }
  }
  // counting sort by level; inside a level rows keep natural sweep order
  std::vector<int> cnt(maxl + 2, 0);
  for (int i = 0; i < n; ++i) cnt[lvl[i] + 1]++;
  for (int l = 0; l <= maxl; ++l) cnt[l + 1] += cnt[l];
  order.assign(n, 0);
  if (ascending)
    for (int i = 0; i < n; ++i) order[cnt[lvl[i]]++] = i;
  else
    for (int i = n - 1; i >= 0; --i) order[cnt[lvl[i]]++] = i;
  return maxl + 1;
}

// Sweep tasks: maximal chains of rows visited consecutively in sweep order
// (ascending: r, r+1, ...; descending: r, r-1, ...) in which every row depends
// on the row visited just before it.  Chains are contiguous row ranges, so the
// chain graph is acyclic; tasks are sorted by chain level (1 + the highest
// level of any other chain a row of the chain depends on), so a task only
// waits on rows of tasks with smaller tickets.
template <class Deps>
static int build_tasks(int n, bool ascending, Deps deps, std::vector<int>& row, std::vector<int>& len) {
  std::vector<int> chain(n), first, clen;
  const int dir = ascending ? 1 : -1;
  for (int idx = 0; idx < n; ++idx) {
    const int r = ascending ? idx : n - 1 - idx;
    const int prev = r - dir;
    bool cont = false;
    if (idx > 0) deps(r, [&](int j) { cont |= (j == prev); });
    if (cont) {
      chain[r] = chain[prev];
      clen[chain[r]]++;
    } else {
      chain[r] = (int)first.size();
      first.push_back(r);
      clen.push_back(1);
    }
  }
  const int nc = (int)first.size();
  std::vector<int> lvl(nc, 0);
  for (int c = 0; c < nc; ++c)  // chains are created in sweep order: a topological order
    for (int s = 0; s < clen[c]; ++s) {
      const int r = first[c] + s * dir;
      deps(r, [&](int j) {
        if (chain[j] != c) lvl[c] = std::max(lvl[c], lvl[chain[j]] + 1);
      });
    }
  std::vector<int> idx(nc);
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return lvl[a] < lvl[b]; });
  row.resize(nc);
  len.resize(nc);
  for (int t = 0; t < nc; ++t) {
    row[t] = first[idx[t]];
    len[t] = clen[idx[t]];
  }
  return nc;
}

template <typename T> static int upload(DevBuf<T>& d, const std::vector<T>& v) {
  BSP_TRY(d.alloc(v.empty() ? 1 : v.size()));
  if (!v.empty())
    BSP_CUDA_TRY(cudaMemcpy(d.get(), v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
  return BSP_OK;
}

template <typename T>
static int copy_dev(DevBuf<T>& dst, const DevBuf<T>& src, cudaStream_t s, bsp_matrix_s* recycle = nullptr) {
  if (recycle) BSP_TRY(take(recycle, dst, src.n ? src.n : 1));
  else BSP_TRY(dst.alloc(src.n ? src.n : 1));
  if (src.n) BSP_CUDA_TRY(cudaMemcpyAsync(dst.get(), src.get(), src.n * sizeof(T), cudaMemcpyDeviceToDevice, s));
  return BSP_OK;
}

// Preconditioner <-> the matrix's cached symbolic analysis (device-to-device copies).
static int sym_transfer(bsp_precond_s* pc, SymbolicCache& C, bool save) {
  cudaStream_t s = pc->h->stream;
#define BSP_SYM_FIELD(f) BSP_TRY(save ? copy_dev(C.f, pc->f, s) : copy_dev(pc->f, C.f, s, pc->A));
  BSP_SYM_FIELD(f_ptr) BSP_SYM_FIELD(f_col) BSP_SYM_FIELD(f_diag) BSP_SYM_FIELD(d_perm)
  BSP_SYM_FIELD(order_lo) BSP_SYM_FIELD(order_up) BSP_SYM_FIELD(task_lo_row) BSP_SYM_FIELD(task_lo_len)
  BSP_SYM_FIELD(task_up_row) BSP_SYM_FIELD(task_up_len) BSP_SYM_FIELD(t_ptr) BSP_SYM_FIELD(t_row)
  BSP_SYM_FIELD(t_blk) BSP_SYM_FIELD(a_diag)
#undef BSP_SYM_FIELD
  if (save) {
    C.wv_lo = pc->wv_lo;
    C.wv_up = pc->wv_up;
    C.ss_lo = pc->ss_lo;
    C.ss_up = pc->ss_up;
    C.plan = pc->plan;
    C.h_perm = pc->h_perm;
    C.f_nnzb = pc->f_nnzb;
    C.n_lev_lo = pc->n_lev_lo;
    C.n_lev_up = pc->n_lev_up;
    C.n_task_lo = pc->n_task_lo;
    C.n_task_up = pc->n_task_up;
    C.valid = true;
    C.laid_out = pc->applied;
  } else {
    pc->wv_lo = C.wv_lo;
    pc->wv_up = C.wv_up;
    pc->ss_lo = C.ss_lo;
    pc->ss_up = C.ss_up;
    pc->plan = C.plan;
    pc->h_perm = C.h_perm;
    pc->f_nnzb = C.f_nnzb;
    pc->n_lev_lo = C.n_lev_lo;
    pc->n_lev_up = C.n_lev_up;
    pc->n_task_lo = C.n_task_lo;
    pc->n_task_up = C.n_task_up;
  }
  return BSP_OK;
}

template <class Deps>
static int make_tasks(bsp_precond_s* pc, bool lower, int n, Deps deps) {
  std::vector<int> row, len;
  const int nt = build_tasks(n, lower, deps, row, len);
  if (lower) {
    pc->n_task_lo = nt;
    BSP_TRY(upload(pc->task_lo_row, row));
    BSP_TRY(upload(pc->task_lo_len, len));
  } else {
    pc->n_task_up = nt;
    BSP_TRY(upload(pc->task_up_row, row));
    BSP_TRY(upload(pc->task_up_len, len));
  }
  return BSP_OK;
}

static int read_status(bsp_handle_s* h, DevStatus* out) {
  BSP_CUDA_TRY(cudaMemcpyAsync(out, h->ws.status.get(), sizeof(DevStatus), cudaMemcpyDeviceToHost,
                               h->stream));
  BSP_CUDA_TRY(cudaStreamSynchronize(h->stream));
  if (out->code != 0) {
    BSP_CUDA_TRY(cudaMemsetAsync(h->ws.status.get(), 0, sizeof(DevStatus), h->stream));
    BSP_CUDA_TRY(cudaStreamSynchronize(h->stream));
  }
  return BSP_OK;
}

// Persistent grid for a kernel: SMs x resident CTAs.
template <class K> static int persistent_grid(const bsp_handle_s* h, K kernel, int threads, size_t smem) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess ||
      per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  return h->num_sms * per_sm;
}

static int run_factor(bsp_precond_s* pc, int mode, const int* order, const int* ptr, const int* col,
                      const int* diag, double* vals, int n) {
  bsp_handle_s* h = pc->h;
  FactorP fp;
  fp.n = n;
  fp.bs = pc->bs;
  fp.mode = mode;
  fp.order = order;
  fp.ptr = ptr;
  fp.col = col;
  fp.diag = diag;
  fp.vals = vals;
  fp.dinv = pc->dinv.get();
  fp.flags = pc->flags.get();
  fp.epoch = ++h->epoch;
  fp.ticket = pc->ticket.get();
  fp.st = h->ws.status.get();
  fp.spin_limit = h->spin_limit;
  BSP_CUDA_TRY(cudaMemsetAsync(pc->ticket.get(), 0, sizeof(unsigned), h->stream));
  // the row-resident kernel when the plan exists and a row fits its staging
  const FactorPlan* plan = pc->plan.get();
  const size_t b2 = (size_t)pc->bs * pc->bs;
  const int depmax = plan ? std::max(plan->max_deps, 4) : 0;
  const size_t per_warp = plan ? (size_t)(plan->max_row + depmax + 3) * b2 * sizeof(double) + kFrPlanBytes : 0;
  if (mode != FACT_DIAG && plan && pc->bs <= 16 && per_warp <= kFactorRowsSmem && ptr == pc->f_ptr.get()) {
    FactorRowsP rp;
    rp.n = n;
    rp.bs = pc->bs;
    rp.mode = mode;
    rp.order = order;
    rp.ptr = ptr;
    rp.col = col;
    rp.diag = diag;
    rp.pp = plan->pp.get();
    rp.pairs = plan->pairs.get();
    rp.vals = vals;
    rp.dinv = fp.dinv;
    rp.flags = fp.flags;
    rp.epoch = fp.epoch;
    rp.ticket = fp.ticket;
    rp.st = fp.st;
    rp.spin_limit = fp.spin_limit;
    rp.nbmax = plan->max_row;
    rp.depmax = depmax;
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, kFactorRowsSmem / per_warp));
    const size_t smem = per_warp * warps;
    auto launch = [&](auto kern) -> int {
      BSP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      const int grid = persistent_grid(h, kern, warps * 32, smem);
      bsp::count_launch(), kern<<<grid, warps * 32, smem, h->stream>>>(rp);
      return BSP_OK;
    };
    if (pc->bs == 8) BSP_TRY(launch(k_factor_rows<8>));
    else if (pc->bs == 16) BSP_TRY(launch(k_factor_rows<16>));
    else if (pc->bs == 4) BSP_TRY(launch(k_factor_rows<4>));
    else BSP_TRY(launch(k_factor_rows<0>));
  } else {
    const size_t smem = (size_t)kFactorWarps * 5 * pc->bs * pc->bs * sizeof(double);
    BSP_CUDA_TRY(cudaFuncSetAttribute(k_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int grid = persistent_grid(h, k_factor, kFactorWarps * 32, smem);
    bsp::count_launch(), k_factor<<<grid, kFactorWarps * 32, smem, h->stream>>>(fp);
  }
  BSP_CUDA_TRY(cudaPeekAtLastError());
  DevStatus st;
  BSP_TRY(read_status(h, &st));
  if (st.code != 0) {
    record_error(std::string("preconditioner set-up: ") + bsp_status_string(st.code) +
                 " at block row " + std::to_string(st.where));
    return st.code;
  }
  return BSP_OK;
}

// ---------------------------------------------------------------- sweep launch
template <int BS, typename VT, typename AT, bool TRANS, int POST>
static int launch_sweep_t(bsp_handle_s* h, const SweepP<VT, AT>& p) {
  constexpr size_t smem = SweepCfg<BS, VT, AT, TRANS, POST>::kSmem;
  static PerDevice ready;
  static std::atomic<int> per_sm{1};  // resident CTAs an SM (every device is the same part)
  if (!ready.has(h->device)) {
    BSP_CUDA_TRY(cudaFuncSetAttribute(k_sweep<BS, VT, AT, TRANS, POST>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    per_sm = persistent_grid(h, k_sweep<BS, VT, AT, TRANS, POST>, kSweepThreads, smem) / h->num_sms;
    ready.set(h->device);
  }
  bsp::count_launch(),
      k_sweep<BS, VT, AT, TRANS, POST><<<h->num_sms * per_sm, kSweepThreads, smem, h->stream>>>(p);
  return BSP_OK;
}

template <typename VT, typename AT, bool TRANS, int POST>
static int launch_sweep(bsp_handle_s* h, int bs, SweepP<VT, AT> p, unsigned* ticket) {
  p.epoch = ++h->epoch;
  p.ticket = ticket;
  p.st = h->ws.status.get();
  p.spin_limit = h->spin_limit;
  // 16-byte staging copies need aligned vectors (the matrix blocks always are)
  p.stage_vec = (reinterpret_cast<uintptr_t>(p.rhs) % 16 == 0) &&
                (p.xold == nullptr || reinterpret_cast<uintptr_t>(p.xold) % 16 == 0);
  BSP_CUDA_TRY(cudaMemsetAsync(ticket, 0, sizeof(unsigned), h->stream));
  constexpr int V = Chunk<VT>::V;
  bool done = false;
  // blocks of more than 4 chunk passes per lane (bs 32 in FP64) would not fit
  // the per-lane registers of the staged kernel: they use the generic kernel
#define BSP_SWEEP_CASE(B)                                          \
  case B:                                                          \
    if constexpr (B % V == 0 && B * B / V <= 128) {               \
      BSP_TRY((launch_sweep_t<B, VT, AT, TRANS, POST>(h, p)));     \
      done = true;                                                 \
    }                                                              \
    break;
  switch (bs) {
    BSP_SWEEP_CASE(2)
    BSP_SWEEP_CASE(4)
    BSP_SWEEP_CASE(8)
    BSP_SWEEP_CASE(16)
    BSP_SWEEP_CASE(32)
    default: break;
  }
#undef BSP_SWEEP_CASE
  if (!done) {
    static std::atomic<int> per_sm{0};
    if (!per_sm) per_sm = persistent_grid(h, k_sweep_generic<VT, AT, TRANS, POST>, kSweepThreads, 0) / h->num_sms;
    const int grid = h->num_sms * per_sm;
    p.task_row = nullptr;  // the generic kernel takes one row per ticket
    bsp::count_launch(), k_sweep_generic<VT, AT, TRANS, POST><<<grid, kSweepThreads, 0, h->stream>>>(p, bs);
  }
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

// ---------------------------------------------------------------- build
// Elimination plan (FactorPlan) of the row-sorted factor structure.
static int build_factor_plan(bsp_precond_s* pc, int n, const std::vector<int>& ptr, const std::vector<int>& col,
                             const std::vector<int>& diag, bool lower_only) {
  auto plan = std::make_shared<FactorPlan>();
  const int64_t nf = (int64_t)col.size();
  std::vector<int> pp(nf + 1, 0);
  std::vector<int2> pairs;
  pairs.reserve(nf);
  // position of column c in the sorted range [a, b) of the factor structure
  auto find = [&](int a, int b, int c) -> int {
    const auto it = std::lower_bound(col.begin() + a, col.begin() + b, c);
    return (it != col.begin() + b && *it == c) ? (int)(it - col.begin()) : -1;
  };
  int max_row = 0, max_deps = 0;
  for (int k = 0; k < n; ++k) {
    max_row = std::max(max_row, ptr[k + 1] - ptr[k]);
    for (int e = ptr[k]; e < ptr[k + 1]; ++e) {
      int deps = 1;
      if (e < diag[k]) {
        const int i = col[e];
        if (!lower_only) {
          // A_kj -= L_ki U_ij for every later j of row k present in U's row i
          for (int e2 = e + 1; e2 < ptr[k + 1]; ++e2) {
            const int pos = find(diag[i] + 1, ptr[i + 1], col[e2]);
            if (pos >= 0) {
              pairs.push_back(make_int2(e2, pos));
              ++deps;
            }
          }
        } else {
          // A_kj -= L_ki L_ji^T for i < j <= k with (j, i) in the pattern
          for (int e2 = e + 1; e2 <= diag[k]; ++e2) {
            const int j = col[e2];
            if (j == k) {
              pairs.push_back(make_int2(e2, -1 - e));
            } else {
              const int pos = find(ptr[j], diag[j], i);
              if (pos >= 0) {
                pairs.push_back(make_int2(e2, pos));
                ++deps;
              }
            }
          }
        }
        max_deps = std::max(max_deps, deps);
      }
      pp[e + 1] = (int)pairs.size();
    }
  }
  plan->max_row = max_row;
  plan->max_deps = max_deps;
  BSP_TRY(upload(plan->pp, pp));
  BSP_TRY(upload(plan->pairs, pairs));
  pc->plan = plan;
  return BSP_OK;
}

static int analyse_factor_structure(bsp_precond_s* pc, bool lower_only) {
  const bsp_matrix_s* A = pc->A;
  const int n = A->n_rows;
  std::vector<int> ptr(n + 1, 0), col, diag(n, -1);
  std::vector<int64_t> perm;
  col.reserve(A->nnzb);
  perm.reserve(A->nnzb);
  std::vector<std::pair<int, int64_t>> row;
  for (int i = 0; i < n; ++i) {
    row.clear();
    for (int t = A->h_row_ptr[i]; t < A->h_row_ptr[i + 1]; ++t) {
      const int j = A->h_col_idx[t];
      if (!lower_only || j <= i) row.emplace_back(j, t);
    }
    std::sort(row.begin(), row.end());
    for (auto& pr : row) {
      if (pr.first == i) diag[i] = (int)col.size();
      col.push_back(pr.first);
      perm.push_back(pr.second);
    }
    ptr[i + 1] = (int)col.size();
    if (diag[i] < 0) {
      record_error("block row " + std::to_string(i) + " has no diagonal block");
      return BSP_ZERO_PIVOT;
    }
  }
  pc->f_nnzb = (int64_t)col.size();
  pc->h_perm = perm;
  BSP_TRY(upload(pc->f_ptr, ptr));
  BSP_TRY(upload(pc->f_col, col));
  BSP_TRY(upload(pc->f_diag, diag));
  BSP_TRY(upload(pc->d_perm, perm));
  // the sweeps are laid out beside the rest (ILU0: unit L, then U with U_ii^-1;
  // IChol0: L with L_ii^-1, then L^T with L_ii^-T)
  SweepPlanner sweeps;
  SweepEntries &lo = sweeps.lo, &up = sweeps.up;
  lo.ptr.assign(n + 1, 0);
  up.ptr.assign(n + 1, 0);
  lo.col.reserve(col.size());
  lo.blk.reserve(col.size());
  for (int i = 0; i < n; ++i) {
    for (int e = ptr[i]; e < diag[i]; ++e) {
      lo.col.push_back(col[e]);
      lo.blk.push_back(e);
      if (lower_only) up.ptr[col[e] + 1]++;
    }
    lo.ptr[i + 1] = (int)lo.col.size();
    if (lower_only) continue;
    for (int e = diag[i] + 1; e < ptr[i + 1]; ++e) {
      up.col.push_back(col[e]);
      up.blk.push_back(e);
    }
    up.ptr[i + 1] = (int)up.col.size();
  }
  if (lower_only) {
    // L^T backward: row i depends on rows j > i with L_ji present
    for (int i = 0; i < n; ++i) up.ptr[i + 1] += up.ptr[i];
    up.col.resize(up.ptr[n]);
    up.blk.resize(up.ptr[n]);
    std::vector<int> fill(up.ptr.begin(), up.ptr.end() - 1);
    for (int j = 0; j < n; ++j)
      for (int e = ptr[j]; e < diag[j]; ++e) {
        const int p = fill[col[e]]++;
        up.col[p] = j;
        up.blk[p] = e;
      }
  }
  sweeps.lo_d = lower_only;
  sweeps.up_d = true;
  sweeps.up_trans = sweeps.up_trans_d = lower_only;
  if (pc->applied) sweeps.start(n, pc->bs);
  // level orders and chain tasks on the sorted structure
  std::vector<int> order;
  auto deps_of = [](const SweepEntries& E) {
    return [&E](int i, auto&& f) {
      for (int t = E.ptr[i]; t < E.ptr[i + 1]; ++t) f(E.col[t]);
    };
  };
  pc->n_lev_lo = level_order(n, true, deps_of(lo), order);
  BSP_TRY(upload(pc->order_lo, order));
  BSP_TRY(make_tasks(pc, true, n, deps_of(lo)));
  pc->n_lev_up = level_order(n, false, deps_of(up), order);
  BSP_TRY(upload(pc->order_up, order));
  BSP_TRY(make_tasks(pc, false, n, deps_of(up)));
  if (lower_only) {
    BSP_TRY(upload(pc->t_ptr, up.ptr));
    BSP_TRY(upload(pc->t_row, up.col));
    BSP_TRY(upload(pc->t_blk, up.blk));
  }
  BSP_TRY(build_factor_plan(pc, n, ptr, col, diag, lower_only));
  return sweeps.finish(pc->wv_lo, pc->wv_up, pc->ss_lo, pc->ss_up);
}

// Factor storage for ILU0 / IChol0: the symbolic part from the matrix's cache
// (computed on first use), then A's values gathered into it on the device.
static int build_factor_structure(bsp_precond_s* pc, bool lower_only) {
  SymbolicCache& C = lower_only ? pc->A->sym->ichol : pc->A->sym->ilu;
  if (C.valid && (C.laid_out || !pc->applied)) {
    BSP_TRY(sym_transfer(pc, C, false));
  } else {
    BSP_TRY(analyse_factor_structure(pc, lower_only));
    BSP_TRY(sym_transfer(pc, C, true));
  }
  const int b2 = pc->bs * pc->bs;
  BSP_TRY(take(pc->A, pc->f_vals, pc->f_nnzb * b2));
  bsp::count_launch(), k_gather_blocks<<<grid_for(pc->h, pc->f_nnzb * b2, 256), 256, 0, pc->h->stream>>>(
      pc->f_nnzb, b2, pc->d_perm.get(), pc->A->vals.get(), pc->f_vals.get());
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

static int analyse_diag_structure(bsp_precond_s* pc) {
  const bsp_matrix_s* A = pc->A;
  const int n = A->n_rows;
  std::vector<int> diag(n, -1);
  for (int i = 0; i < n; ++i) {
    for (int t = A->h_row_ptr[i]; t < A->h_row_ptr[i + 1]; ++t)
      if (A->h_col_idx[t] == i) diag[i] = t;
    if (diag[i] < 0) {
      record_error("block row " + std::to_string(i) + " has no diagonal block");
      return BSP_ZERO_PIVOT;
    }
  }
  BSP_TRY(upload(pc->a_diag, diag));
  if (pc->kind == BSP_PC_SOR_LU || pc->kind == BSP_PC_SOR_CHOL) {
    std::vector<int> order;
    const auto& rp = A->h_row_ptr;
    const auto& ci = A->h_col_idx;
    // the dependent entries of a forward (j < i) and a backward sweep
    SweepPlanner sweeps;
    SweepEntries &lo = sweeps.lo, &up = sweeps.up;
    lo.ptr.assign(n + 1, 0);
    up.ptr.assign(n + 1, 0);
    for (int i = 0; i < n; ++i) {
      for (int t = rp[i]; t < rp[i + 1]; ++t) {
        if (ci[t] == i) continue;
        SweepEntries& E = ci[t] < i ? lo : up;
        E.col.push_back(ci[t]);
        E.blk.push_back(t);
      }
      lo.ptr[i + 1] = (int)lo.col.size();
      up.ptr[i + 1] = (int)up.col.size();
    }
    sweeps.in_place = true;
    sweeps.start(n, pc->bs);
    auto deps_of = [](const SweepEntries& E) {
      return [&E](int i, auto&& f) {
        for (int t = E.ptr[i]; t < E.ptr[i + 1]; ++t) f(E.col[t]);
      };
    };
    pc->n_lev_lo = level_order(n, true, deps_of(lo), order);
    BSP_TRY(upload(pc->order_lo, order));
    BSP_TRY(make_tasks(pc, true, n, deps_of(lo)));
    pc->n_lev_up = level_order(n, false, deps_of(up), order);
    BSP_TRY(upload(pc->order_up, order));
    BSP_TRY(make_tasks(pc, false, n, deps_of(up)));
    BSP_TRY(sweeps.finish(pc->wv_lo, pc->wv_up, pc->ss_lo, pc->ss_up));
  }
  return BSP_OK;
}

static int build_diag_inverse(bsp_precond_s* pc) {
  SymbolicCache& C = pc->A->sym->sor;
  const bool sor = pc->kind == BSP_PC_SOR_LU || pc->kind == BSP_PC_SOR_CHOL;
  if (C.valid && (!sor || C.n_task_lo > 0)) {
    BSP_TRY(sym_transfer(pc, C, false));
  } else {
    BSP_TRY(analyse_diag_structure(pc));
    BSP_TRY(sym_transfer(pc, C, true));
  }
  // makeADInv: invert every diagonal block (rows independent)
  return run_factor(pc, FACT_DIAG, nullptr, pc->A->row_ptr.get(), pc->A->col_idx.get(), pc->a_diag.get(),
                    pc->A->vals.get(), pc->n);
}

// The factors changed: every copy of them in sweep order is stale.
static void sweep_invalidate(bsp_precond_s* pc) {
  for (int k = 0; k < 3; ++k) {
    pc->vv_lo[k].valid = pc->vv_up[k].valid = false;
    pc->sv_lo[k].valid = pc->sv_up[k].valid = false;
  }
  pc->level_ordered = false;
}

static int make_lowp_copies(bsp_precond_s* pc) {
  if (pc->precision == BSP_PREC_F64) return BSP_OK;
  const int b2 = pc->bs * pc->bs;
  const int64_t nd = (int64_t)pc->n * b2;
  const int64_t nf = pc->f_nnzb * b2;
  if (pc->precision == BSP_PREC_F32) {
    BSP_TRY(take(pc->A, pc->dinv32, nd));
    bsp::count_launch(), k_convert<float><<<grid_for(pc->h, nd, 256), 256, 0, pc->h->stream>>>(nd, pc->dinv.get(), pc->dinv32.get());
    if (nf > 0) {
      BSP_TRY(take(pc->A, pc->f_vals32, nf));
      bsp::count_launch(), k_convert<float><<<grid_for(pc->h, nf, 256), 256, 0, pc->h->stream>>>(nf, pc->f_vals.get(), pc->f_vals32.get());
    }
  } else {
    BSP_TRY(take(pc->A, pc->dinv16, nd));
    bsp::count_launch(), k_convert<__nv_bfloat16><<<grid_for(pc->h, nd, 256), 256, 0, pc->h->stream>>>(nd, pc->dinv.get(), pc->dinv16.get());
    if (nf > 0) {
      BSP_TRY(take(pc->A, pc->f_vals16, nf));
      bsp::count_launch(), k_convert<__nv_bfloat16><<<grid_for(pc->h, nf, 256), 256, 0, pc->h->stream>>>(nf, pc->f_vals.get(), pc->f_vals16.get());
    }
  }
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

int precond_build(bsp_precond_s* pc) {
  const int n = pc->n, b2 = pc->bs * pc->bs;
  sweep_invalidate(pc);
  BSP_TRY(take(pc->A, pc->dinv, (size_t)std::max(n, 1) * b2));
  BSP_TRY(take(pc->A, pc->flags, std::max(n, 1)));
  BSP_TRY(take(pc->A, pc->ticket, 1));
  BSP_TRY(pc->wticket.alloc(1));
  BSP_CUDA_TRY(cudaMemset(pc->wticket.get(), 0, sizeof(unsigned)));
  BSP_CUDA_TRY(cudaMemset(pc->flags.get(), 0, std::max(n, 1) * sizeof(int)));
  switch (pc->kind) {
    case BSP_PC_NONE:
      return BSP_OK;
    case BSP_PC_DIAG_LU:
    case BSP_PC_DIAG_CHOL:
    case BSP_PC_SOR_LU:
    case BSP_PC_SOR_CHOL:
      BSP_TRY(build_diag_inverse(pc));
      break;
    case BSP_PC_ILU0:
      BSP_TRY(build_factor_structure(pc, false));
      BSP_TRY(run_factor(pc, FACT_ILU0, pc->order_lo.get(), pc->f_ptr.get(), pc->f_col.get(),
                         pc->f_diag.get(), pc->f_vals.get(), n));
      break;
    case BSP_PC_ICHOL0:
      BSP_TRY(build_factor_structure(pc, true));
      BSP_TRY(run_factor(pc, FACT_ICHOL0, pc->order_lo.get(), pc->f_ptr.get(), pc->f_col.get(),
                         pc->f_diag.get(), pc->f_vals.get(), n));
      break;
    default:
      record_error("unknown preconditioner kind");
      return BSP_INVALID;
  }
  return make_lowp_copies(pc);
}

__global__ void k_add_perm(int64_t nblk, int b2, const int64_t* __restrict__ perm, const double* __restrict__ dF,
                           double* __restrict__ f) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nblk * b2; e += (int64_t)gridDim.x * blockDim.x)
    f[e] += dF[perm[e / b2] * b2 + e % b2];
}

// f_b += relax * f0_b on every off-diagonal block b of the factor (strictly
// lower blocks of an L L^T factor, both triangles of an LU factor): the
// relaxation of the learned factors.  One warp per factor row; f0 may be f.
__global__ void k_relax_offdiag(int n, int b2, const int* __restrict__ f_ptr, const int* __restrict__ f_diag,
                                double relax, const double* f0, double* f) {
  const int lane = threadIdx.x & 31;
  const int warps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n; i += warps) {
    const int d = f_diag[i];
    for (int b = f_ptr[i]; b < f_ptr[i + 1]; ++b)
      if (b != d)
        for (int o = lane; o < b2; o += 32) f[(int64_t)b * b2 + o] += relax * f0[(int64_t)b * b2 + o];
  }
}

static int relax_offdiag(bsp_precond_s* pc, const double* f0) {
  if (pc->relax == 0.0 || pc->n == 0) return BSP_OK;
  const int grid = (int)std::min<int64_t>(((int64_t)pc->n * 32 + 255) / 256, (int64_t)pc->h->num_sms * 16);
  bsp::count_launch(), k_relax_offdiag<<<grid, 256, 0, pc->h->stream>>>(
      pc->n, pc->bs * pc->bs, pc->f_ptr.get(), pc->f_diag.get(), pc->relax, f0, pc->f_vals.get());
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

// Learned factors: the block-ILU0 factors (LU form) or the block-IChol0 factor
// (L L^T form), off-diagonal blocks scaled by 1 + relax, plus a correction dF
// given in A's block order (null: none); the diagonal inverses are recomputed
// from the corrected U_ii / L_ii (general inverses).
int precond_build_learned(bsp_precond_s* pc, const double* dF) {
  const int n = pc->n, b2 = pc->bs * pc->bs;
  sweep_invalidate(pc);
  BSP_TRY(take(pc->A, pc->dinv, (size_t)std::max(n, 1) * b2));
  BSP_TRY(take(pc->A, pc->flags, std::max(n, 1)));
  BSP_TRY(take(pc->A, pc->ticket, 1));
  BSP_TRY(pc->wticket.alloc(1));
  BSP_CUDA_TRY(cudaMemset(pc->wticket.get(), 0, sizeof(unsigned)));
  BSP_CUDA_TRY(cudaMemset(pc->flags.get(), 0, std::max(n, 1) * sizeof(int)));
  // LU form on the ILU0 factors; L L^T form on the IChol0 factor (A.lowTri())
  const bool llt = pc->kind == BSP_PC_LEARNED_LLT;
  BSP_TRY(build_factor_structure(pc, llt));
  BSP_TRY(run_factor(pc, llt ? FACT_ICHOL0 : FACT_ILU0, pc->order_lo.get(), pc->f_ptr.get(), pc->f_col.get(),
                     pc->f_diag.get(), pc->f_vals.get(), n));
  BSP_TRY(relax_offdiag(pc, pc->f_vals.get()));
  // dF null: no correction, so the diagonal blocks and the factorisation's own
  // inverses of them stand
  if (dF) {
    const int64_t tot = pc->f_nnzb * b2;
    if (tot > 0)
      bsp::count_launch(), k_add_perm<<<grid_for(pc->h, tot, 256), 256, 0, pc->h->stream>>>(
          pc->f_nnzb, b2, pc->d_perm.get(), dF, pc->f_vals.get());
    BSP_CUDA_TRY(cudaPeekAtLastError());
    BSP_TRY(run_factor(pc, FACT_DIAG, nullptr, pc->f_ptr.get(), pc->f_col.get(), pc->f_diag.get(),
                       pc->f_vals.get(), n));
  }
  return make_lowp_copies(pc);
}

// ---------------------------------------------------------------- apply
// z = M^{-1} r (z may alias r).  AT = double (FP64) or float (mixed precision).
template <typename VT, typename AT>
static void set_tasks(SweepP<VT, AT>& p, const bsp_precond_s* pc, bool lower) {
  p.task_row = lower ? pc->task_lo_row.get() : pc->task_up_row.get();
  p.task_len = lower ? pc->task_lo_len.get() : pc->task_up_len.get();
  p.n_tasks = lower ? pc->n_task_lo : pc->n_task_up;
  p.task_dir = lower ? 1 : -1;
}

template <typename AT> static int fill_sentinel(bsp_handle_s* h, AT* x, int64_t count) {
  if constexpr (sizeof(AT) == 8)
    bsp::count_launch(), k_fill_sentinel64<<<grid_for(h, count, 256), 256, 0, h->stream>>>(
        count, reinterpret_cast<unsigned long long*>(x));
  else
    bsp::count_launch(), k_fill_sentinel32<<<grid_for(h, count, 256), 256, 0, h->stream>>>(
        count, reinterpret_cast<unsigned*>(x));
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

template <typename VT> constexpr int prec_of() {
  return std::is_same<VT, double>::value ? BSP_PREC_F64 : std::is_same<VT, float>::value ? BSP_PREC_F32 : BSP_PREC_BF16;
}

// The copies in sweep order that an application in precision `prec` needs, and
// its vectors; made on first use.  Launches nothing that touches r or z.
static int wave_ready(bsp_precond_s* pc, int prec) {
  const bool sor = pc->kind == BSP_PC_SOR_LU || pc->kind == BSP_PC_SOR_CHOL;
  for (const bool lower : {true, false}) {
    const WaveSym& S = lower ? *pc->wv_lo : *pc->wv_up;
    WaveVals& V = lower ? pc->vv_lo[prec] : pc->vv_up[prec];
    if (sor && (lower ? pc->type < 0 : pc->type > 0)) continue;  // that direction is not swept
    if (V.valid) continue;
    const size_t vb = wave_val_bytes(S, prec);
    if (V.vals.n < vb) BSP_TRY(take(pc->A, V.vals, vb));
    if (sor) BSP_TRY(wave_gather(pc->h, S, prec, pc->A->vals.get(), pc->dinv.get(), V, true, pc->w));
    else BSP_TRY(wave_gather(pc->h, S, prec, pc->f_vals.get(), pc->dinv.get(), V));
  }
  const size_t n_lo = wave_item_values(*pc->wv_lo, 1), n_up = wave_item_values(*pc->wv_up, 1);
  const size_t need[3] = {sor ? 0 : n_up, sor ? 0 : n_lo, sor ? std::max(n_lo, n_up) : 0};
  for (int i = 0; i < 3; ++i)
    if (pc->s64[i].n < need[i]) BSP_TRY(take(pc->A, pc->s64[i], need[i]));
  return BSP_OK;
}
static int stream_ready(bsp_precond_s* pc, int prec) {
  for (const bool lower : {true, false}) {
    const StreamSym& S = lower ? *pc->ss_lo : *pc->ss_up;
    StreamVals& V = lower ? pc->sv_lo[prec] : pc->sv_up[prec];
    if (V.valid) continue;
    const size_t vb = stream_val_bytes(S, pc->bs, prec), db = stream_dval_bytes(S, pc->bs, prec);
    if (V.vals.n < vb) BSP_TRY(take(pc->A, V.vals, vb));
    if (db && V.dvals.n < db) BSP_TRY(take(pc->A, V.dvals, db));
    BSP_TRY(stream_gather(pc->h, S, pc->bs, prec, pc->f_vals.get(), pc->dinv.get(), V));
  }
  return BSP_OK;
}

// Which sweeps an application with FP64 vectors runs through.  Where the copies
// in sweep order do not fit memory the level-ordered kernels, which read the
// factors in place, take it (until the factors change).
enum class Path { kLevels, kWave, kStream };
static int sweep_path(bsp_precond_s* pc, int prec, const void* r, const void* z, Path* out) {
  *out = Path::kLevels;
  if (pc->level_ordered) return BSP_OK;
  const bool wave = pc->wv_lo && pc->wv_up;
  // the streamed sweeps read vectors in 16-byte pieces
  const bool stream = pc->ss_lo && pc->ss_up && reinterpret_cast<uintptr_t>(z) % 16 == 0 &&
                      reinterpret_cast<uintptr_t>(r) % 16 == 0;
  if (!wave && !stream) return BSP_OK;
  const int st = wave ? wave_ready(pc, prec) : stream_ready(pc, prec);
  if (st == BSP_OUT_OF_MEMORY) {
    record_error("");
    for (int k = 0; k < 3; ++k) {
      pc->vv_lo[k] = WaveVals{};
      pc->vv_up[k] = WaveVals{};
      pc->sv_lo[k] = StreamVals{};
      pc->sv_up[k] = StreamVals{};
    }
    pc->level_ordered = true;
    // a vector that was to grow has lost its old place
    for (auto& v : pc->s64)
      if (v.n < (size_t)pc->n * pc->bs) BSP_TRY(take(pc->A, v, (size_t)pc->n * pc->bs));
    return BSP_OK;
  }
  BSP_TRY(st);
  *out = wave ? Path::kWave : Path::kStream;
  return BSP_OK;
}

// z = M^{-1} r through the lock-step sweeps.
static int apply_wave(bsp_precond_s* pc, int prec, const double* r, double* z) {
  bsp_handle_s* h = pc->h;
  double *w = pc->s64[0].get(), *rp = pc->s64[1].get();
  BSP_TRY(wave_prepare(h, *pc->wv_lo, *pc->wv_up, r, rp, w, z));
  BSP_TRY(wave_sweep(h, *pc->wv_lo, prec, pc->vv_lo[prec], rp, w, pc->wticket.get()));
  return wave_sweep(h, *pc->wv_up, prec, pc->vv_up[prec], w, z, pc->wticket.get());
}

// The same through the streamed sweeps.
static int apply_stream(bsp_precond_s* pc, int prec, const double* r, double* z) {
  bsp_handle_s* h = pc->h;
  const int64_t nv = (int64_t)pc->n * pc->bs;
  double* w = pc->s64[0].get();
  BSP_TRY(fill_sentinel(h, w, nv));
  BSP_TRY(stream_sweep(h, *pc->ss_lo, pc->bs, prec, pc->sv_lo[prec], r, w, pc->ticket.get()));
  BSP_TRY(fill_sentinel(h, z, nv));
  return stream_sweep(h, *pc->ss_up, pc->bs, prec, pc->sv_up[prec], w, z, pc->ticket.get());
}

// z = M^{-1} r for SOR: nu sweeps each way of x_i = c_i - sum_dep (w D_i A_ij) x_j,
// c_i formed by a pass over the other entries before each (z may alias r).
template <typename VT>
static int apply_sor_wave(bsp_precond_s* pc, const double* r, double* z, const VT* avals, const VT* dinv,
                          const std::vector<int>& dirs) {
  bsp_handle_s* h = pc->h;
  const bsp_matrix_s* A = pc->A;
  constexpr int prec = prec_of<VT>();
  double *rp = pc->s64[2].get(), *bufs[2] = {pc->s64[0].get(), pc->s64[1].get()};
  const double* xold = nullptr;
  for (size_t s = 0; s < dirs.size(); ++s) {
    const bool fwd = dirs[s] < 0;
    const WaveSym& S = fwd ? *pc->wv_lo : *pc->wv_up;
    const WaveVals& V = fwd ? pc->vv_lo[prec] : pc->vv_up[prec];
    double* out = s + 1 == dirs.size() ? z : bufs[s & 1];
    BSP_TRY(wave_sor_prepare(h, S, prec, fwd, A->row_ptr.get(), A->col_idx.get(), avals, dinv, pc->w, r, xold, rp, out));
    BSP_TRY(wave_sweep(h, S, prec, V, rp, out, pc->wticket.get()));
    xold = out;
  }
  return BSP_OK;
}

// z = M^{-1} r (z may alias r).  Every sweep with dependencies writes into a
// buffer pre-filled with the sentinel and reads its right-hand side from a
// different buffer; sa, sb, sc are scratch vectors of n*bs values.
template <typename VT, typename AT>
static int apply_typed(bsp_precond_s* pc, const AT* r, AT* z, const VT* fvals, const VT* dinv,
                       const VT* avals, AT* sa, AT* sb, AT* sc) {
  bsp_handle_s* h = pc->h;
  const bsp_matrix_s* A = pc->A;
  const int n = pc->n, bs = pc->bs;
  const int64_t nv = (int64_t)n * bs;
  unsigned* tk = pc->ticket.get();
  SweepP<VT, AT> p{};
  p.n = n;
  p.flags = pc->flags.get();
  switch (pc->kind) {
    case BSP_PC_NONE:
      if (z != r) BSP_CUDA_TRY(cudaMemcpyAsync(z, r, (size_t)n * bs * sizeof(AT), cudaMemcpyDeviceToDevice, h->stream));
      return BSP_OK;
    case BSP_PC_DIAG_LU:
    case BSP_PC_DIAG_CHOL:
      p.range = RANGE_NONE;
      p.dinv = dinv;
      p.rhs = r;
      p.x = z;
      p.vals = avals;
      return launch_sweep<VT, AT, false, POST_D>(h, bs, p, tk);
    case BSP_PC_SOR_LU:
    case BSP_PC_SOR_CHOL: {
      // operator() (preconditioners.hpp:227-234): x = 0; nu backward, or nu
      // forward + nu backward, or nu forward sweeps; r = x.
      p.ptr = A->row_ptr.get();
      p.idx = A->col_idx.get();
      p.range = RANGE_SPLIT;
      p.vals = avals;
      p.dinv = dinv;
      p.w = (AT)pc->w;
      std::vector<int> dirs;
      if (pc->type < 0) dirs.assign(pc->nu, +1);
      else if (pc->type == 0) { dirs.assign(pc->nu, -1); dirs.insert(dirs.end(), pc->nu, +1); }
      else dirs.assign(pc->nu, -1);
      if constexpr (std::is_same<AT, double>::value) {
        Path path;
        BSP_TRY(sweep_path(pc, prec_of<VT>(), r, z, &path));
        if (path == Path::kWave) return apply_sor_wave<VT>(pc, r, z, avals, dinv, dirs);
        // an allocation may have given these another place
        sa = pc->s64[0].get(), sb = pc->s64[1].get(), sc = pc->s64[2].get();
      }
      const AT* rhs = r;
      if (z == r) {  // in place: keep a copy of the right-hand side
        BSP_CUDA_TRY(cudaMemcpyAsync(sc, r, nv * sizeof(AT), cudaMemcpyDeviceToDevice, h->stream));
        rhs = sc;
      }
      p.rhs = rhs;
      const AT* xold = nullptr;
      AT* bufs[2] = {sa, sb};
      for (size_t s = 0; s < dirs.size(); ++s) {
        const bool last = s + 1 == dirs.size();
        AT* out = last ? z : bufs[s & 1];
        BSP_TRY(fill_sentinel(h, out, nv));
        p.dep_dir = dirs[s];
        p.order = dirs[s] < 0 ? pc->order_lo.get() : pc->order_up.get();
        set_tasks(p, pc, dirs[s] < 0);
        p.xold = xold;
        p.x = out;
        BSP_TRY((launch_sweep<VT, AT, false, POST_SOR>(h, bs, p, tk)));
        xold = out;
      }
      return BSP_OK;
    }
    case BSP_PC_ILU0:
    case BSP_PC_LEARNED_LU: {
      if constexpr (std::is_same<AT, double>::value) {
        Path path;
        BSP_TRY(sweep_path(pc, prec_of<VT>(), r, z, &path));
        if (path == Path::kWave) return apply_wave(pc, prec_of<VT>(), r, z);
        if (path == Path::kStream) return apply_stream(pc, prec_of<VT>(), r, z);
        sa = pc->s64[0].get(), sb = pc->s64[1].get(), sc = pc->s64[2].get();
      }
      p.ptr = pc->f_ptr.get();
      p.idx = pc->f_col.get();
      p.diag = pc->f_diag.get();
      p.vals = fvals;
      p.dinv = dinv;
      // forward: unit L
      p.range = RANGE_LOWER;
      p.order = pc->order_lo.get();
      set_tasks(p, pc, true);
      p.rhs = r;
      p.x = sa;
      BSP_TRY(fill_sentinel(h, sa, nv));
      BSP_TRY((launch_sweep<VT, AT, false, POST_NONE>(h, bs, p, tk)));
      // backward: U with inverted diagonal
      p.range = RANGE_UPPER;
      p.order = pc->order_up.get();
      set_tasks(p, pc, false);
      p.rhs = sa;
      p.x = z;
      BSP_TRY(fill_sentinel(h, z, nv));
      return launch_sweep<VT, AT, false, POST_D>(h, bs, p, tk);
    }
    case BSP_PC_ICHOL0:
    case BSP_PC_LEARNED_LLT: {
      if constexpr (std::is_same<AT, double>::value) {
        Path path;
        BSP_TRY(sweep_path(pc, prec_of<VT>(), r, z, &path));
        if (path == Path::kWave) return apply_wave(pc, prec_of<VT>(), r, z);
        if (path == Path::kStream) return apply_stream(pc, prec_of<VT>(), r, z);
        sa = pc->s64[0].get(), sb = pc->s64[1].get(), sc = pc->s64[2].get();
      }
      p.ptr = pc->f_ptr.get();
      p.idx = pc->f_col.get();
      p.diag = pc->f_diag.get();
      p.vals = fvals;
      p.dinv = dinv;
      p.range = RANGE_LOWER;
      p.order = pc->order_lo.get();
      set_tasks(p, pc, true);
      p.rhs = r;
      p.x = sa;
      BSP_TRY(fill_sentinel(h, sa, nv));
      BSP_TRY((launch_sweep<VT, AT, false, POST_D>(h, bs, p, tk)));
      // backward: L^T through the transposed structure, diagonal L_ii^{-T}
      p.ptr = pc->t_ptr.get();
      p.idx = pc->t_row.get();
      p.blk = pc->t_blk.get();
      p.range = RANGE_ALL;
      p.order = pc->order_up.get();
      set_tasks(p, pc, false);
      p.rhs = sa;
      p.x = z;
      BSP_TRY(fill_sentinel(h, z, nv));
      return launch_sweep<VT, AT, true, POST_DT>(h, bs, p, tk);
    }
    default:
      return BSP_INVALID;
  }
}

// Transposed structures and tasks for M^-T (LU-type factors).
static int build_transposed(bsp_precond_s* pc) {
  const bsp_matrix_s* A = pc->A;
  const int n = A->n_rows;
  // the factor's row-sorted structure (the order analyse_factor_structure uses)
  std::vector<int> ptr(n + 1, 0), col;
  col.reserve(A->nnzb);
  std::vector<int> row;
  for (int i = 0; i < n; ++i) {
    row.assign(A->h_col_idx.begin() + A->h_row_ptr[i], A->h_col_idx.begin() + A->h_row_ptr[i + 1]);
    std::sort(row.begin(), row.end());
    col.insert(col.end(), row.begin(), row.end());
    ptr[i + 1] = (int)col.size();
  }
  // per column: strictly-upper entries (rows i < j) and strictly-lower (rows j > i)
  std::vector<std::vector<std::pair<int, int64_t>>> up(n), lo(n);
  for (int i = 0; i < n; ++i)
    for (int e = ptr[i]; e < ptr[i + 1]; ++e) {
      const int j = col[e];
      if (j > i) up[j].emplace_back(i, e);
      else if (j < i) lo[j].emplace_back(i, e);
    }
  auto flatten = [&](const std::vector<std::vector<std::pair<int, int64_t>>>& lists, DevBuf<int>& dptr,
                     DevBuf<int>& drow, DevBuf<int64_t>& dblk) -> int {
    std::vector<int> p(n + 1, 0), r;
    std::vector<int64_t> b;
    for (int c = 0; c < n; ++c) {
      for (auto& pr : lists[c]) {
        r.push_back(pr.first);
        b.push_back(pr.second);
      }
      p[c + 1] = (int)r.size();
    }
    if (r.empty()) {
      r.push_back(0);
      b.push_back(0);
    }
    BSP_TRY(upload(dptr, p));
    BSP_TRY(upload(drow, r));
    BSP_TRY(upload(dblk, b));
    return BSP_OK;
  };
  BSP_TRY(flatten(up, pc->tu_ptr, pc->tu_row, pc->tu_blk));
  BSP_TRY(flatten(lo, pc->tl_ptr, pc->tl_row, pc->tl_blk));
  std::vector<int> order, trow, tlen;
  auto up_deps = [&](int j, auto&& f) {
    for (auto& pr : up[j]) f(pr.first);
  };
  auto lo_deps = [&](int i, auto&& f) {
    for (auto& pr : lo[i]) f(pr.first);
  };
  level_order(n, true, up_deps, order);
  BSP_TRY(upload(pc->order_tu, order));
  pc->n_task_tu = build_tasks(n, true, up_deps, trow, tlen);
  BSP_TRY(upload(pc->task_tu_row, trow));
  BSP_TRY(upload(pc->task_tu_len, tlen));
  level_order(n, false, lo_deps, order);
  BSP_TRY(upload(pc->order_tl, order));
  pc->n_task_tl = build_tasks(n, false, lo_deps, trow, tlen);
  BSP_TRY(upload(pc->task_tl_row, trow));
  BSP_TRY(upload(pc->task_tl_len, tlen));
  pc->has_trans = true;
  return BSP_OK;
}

// out = M^-T g = L^-T (U^-T g): a forward sweep over U's columns with the
// transposed inverted diagonal, then a backward sweep over L's columns (unit
// diagonal).  FP64; g, w and out must be distinct.
int precond_apply_transposed(bsp_precond_s* pc, const double* g, double* w, double* out) {
  if (pc->kind != BSP_PC_ILU0 && pc->kind != BSP_PC_LEARNED_LU) return BSP_INVALID;
  if (!pc->has_trans) BSP_TRY(build_transposed(pc));
  bsp_handle_s* h = pc->h;
  const int n = pc->n, bs = pc->bs;
  const int64_t nv = (int64_t)n * bs;
  SweepP<double, double> p{};
  p.n = n;
  p.flags = pc->flags.get();
  p.vals = pc->f_vals.get();
  p.dinv = pc->dinv.get();
  p.range = RANGE_ALL;
  // U^T w = g, forward
  p.ptr = pc->tu_ptr.get();
  p.idx = pc->tu_row.get();
  p.blk = pc->tu_blk.get();
  p.order = pc->order_tu.get();
  p.task_row = pc->task_tu_row.get();
  p.task_len = pc->task_tu_len.get();
  p.n_tasks = pc->n_task_tu;
  p.task_dir = 1;
  p.rhs = g;
  p.x = w;
  BSP_TRY(fill_sentinel(h, w, nv));
  BSP_TRY((launch_sweep<double, double, true, POST_DT>(h, bs, p, pc->ticket.get())));
  // L^T out = w, backward
  p.ptr = pc->tl_ptr.get();
  p.idx = pc->tl_row.get();
  p.blk = pc->tl_blk.get();
  p.order = pc->order_tl.get();
  p.task_row = pc->task_tl_row.get();
  p.task_len = pc->task_tl_len.get();
  p.n_tasks = pc->n_task_tl;
  p.task_dir = -1;
  p.rhs = w;
  p.x = out;
  BSP_TRY(fill_sentinel(h, out, nv));
  return launch_sweep<double, double, true, POST_NONE>(h, bs, p, pc->ticket.get());
}

__global__ void k_copy_add_perm(int64_t nblk, int b2, const int64_t* __restrict__ perm, const double* __restrict__ f0,
                                const double* __restrict__ dF, double* __restrict__ f) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nblk * b2; e += (int64_t)gridDim.x * blockDim.x)
    f[e] = f0[e] + dF[perm[e / b2] * b2 + e % b2];
}

// Structure of a learned-LU preconditioner whose factors are set by
// precond_learned_refresh (no factorisation).
int precond_learned_init(bsp_precond_s* pc) {
  const int n = pc->n, b2 = pc->bs * pc->bs;
  BSP_TRY(take(pc->A, pc->dinv, (size_t)std::max(n, 1) * b2));
  BSP_TRY(take(pc->A, pc->flags, std::max(n, 1)));
  BSP_TRY(take(pc->A, pc->ticket, 1));
  BSP_TRY(pc->wticket.alloc(1));
  BSP_CUDA_TRY(cudaMemset(pc->wticket.get(), 0, sizeof(unsigned)));
  BSP_CUDA_TRY(cudaMemset(pc->flags.get(), 0, std::max(n, 1) * sizeof(int)));
  return build_factor_structure(pc, pc->kind == BSP_PC_LEARNED_LLT);
}

// work's factors = ilu's factors + dF (A order) + work->relax * ilu's off-diagonal
// factor blocks; work shares ilu's structure
// (both built on the same matrix) and gets fresh diagonal inverses.
int precond_learned_refresh(bsp_precond_s* work, const bsp_precond_s* ilu, const double* dF) {
  if (work->f_nnzb != ilu->f_nnzb || work->n != ilu->n || work->bs != ilu->bs) return BSP_INVALID;
  sweep_invalidate(work);
  const int b2 = work->bs * work->bs;
  const int64_t tot = work->f_nnzb * b2;
  if (tot > 0)
    bsp::count_launch(), k_copy_add_perm<<<grid_for(work->h, tot, 256), 256, 0, work->h->stream>>>(
        work->f_nnzb, b2, work->d_perm.get(), ilu->f_vals.get(), dF, work->f_vals.get());
  BSP_CUDA_TRY(cudaPeekAtLastError());
  BSP_TRY(relax_offdiag(work, ilu->f_vals.get()));
  return run_factor(work, FACT_DIAG, nullptr, work->f_ptr.get(), work->f_col.get(), work->f_diag.get(),
                    work->f_vals.get(), work->n);
}

// z = M^{-1} r.  precision selects the stored factors (FP64 / FP32 / BF16);
// vec64 selects FP64 vectors (the Krylov path, always FP64 accumulation) or
// FP32 vectors (low-precision vectors, FP32 accumulation).
int precond_apply_typed(bsp_precond_s* pc, int precision, bool vec64, const void* r, void* z) {
  const size_t nv = (size_t)std::max(pc->n, 1) * pc->bs;
  if (precision == BSP_PREC_F32 && !pc->dinv32.get()) return BSP_INVALID;
  if (precision == BSP_PREC_BF16 && !pc->dinv16.get()) return BSP_INVALID;
  if (precision == BSP_PREC_F64 || vec64) {
    for (auto& s : pc->s64)
      if (s.n < nv) BSP_TRY(take(pc->A, s, nv));
    double *a = pc->s64[0].get(), *b = pc->s64[1].get(), *c = pc->s64[2].get();
    if (precision == BSP_PREC_F64)
      return apply_typed<double, double>(pc, (const double*)r, (double*)z, pc->f_vals.get(),
                                         pc->dinv.get(), pc->A->vals.get(), a, b, c);
    if (precision == BSP_PREC_F32)
      return apply_typed<float, double>(pc, (const double*)r, (double*)z, pc->f_vals32.get(),
                                        pc->dinv32.get(), pc->A->vals32.get(), a, b, c);
    return apply_typed<__nv_bfloat16, double>(pc, (const double*)r, (double*)z, pc->f_vals16.get(),
                                              pc->dinv16.get(), pc->A->vals16.get(), a, b, c);
  }
  for (auto& s : pc->s32)
    if (s.n < nv) BSP_TRY(take(pc->A, s, nv));
  float *a = pc->s32[0].get(), *b = pc->s32[1].get(), *c = pc->s32[2].get();
  if (precision == BSP_PREC_F32)
    return apply_typed<float, float>(pc, (const float*)r, (float*)z, pc->f_vals32.get(),
                                     pc->dinv32.get(), pc->A->vals32.get(), a, b, c);
  return apply_typed<__nv_bfloat16, float>(pc, (const float*)r, (float*)z, pc->f_vals16.get(),
                                           pc->dinv16.get(), pc->A->vals16.get(), a, b, c);
}

int precond_apply(bsp_precond_s* pc, int precision, const void* r, void* z) {
  return precond_apply_typed(pc, precision, true, r, z);
}

// Make the low-precision copies of the factors (and of A for SOR/Diag) that a
// mixed-precision solve needs, if the preconditioner was built without them.
int precond_ensure_precision(bsp_precond_s* pc, int precision) {
  if (precision == BSP_PREC_F64) return BSP_OK;
  if (precision == BSP_PREC_F32 && pc->dinv32.get()) return BSP_OK;
  if (precision == BSP_PREC_BF16 && pc->dinv16.get()) return BSP_OK;
  if (pc->kind == BSP_PC_SOR_LU || pc->kind == BSP_PC_SOR_CHOL || pc->kind == BSP_PC_DIAG_LU ||
      pc->kind == BSP_PC_DIAG_CHOL)
    BSP_TRY(bsp_matrix_make_lowp(pc->A, precision == BSP_PREC_F32 ? BSP_F32 : BSP_BF16));
  const int saved = pc->precision;
  pc->precision = precision;
  const int s = make_lowp_copies(pc);
  pc->precision = saved;
  return s;
}

int precond_check_status(bsp_precond_s* pc) {
  DevStatus st;
  BSP_TRY(read_status(pc->h, &st));
  if (st.code != 0) {
    record_error(std::string("preconditioner apply: ") + bsp_status_string(st.code) +
                 " at block row " + std::to_string(st.where));
    return st.code;
  }
  return BSP_OK;
}

int precond_create(bsp_handle_s* h, bsp_matrix_s* A, const bsp_precond_params* params, bool applied,
                   bsp_precond_s** out) {
  if (!h || !A || !params || !out) return BSP_INVALID;
  *out = nullptr;
  if (A->n_rows != A->n_cols) {
    record_error("preconditioners need a square matrix");
    return BSP_INVALID;
  }
  if (A->bs > 32) {
    record_error("preconditioners support block sizes up to 32");
    return BSP_INVALID;
  }
  if (A->cbs && params->kind == BSP_PC_ICHOL0) {
    // the reference's IChol0 is real only (blocksp_solvers.hpp:485)
    record_error("IChol0 is not defined for complex matrices");
    return BSP_INVALID;
  }
  BSP_CUDA_TRY(cudaSetDevice(h->device));
  auto pc = std::make_unique<bsp_precond_s>();
  pc->h = h;
  pc->device = h->device;
  pc->A = A;
  pc->kind = params->kind;
  pc->n = A->n_rows;
  pc->bs = A->bs;
  pc->w = params->sor_w;
  pc->nu = params->sor_nu;
  pc->type = params->sor_type;
  pc->precision = params->precision;
  pc->applied = applied;
  if (pc->kind == BSP_PC_SOR_LU || pc->kind == BSP_PC_SOR_CHOL) {
    if (pc->nu < 1) {
      record_error("SOR needs nu >= 1");
      return BSP_INVALID;
    }
  }
  if (pc->precision != BSP_PREC_F64) {
    BSP_TRY(bsp_matrix_make_lowp(A, pc->precision == BSP_PREC_F32 ? BSP_F32 : BSP_BF16));
  }
  BSP_TRY(precond_build(pc.get()));
  BSP_CUDA_TRY(cudaStreamSynchronize(h->stream));
  *out = pc.release();
  return BSP_OK;
}

}  // namespace bsp

// ================================================================= C ABI
extern "C" {

int bsp_precond_create(bsp_handle_t h, bsp_matrix_t A, const bsp_precond_params* params,
                       bsp_precond_t* out) {
  return precond_create(h, A, params, true, out);
}

int bsp_precond_destroy(bsp_precond_t pc) {
  if (!pc) return BSP_OK;
  cudaSetDevice(pc->device);
  // the matrix outlives its preconditioners: its bin keeps their device memory
  // for the next preconditioner built on it (no cudaFree / cudaMalloc pair)
  if (pc->A && cudaDeviceSynchronize() == cudaSuccess) {
    bsp_matrix_s* A = pc->A;
    give(A, pc->f_vals); give(A, pc->f_vals32); give(A, pc->f_vals16);
    give(A, pc->dinv); give(A, pc->dinv32); give(A, pc->dinv16);
    give(A, pc->f_ptr); give(A, pc->f_col); give(A, pc->f_diag); give(A, pc->d_perm);
    give(A, pc->t_ptr); give(A, pc->t_row); give(A, pc->t_blk); give(A, pc->a_diag);
    give(A, pc->order_lo); give(A, pc->order_up);
    give(A, pc->task_lo_row); give(A, pc->task_lo_len); give(A, pc->task_up_row); give(A, pc->task_up_len);
    give(A, pc->flags);
    for (int i = 0; i < 3; ++i) {
      give(A, pc->s64[i]);
      give(A, pc->s32[i]);
      give(A, pc->vv_lo[i].vals);
      give(A, pc->vv_up[i].vals);
      give(A, pc->sv_lo[i].vals); give(A, pc->sv_lo[i].dvals);
      give(A, pc->sv_up[i].vals); give(A, pc->sv_up[i].dvals);
    }
  }
  delete pc;
  return BSP_OK;
}

int bsp_precond_apply_dev(bsp_handle_t h, bsp_precond_t pc, double* r) {
  if (!h || !pc || !r) return BSP_INVALID;
  BSP_CUDA_TRY(cudaSetDevice(h->device));
  return precond_apply(pc, BSP_PREC_F64, r, r);
}

int bsp_precond_apply(bsp_handle_t h, bsp_precond_t pc, double* r_host) {
  if (!h || !pc || !r_host) return BSP_INVALID;
  BSP_CUDA_TRY(cudaSetDevice(h->device));
  const size_t nv = (size_t)pc->n * pc->bs;
  BSP_TRY(h->stage(nv, 1));
  double* d = h->stage_in.get();
  BSP_CUDA_TRY(cudaMemcpyAsync(d, r_host, nv * sizeof(double), cudaMemcpyHostToDevice, h->stream));
  BSP_TRY(precond_apply(pc, BSP_PREC_F64, d, d));
  BSP_CUDA_TRY(cudaMemcpyAsync(r_host, d, nv * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  BSP_CUDA_TRY(cudaStreamSynchronize(h->stream));
  return precond_check_status(pc);
}

int bsp_precond_export(bsp_precond_t pc, double* vals_host, int64_t capacity) {
  if (!pc || !vals_host) return BSP_INVALID;
  BSP_CUDA_TRY(cudaSetDevice(pc->device));
  const int b2 = pc->bs * pc->bs;
  if (pc->kind == BSP_PC_ILU0 || pc->kind == BSP_PC_ICHOL0 || pc->kind == BSP_PC_LEARNED_LU ||
      pc->kind == BSP_PC_LEARNED_LLT) {
    // blocks in the caller's layout: ILU0 / learned LU in A's block order; IChol0 in the
    // order of A.lowTri() (A's rows, blocks with col <= row in stored order)
    const int64_t nf = pc->f_nnzb;
    if (capacity < nf * b2) return BSP_INVALID;
    std::vector<double> f(nf * b2);
    BSP_CUDA_TRY(cudaMemcpy(f.data(), pc->f_vals.get(), f.size() * sizeof(double), cudaMemcpyDeviceToHost));
    if (pc->kind != BSP_PC_ICHOL0 && pc->kind != BSP_PC_LEARNED_LLT) {
      for (int64_t e = 0; e < nf; ++e)
        std::copy(f.begin() + e * b2, f.begin() + (e + 1) * b2, vals_host + pc->h_perm[e] * b2);
    } else {
      // rank of each A block among the lower blocks of its row, in A order
      std::vector<int64_t> low_pos(pc->A->nnzb, -1);
      int64_t c = 0;
      for (int i = 0; i < pc->n; ++i)
        for (int t = pc->A->h_row_ptr[i]; t < pc->A->h_row_ptr[i + 1]; ++t)
          if (pc->A->h_col_idx[t] <= i) low_pos[t] = c++;
      for (int64_t e = 0; e < nf; ++e)
        std::copy(f.begin() + e * b2, f.begin() + (e + 1) * b2, vals_host + low_pos[pc->h_perm[e]] * b2);
    }
  } else {
    if (capacity < (int64_t)pc->n * b2) return BSP_INVALID;
    BSP_CUDA_TRY(cudaMemcpy(vals_host, pc->dinv.get(), (size_t)pc->n * b2 * sizeof(double), cudaMemcpyDeviceToHost));
  }
  return BSP_OK;
}

int bsp_precond_info(bsp_precond_t pc, int* kind, int* n_levels_lower, int* n_levels_upper,
                     int64_t* factor_nnzb) {
  if (!pc) return BSP_INVALID;
  if (kind) *kind = pc->kind;
  if (n_levels_lower) *n_levels_lower = pc->n_lev_lo;
  if (n_levels_upper) *n_levels_upper = pc->n_lev_up;
  if (factor_nnzb) *factor_nnzb = pc->f_nnzb;
  return BSP_OK;
}

}  // extern "C"
