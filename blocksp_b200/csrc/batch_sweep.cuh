// batch_sweep.cuh — the batched solver's level-ordered sweeps.
//
// They run a group whose rows the lock-step sweeps (sweep_wave.cuh) would cut
// into super-tasks that follow one another: sweep_cost.h states the rule.  An
// iteration of 12 systems of 10,000 rows, one right-hand side, lock-step | these,
// in us: 2D grids of 4 x 4 blocks 214 | 939, the same in random order 1024 | 206,
// Delaunay meshes of 8 x 8 blocks 1842 | 663.
#pragma once
#include "blockops.cuh"
#include "sentinel.cuh"

namespace bsp {

// Multi-RHS sync-free IChol0 sweeps over the chains of every active system.
// TRANS = false: w_i = L_ii^-1 (r_i - sum_{j<i} L_ij w_j)      (forward, L by rows)
// TRANS = true:  z_i = L_ii^-T (w_i - sum_{j>i} L_ji^T z_j)    (backward, L by columns)
// (blocksp_preconditioners.hpp:432-489, per RHS.)
struct BSweepP {
  int n_tasks;
  const int* task_row;
  const int* task_len;
  const int* task_sys;
  int task_dir;
  const int* sys_active;
  const int* ptr;
  const int* idx;
  const int64_t* blk;  // null: entry index
  const int* diag;     // forward: entries [ptr[i], diag[i])
  const double* vals;
  const double* dinv;
  const double* rhs;
  double* x;
  unsigned* ticket;
  DevStatus* st;
  unsigned spin_limit;  // polls before a wait gives up with BSP_TIMEOUT
};

constexpr int kBSweepThreads = 256;

template <int BS, int R, bool TRANS>
__global__ void __launch_bounds__(kBSweepThreads) k_bt_sweep(const BSweepP p) {
  using M = BlockMap<BS, double>;
  using CV = typename Chunk<double>::vec;
  constexpr int V = M::V, G = M::G, P = M::P, CPR = M::CPR, RPP = M::RPP, CPB = M::CPB;
  constexpr int GPC = kBSweepThreads / G;
  constexpr int LD = R * BS;
  // dependency entries whose blocks are loaded ahead: fewer with more RHS,
  // whose x values take the registers
  constexpr int NPF = (P == 1) ? (R >= 4 ? 2 : 4) : (P == 2 && R < 4 ? 2 : 1);
  constexpr int XV = TRANS ? P : V;
  __shared__ double sm_s[GPC][LD];
  __shared__ double sm_x[GPC][LD];
  const int gl = threadIdx.x % G;
  const int gid = threadIdx.x / G;
  const int lane = threadIdx.x & 31;
  const int gbase = lane - gl;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << gbase);
  const int c0 = (gl % CPR) * V;
  const CV* vb = reinterpret_cast<const CV*>(p.vals);
  double* s = sm_s[gid];
  double* xs = sm_x[gid];
  while (true) {
    int t = 0;
    if (gl == 0) t = (int)atomicAdd(p.ticket, 1u);
    t = __shfl_sync(gmask, t, gbase);
    if (t >= p.n_tasks) break;
    if (!p.sys_active[__ldg(p.task_sys + t)]) continue;
    const int i0 = __ldg(p.task_row + t);
    const int len = __ldg(p.task_len + t);
    CV nf[NPF][P], nd[P];
    int nbeg, nend;
    auto range = [&](int r, int& b0, int& b1) {
      b0 = __ldg(p.ptr + r);
      b1 = TRANS ? __ldg(p.ptr + r + 1) : __ldg(p.diag + r);
    };
    auto prefetch = [&](int r, int& b0, int& b1) {
      range(r, b0, b1);
#pragma unroll
      for (int u = 0; u < NPF; ++u) {
        if (b0 + u < b1) {
          const int64_t b = p.blk ? __ldg(p.blk + b0 + u) : (int64_t)(b0 + u);
#pragma unroll
          for (int q = 0; q < P; ++q) nf[u][q] = ld_stream(vb + b * CPB + q * G + gl);
        }
      }
      const CV* db = reinterpret_cast<const CV*>(p.dinv) + (int64_t)r * CPB;
#pragma unroll
      for (int q = 0; q < P; ++q) nd[q] = ld_stream(db + q * G + gl);
    };
    prefetch(i0, nbeg, nend);
    for (int step = 0; step < len; ++step) {
      const int i = i0 + step * p.task_dir;
      const int prev = step > 0 ? i - p.task_dir : -1;
      const int beg = nbeg, end = nend;
      CV pf[NPF][P], pd[P];
#pragma unroll
      for (int u = 0; u < NPF; ++u)
#pragma unroll
        for (int q = 0; q < P; ++q) pf[u][q] = nf[u][q];
#pragma unroll
      for (int q = 0; q < P; ++q) pd[q] = nd[q];
      if (step + 1 < len) prefetch(i + p.task_dir, nbeg, nend);
      double acc[P][R];   // forward: per block row q and RHS
      double tac[R][V];   // backward: per RHS and column
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int q = 0; q < P; ++q) acc[q][r] = 0.0;
#pragma unroll
        for (int v = 0; v < V; ++v) tac[r][v] = 0.0;
      }
      // x values of dependency j for every RHS: from shared memory when j is
      // the chain's previous row, else from global memory (polled)
      auto load_x = [&](bool from_prev, int j, double (&xv)[R][XV]) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if constexpr (!TRANS) {
            if (from_prev) {
#pragma unroll
              for (int v = 0; v < V; ++v) xv[r][v] = xs[r * BS + c0 + v];
            } else {
              ld_vec_cg<V>(p.x + (int64_t)j * LD + r * BS + c0, xv[r]);
            }
          } else {
#pragma unroll
            for (int q = 0; q < P; ++q) {
              const int rr = q * RPP + gl / CPR;
              xv[r][q] = from_prev ? xs[r * BS + rr] : __ldcg(p.x + (int64_t)j * LD + r * BS + rr);
            }
          }
        }
      };
      auto poll_x = [&](int j, double (&xv)[R][XV]) {
        bool pending = false;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < XV; ++v) pending |= is_sentinel(xv[r][v]);
        unsigned spins = 0;
        while (pending) {
          poll_pause(spins);
          pending = false;
#pragma unroll
          for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int v = 0; v < XV; ++v) {
              const int64_t k = TRANS ? (int64_t)j * LD + r * BS + v * RPP + gl / CPR
                                      : (int64_t)j * LD + r * BS + c0 + v;
              xv[r][v] = ld_poll(p.x + k);
              pending |= is_sentinel(xv[r][v]);
            }
          }
          if (pending) {
            if (++spins > p.spin_limit) {
              set_status(p.st, BSP_TIMEOUT, i);
              break;
            }
            if ((spins & 255u) == 0u && *reinterpret_cast<volatile int*>(&p.st->code) != 0) break;
          }
        }
      };
      auto fma_entry = [&](const CV (&a)[P], const double (&xv)[R][XV]) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          double av[V];
          unpack(a[q], av);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if constexpr (!TRANS) {
#pragma unroll
              for (int v = 0; v < V; ++v) acc[q][r] = fma(av[v], xv[r][v], acc[q][r]);
            } else {
#pragma unroll
              for (int v = 0; v < V; ++v) tac[r][v] = fma(av[v], xv[r][q], tac[r][v]);
            }
          }
        }
      };
      {
        double xv[NPF][R][XV];
        int jj[NPF];
        bool has[NPF];
#pragma unroll
        for (int u = 0; u < NPF; ++u) {
          has[u] = beg + u < end;
          if (has[u]) {
            jj[u] = __ldg(p.idx + beg + u);
            load_x(jj[u] == prev, jj[u], xv[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < NPF; ++u) {
          if (has[u]) {
            if (jj[u] != prev) poll_x(jj[u], xv[u]);
            fma_entry(pf[u], xv[u]);
          }
        }
      }
      for (int e = beg + NPF; e < end; ++e) {
        const int j = __ldg(p.idx + e);
        const int64_t b = p.blk ? __ldg(p.blk + e) : (int64_t)e;
        CV a[P];
#pragma unroll
        for (int q = 0; q < P; ++q) a[q] = ld_stream(vb + b * CPB + q * G + gl);
        double xv[R][XV];
        load_x(j == prev, j, xv);
        if (j != prev) poll_x(j, xv);
        fma_entry(a, xv);
      }
      // s = rhs_i - sum
      if constexpr (!TRANS) {
#pragma unroll
        for (int q = 0; q < P; ++q)
#pragma unroll
          for (int r = 0; r < R; ++r) acc[q][r] = row_reduce<CPR>(acc[q][r], gmask);
        if (gl % CPR == 0) {
#pragma unroll
          for (int q = 0; q < P; ++q) {
            const int rr = q * RPP + gl / CPR;
#pragma unroll
            for (int r = 0; r < R; ++r)
              s[r * BS + rr] = __ldcg(p.rhs + (int64_t)i * LD + r * BS + rr) - acc[q][r];
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v)
#pragma unroll
            for (int o = CPR; o < G; o <<= 1) tac[r][v] += __shfl_xor_sync(gmask, tac[r][v], o);
        if (gl < CPR) {
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int v = 0; v < V; ++v)
              s[r * BS + c0 + v] = __ldcg(p.rhs + (int64_t)i * LD + r * BS + c0 + v) - tac[r][v];
        }
      }
      __syncwarp(gmask);
      if constexpr (!TRANS) {
        // x_i = L_ii^-1 s: lane holds Dinv[row q][c0..c0+V)
#pragma unroll
        for (int q = 0; q < P; ++q) {
          double av[V];
          unpack(pd[q], av);
          double o[R];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            o[r] = 0.0;
#pragma unroll
            for (int v = 0; v < V; ++v) o[r] = fma(av[v], s[r * BS + c0 + v], o[r]);
            o[r] = row_reduce<CPR>(o[r], gmask);
          }
          if (gl % CPR == 0) {
            const int rr = q * RPP + gl / CPR;
#pragma unroll
            for (int r = 0; r < R; ++r) {
              p.x[(int64_t)i * LD + r * BS + rr] = o[r];
              xs[r * BS + rr] = o[r];
            }
          }
        }
      } else {
        // x_i = L_ii^-T s: lane holds Dinv[rr][c0..c0+V) and adds Dinv[rr][c] s[rr]
        double o[R][V];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v) o[r][v] = 0.0;
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const int rr = q * RPP + gl / CPR;
          double av[V];
          unpack(pd[q], av);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double sr = s[r * BS + rr];
#pragma unroll
            for (int v = 0; v < V; ++v) o[r][v] = fma(av[v], sr, o[r][v]);
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v)
#pragma unroll
            for (int off = CPR; off < G; off <<= 1) o[r][v] += __shfl_xor_sync(gmask, o[r][v], off);
        if (gl < CPR) {
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int v = 0; v < V; ++v) {
              p.x[(int64_t)i * LD + r * BS + c0 + v] = o[r][v];
              xs[r * BS + c0 + v] = o[r][v];
            }
        }
      }
      __syncwarp(gmask);
    }
  }
}

}  // namespace bsp
