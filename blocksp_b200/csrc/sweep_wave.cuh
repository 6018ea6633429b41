// sweep_wave.cuh — the lock-step block triangular sweep kernel (sm_100a).
//
// One CTA (one per SM) runs one super-task of a plan (wave_plan.h) at a time,
// taken with an atomic ticket in dependency-level order.  Its warps have fixed
// roles:
//   * two sets of 8 compute warps run the plan's steps in turn, in lock step,
//     one hardware barrier a step.  A block is spread over G lanes (a 16 x 16
//     block over one warp, over two with several right-hand sides) that read it
//     as 16-byte pieces straight into registers, DEPTH turns of their set ahead.  After the barrier they read
//     the operands of their items (rows of earlier steps, the right-hand side,
//     external rows) from shared memory, multiply, reduce over the lanes that
//     share a block row, and leave the row in shared memory for the next step.
//     What the next step does not wait for (the row's copy in global memory
//     for other CTAs, the blocks and records of the set's next turns) runs
//     while the other set computes;
//   * the stage warp brings the item records and the right-hand side rows into
//     a ring of kSlots steps (both lie in item order, one bulk copy each a
//     step);
//   * the fetch warps take the steps in turn and bring in the rows of other
//     super-tasks: the output vector is pre-filled with a signalling-NaN
//     sentinel and a row is published by its values, so a fetch warp re-reads
//     (bounded) until no word is the sentinel;
//   * the gate warp waits on the ring's mbarriers and joins the step barrier
//     once the step's operands are there: waiting compute warps are parked in
//     the barrier and take no issue slots from the warps that poll (a failed
//     mbarrier test returns at once, so 16 polling warps would).
//
// What bounds it: the number of dependency levels times the time of a step
// (about 0.3 us: barrier, shared-memory operands, multiply-adds and lane
// reduction, one after another), on large systems too: at 64^3 with 8 x 8 blocks
// DRAM is 37 to 44 % busy and the issue slots 20 %, and two stalls of three are
// at the step barrier.  Every block is read once.  One application (two sweeps
// and the preparation), measured against the kernels it takes the place of on
// these patterns (level-ordered polling rows; for 8 x 8 and 16 x 16 blocks chains
// that poll shared memory; sweep_cost.h has the patterns where those stay ahead):
//   ILU0   64^3, 8 x 8           377 -> 300 us (3.2 TB/s)
//   ILU0   48^3, 16 x 16         720 -> 351 us
//   IChol0 300 x 257, 4 x 4     4940 -> 362 us (556 levels, twice)
//   ILU0   40 x 36 x 44, 4 x 4   718 -> 125 us
//   IChol0 64 x 64, 4 x 4        704 ->  85 us
//   IChol0 24 x 20, 2 x 2        273 ->  39 us
// A polling hop cost 4.6 us a level there; here only rows that cross a CTA are
// polled (about 1.3 us each).  Tried and worse: blocks staged in shared memory
// by bulk copies and read back (twice the shared-memory traffic, 0.7 us a
// step), one set of compute warps (0.42 us a step on 2D grids instead of 0.3),
// prefetching the blocks into L2 further ahead (no gain).
#pragma once
#include "per_device.h"
#include "sentinel.cuh"
#include "stage.cuh"
#include "sweep_wave.hpp"

namespace bsp {

template <int BS, typename VT, int R> struct WaveMap : WaveDim<BS, R> {
  using D = WaveDim<BS, R>;
  static constexpr int V = !D::kChunk ? BS : BS == 1 ? 1 : BS < 16 ? 2 : sizeof(VT) == 8 ? 2 : 4;
  static constexpr int CPR = D::kChunk ? BS / V : 1;                                  // lanes per block row
  static constexpr int PR = D::kChunk ? BS * BS / V / (D::G * D::WPI) : 1;            // block rows per lane
  static constexpr int RPP = D::G / CPR;                                              // block rows per pass
  static constexpr int NV = PR * V;                                                   // values per lane and block
  static constexpr int VP = D::kChunk ? V : 1;                                        // values per piece
};

// Stride of a vector row of rw values in item order: whole 16-byte pieces.
__host__ __device__ constexpr int wave_ld_of(int rw) { return (rw + 1) / 2 * 2; }

template <int BS, typename VT, bool HAS_D, int NE, int R> struct WaveCfg {
  using M = WaveMap<BS, VT, R>;
  static constexpr int RW = R * BS;             // values of a vector row
  static constexpr int LD = wave_ld_of(RW);      // its stride in shared memory and in item order
  static constexpr int NB = NE + (HAS_D ? 1 : 0);
  static constexpr int kRegs = NB * M::NV * (int)sizeof(VT) / 4;  // registers of a step's blocks (at least)
  static constexpr int DEPTH = kRegs * 2 <= 36 ? 2 : 1;
  static constexpr int LOOK = 2 * DEPTH;  // steps ahead whose headers and records are staged
  static_assert(LOOK + 2 < kSlots, "headers of the steps read ahead are staged");
  static constexpr int ECAP = wave_ecap<BS, R>();
  static constexpr int kRows = kRing * M::W + 1 + kSlots * (M::W + ECAP);
  static constexpr int OFF_REC = (kRows * LD * 8 + 15) / 16 * 16;
  static constexpr int OFF_HDR = OFF_REC + kSlots * M::W * 16;  // {first item, items} of every staged step
  static constexpr int OFF_BAR = OFF_HDR + kSlots * 8;
  static constexpr int kSmem = OFF_BAR + 3 * kSlots * 8;
  static constexpr int kFetchWarps = M::kFetchWarps;
  static constexpr int kThreads = (2 * kWaveWarps + 2 + kFetchWarps) * 32;
  static_assert(kSmem <= 226 * 1024, "a CTA's vector rows do not fit shared memory");
};

template <typename VT> struct WaveP {
  int n_super;
  const int* super_step;
  const int* super_group;
  const int* group_active;  // null: every group runs
  const int2* step;
  const int4* rec;
  const int* ext_row;
  const VT* vals;
  const double* rhs;  // in item order
  double* x;          // rows of xs values, as the records and ext_row name them
  int xs;
  unsigned spin_limit;
  unsigned* ticket;
  DevStatus* st;
};

// ---- mbarriers and bulk copies
__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait of one thread for a phase; nap: between polls, for waits that
// are not on a step's path.  The copies and arrivals it waits for are always
// made, so running out (seconds) means a broken launch and is reported.
__device__ __forceinline__ void mbar_wait(uint32_t bar, unsigned parity, bool nap, DevStatus* st) {
  for (unsigned i = 0; !mbar_try(bar, parity); ++i) {
    if (i >= kSpinLimit) {
      set_status(st, BSP_TIMEOUT, -1);
      return;
    }
    if (nap || i >= 64) __nanosleep(i < 65536 ? (nap ? 64 : 20) : 1000);
  }
}
// bytes (a multiple of 16) from 16-byte aligned global to shared memory.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, unsigned bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void async_proxy_fence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Barriers of part of the CTA (sync, or arrive without waiting); the warp's
// lanes meet first, as a warp counts once.
template <int NT> __device__ __forceinline__ void named_sync(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory");
}
template <int NT> __device__ __forceinline__ void named_arrive(int id) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(NT) : "memory");
}
__device__ __forceinline__ void st_publish(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
// A piece of V consecutive stored values (V * sizeof(VT) <= 16, aligned to
// that) as it sits in registers: loaded past L1 where the statement stands
// (ahead of its use) straight into the registers it is used from, since a copy
// would wait for the load.
template <typename VT, int V> struct WavePiece;
template <> struct WavePiece<double, 2> {
  double a, b;
  __device__ __forceinline__ void load(const double* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p));
  }
  __device__ __forceinline__ double get(int i) const { return i == 0 ? a : b; }
};
template <> struct WavePiece<double, 1> {
  double a;
  __device__ __forceinline__ void load(const double* p) {
    asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(a) : "l"(p));
  }
  __device__ __forceinline__ double get(int) const { return a; }
};
template <> struct WavePiece<float, 4> {
  float a, b, c, d;
  __device__ __forceinline__ void load(const float* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "l"(p));
  }
  __device__ __forceinline__ double get(int i) const { return i == 0 ? a : i == 1 ? b : i == 2 ? c : d; }
};
template <> struct WavePiece<float, 2> {
  float a, b;
  __device__ __forceinline__ void load(const float* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "l"(p));
  }
  __device__ __forceinline__ double get(int i) const { return i == 0 ? a : b; }
};
template <> struct WavePiece<float, 1> {
  float a;
  __device__ __forceinline__ void load(const float* p) {
    asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(a) : "l"(p));
  }
  __device__ __forceinline__ double get(int) const { return a; }
};
// a BF16 value is the upper half of the FP32 one
template <> struct WavePiece<__nv_bfloat16, 4> {
  unsigned a, b;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "l"(p));
  }
  __device__ __forceinline__ double get(int i) const {
    const unsigned w = i < 2 ? a : b;
    return __uint_as_float(i & 1 ? w & 0xffff0000u : w << 16);
  }
};
template <> struct WavePiece<__nv_bfloat16, 2> {
  unsigned a;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(a) : "l"(p));
  }
  __device__ __forceinline__ double get(int i) const { return __uint_as_float(i ? a & 0xffff0000u : a << 16); }
};
template <> struct WavePiece<__nv_bfloat16, 1> {
  unsigned short a;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(a) : "l"(p));
  }
  __device__ __forceinline__ double get(int) const { return __uint_as_float((unsigned)a << 16); }
};
// V consecutive doubles of shared memory (16-byte aligned when V is even).
template <int V> __device__ __forceinline__ void wave_vec(const double* p, double* a) {
  if constexpr (V % 2 == 0) {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      const double2 t = reinterpret_cast<const double2*>(p)[i];
      a[2 * i] = t.x;
      a[2 * i + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) a[i] = p[i];
  }
}

template <int BS, typename VT, bool HAS_D, int NE, int R>
__global__ void __launch_bounds__(WaveCfg<BS, VT, HAS_D, NE, R>::kThreads, 1) k_wave(const WaveP<VT> p) {
  using M = WaveMap<BS, VT, R>;
  using C = WaveCfg<BS, VT, HAS_D, NE, R>;
  constexpr int RW = C::RW, LD = C::LD, W = M::W, DEPTH = C::DEPTH, NB = C::NB, V = M::V, PR = M::PR, NV = M::NV;
  constexpr int B2 = BS * BS, NCW = 2 * kWaveWarps, LOOK = C::LOOK, kBarThreads = (NCW + 1) * 32;
  extern __shared__ __align__(128) unsigned char wv_smem[];
  __shared__ int s_task;
  double* const vec = reinterpret_cast<double*>(wv_smem);
  const uint32_t bars = smem_addr(wv_smem + C::OFF_BAR);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto full_a = [&](int s) { return bars + 8u * s; };                 // records and right-hand sides
  auto full_b = [&](int s) { return bars + 8u * (kSlots + s); };      // external rows
  auto empty = [&](int s) { return bars + 8u * (2 * kSlots + s); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(full_a(s), 1);
      mbar_init(full_b(s), 1);
      mbar_init(empty(s), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < LD; i += blockDim.x) vec[(size_t)kRing * W * LD + i] = 0.0;  // the zero row
  // an absent item of a step reads through an old record, at first one of zero rows
  for (int i = threadIdx.x; i < kSlots * W; i += blockDim.x)
    reinterpret_cast<int4*>(wv_smem + C::OFF_REC)[i] = make_int4((kRing * W) * 0x10001, (kRing * W) * 0x10001, -1, 0);
  // the records are next written by bulk copies
  async_proxy_fence();
  __syncthreads();
  unsigned par0 = 0;  // phase of every slot at the start of the super-task

  while (true) {
    __syncwarp();  // the roles end in lane-dependent code; barriers want whole warps
    if (threadIdx.x == 0) {
      const unsigned t = atomicAdd(p.ticket, 1u);
      // every CTA takes one ticket past the end: the last one resets it
      if (t == (unsigned)p.n_super + gridDim.x - 1u) atomicExch(p.ticket, 0u);
      s_task = (int)min(t, (unsigned)p.n_super);
    }
    __syncwarp();
    __syncthreads();
    const int task = s_task;
    __syncthreads();
    if (task >= p.n_super) break;
    if (p.group_active && !p.group_active[__ldg(p.super_group + task)]) continue;
    const int t0 = __ldg(p.super_step + task), T = __ldg(p.super_step + task + 1) - t0;
    auto phase = [&](int t) { return ((unsigned)(t / kSlots) ^ (par0 >> (t % kSlots))) & 1u; };

    if (warp < NCW) {
      // ------------------------------------------------------------ compute
      const int set = warp / kWaveWarps, w = warp % kWaveWarps;
      const int k0 = M::WPI == 2 ? w >> 1 : w * M::IPW + lane / M::G;  // the lane's item
      const int gl = lane % M::G;
      const int half = M::WPI == 2 ? w & 1 : 0;
      const int rr = M::kChunk ? half * (BS / 2) + gl / M::CPR : gl;  // first block row of the lane
      const bool has_row = M::kChunk || gl < BS;
      const int r0 = has_row ? rr : BS - 1;
      const int c0 = M::kChunk ? gl % M::CPR * V : 0;
      // the block row and the first right-hand side that a lane ends up with
      // after the reduction, and whether it is the lane that writes them
      constexpr int REST = M::CPR / PR;                   // lanes that share a row once each has one
      constexpr bool SPLIT = R > 1 && REST > 1 && BS < 16;  // the last exchange divides the right-hand sides
      constexpr int RL = SPLIT ? R / 2 : R;
      int fr = r0;
      if constexpr (PR == 4) fr += (gl & (M::CPR / 2) ? 2 * M::RPP : 0) + (gl & (M::CPR / 4) ? M::RPP : 0);
      if constexpr (PR == 2) fr += gl & (M::CPR / 2) ? M::RPP : 0;
      const int fq = (SPLIT && (gl & 1) ? RL * BS : 0) + fr;
      const bool owner = has_row && (gl & (REST - 1) & ~(SPLIT ? 1 : 0)) == 0;
      using Piece = WavePiece<VT, M::VP>;
      constexpr int NP = NV / M::VP;
      Piece blk[DEPTH][NB][NP];
      int cnt[DEPTH];
      const VT* const lane_vals = p.vals + (int64_t)k0 * (M::kItemMajor ? NB * B2 : B2) +
                                  (M::kChunk ? half * (B2 / 2) + gl * V : r0);
      // Every lane reads on every step, an absent item what follows the
      // step's blocks (W items lie past the last one): a conditional load
      // would be merged with the registers' old contents by a copy that waits
      // for it.  Past the end the last step is read again.
      auto read_ahead = [&](int t, Piece (&b)[NB][NP], int& n) {
        const int2 hd = *reinterpret_cast<const int2*>(wv_smem + C::OFF_HDR + min(t, T - 1) % kSlots * 8);
        n = t < T ? hd.y : 0;
        const VT* src = lane_vals;
        if constexpr (M::kItemMajor) src += (int64_t)hd.x * (NB * B2);
        else src += (int64_t)hd.x * NB * B2;
#pragma unroll
        for (int e = 0; e < NB; ++e) {
          const VT* be = src + (M::kItemMajor ? e : e * hd.y) * B2;
#pragma unroll
          for (int q = 0; q < NP; ++q) b[e][q].load(be + q * (M::kChunk ? M::G * V : BS));
        }
      };
      unsigned op[4];  // byte offsets of the lane's operands in the set's next step
      int row;         // the row an item completes, -1: none, -2: no item
      const unsigned c8 = c0 * 8u;
      auto decode = [&](int t, int n) {
        const int4 rc = reinterpret_cast<const int4*>(wv_smem + C::OFF_REC + k0 * 16)[t % kSlots * W];
        op[0] = ((unsigned)rc.x & 0xffffu) * (LD * 8u) + c8;
        op[1] = ((unsigned)rc.x >> 16) * (LD * 8u) + c8;
        op[2] = ((unsigned)rc.y & 0xffffu) * (LD * 8u) + c8;
        op[3] = ((unsigned)rc.y >> 16) * (LD * 8u) + c8;
        row = k0 < n ? rc.z : -2;
      };
      double* const lane_out = vec + k0 * LD + fq;
      named_sync<kBarThreads>(3);  // the first steps' records are there
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) read_ahead(set + 2 * d, blk[d], cnt[d]);
      if (set < T) decode(set, cnt[0]);
      if (set == 1) named_arrive<kBarThreads>(1);
      auto one = [&](int t, Piece (&b)[NB][NP], int& n, const int& n_next) {
        // the earlier steps' rows and this step's staged operands are there
        named_sync<kBarThreads>(1 + set);
        double out[RL];
        double sum[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          double acc[NB][PR];
#pragma unroll
          for (int e = 0; e < NB; ++e) {
            double v[V];
            wave_vec<V>(reinterpret_cast<const double*>(wv_smem + op[HAS_D ? e : e + 1]) + q * BS, v);
#pragma unroll
            for (int i = 0; i < PR; ++i) {
              auto val = [&](int c) { return b[e][(i * V + c) / M::VP].get((i * V + c) % M::VP); };
              double s = val(0) * v[0];
#pragma unroll
              for (int c = 1; c < V; ++c) s = fma(val(c), v[c], s);
              acc[e][i] = s;
            }
          }
          double s[PR];
#pragma unroll
          for (int i = 0; i < PR; ++i) {
            s[i] = acc[0][i] + acc[1][i];
            if constexpr (NB == 3) s[i] += acc[2][i];
            if constexpr (NB == 4) s[i] += acc[2][i] + acc[3][i];
          }
          // sum over the CPR lanes of a block row; a lane with several rows
          // hands half of them over in an exchange until one is left
          int o = M::CPR / 2;
#pragma unroll
          for (int n = PR / 2; n >= 1; n >>= 1, o >>= 1) {
            const bool hi = (gl & o) != 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
              const double give = hi ? s[i] : s[i + n];
              s[i] = (hi ? s[i + n] : s[i]) + __shfl_xor_sync(0xffffffffu, give, o);
            }
          }
#pragma unroll
          for (; o >= (SPLIT ? 2 : 1); o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
          sum[q] = s[0];
        }
#pragma unroll
        for (int q = 0; q < RL; ++q) {
          if constexpr (SPLIT) {
            const bool hi = (gl & 1) != 0;
            const double give = hi ? sum[q] : sum[q + RL];
            out[q] = (hi ? sum[q + RL] : sum[q]) + __shfl_xor_sync(0xffffffffu, give, 1);
          } else {
            out[q] = sum[q];
          }
          if constexpr (!HAS_D) out[q] += reinterpret_cast<const double*>(wv_smem + op[0])[q * BS + fq - c0];
        }
        if (owner && row >= -1) {
          double* xo = lane_out + t % kRing * W * LD;
#pragma unroll
          for (int q = 0; q < RL; ++q) xo[q * BS] = out[q];
        }
        if (t + 1 < T) named_arrive<kBarThreads>(1 + (set ^ 1));
        if (owner && row >= 0) {
          double* xg = p.x + (int64_t)row * p.xs + fq;
#pragma unroll
          for (int q = 0; q < RL; ++q) st_publish(xg + q * BS, out[q]);
        }
        read_ahead(t + 2 * DEPTH, b, n);
        if (t + 2 < T) decode(t + 2, n_next);
      };
      for (int t = set; t < T; t += 2 * DEPTH) {
#pragma unroll
        for (int d = 0; d < DEPTH; ++d)
          if (t + 2 * d < T) one(t + 2 * d, blk[d], cnt[d], cnt[(d + 1) % DEPTH]);
      }
    } else if (warp == NCW) {
      // --------------------------------------------------------------- gate
      if (lane == 0)
        for (int t = 0; t < min(LOOK, T); ++t) mbar_wait(full_a(t % kSlots), phase(t), false, p.st);
      named_sync<kBarThreads>(3);
      for (int t = 0; t < T; ++t) {
        if (lane == 0) {
          const int ta = min(t + LOOK, T - 1);
          mbar_wait(full_a(ta % kSlots), phase(ta), false, p.st);
          mbar_wait(full_b(t % kSlots), phase(t), false, p.st);
        }
        named_sync<kBarThreads>(1 + (t & 1));
        // step t - 1 is over: its slot is free (the last one's after the loop)
        if (t > 0 && lane == 0) mbar_arrive(empty((t - 1) % kSlots));
      }
      if (lane == 0) mbar_arrive(empty((T - 1) % kSlots));
    } else if (warp == NCW + 1) {
      // -------------------------------------------------------------- stage
      // lane l takes steps l, l + 32, ...
      const int* hp = reinterpret_cast<const int*>(p.step + t0);
      auto first = [&](int t) { return __ldg(hp + 2 * min(t, T)); };
      int a = first(lane), b = first(lane + 1);
      for (int tb = 0; tb < T; tb += 32) {
        const int na = first(tb + 32 + lane), nb = first(tb + 33 + lane);
        for (int l = 0; l < 32 && tb + l < T; ++l) {
          if (lane == l) {
            const int t = tb + l, slot = t % kSlots, n = b - a;
            mbar_wait(empty(slot), phase(t) ^ 1u, true, p.st);
            *reinterpret_cast<int2*>(wv_smem + C::OFF_HDR + slot * 8) = make_int2(a, n);
            mbar_expect(full_a(slot), (unsigned)n * (16u + LD * 8u));
            if (n > 0) {
              bulk_copy(smem_addr(wv_smem + C::OFF_REC + slot * W * 16), p.rec + a, (unsigned)n * 16u, full_a(slot));
              bulk_copy(smem_addr(vec + (size_t)(kRing * W + 1 + slot * W) * LD), p.rhs + (int64_t)a * LD,
                        (unsigned)n * (LD * 8u), full_a(slot));
            }
          }
          __syncwarp();
        }
        a = na;
        b = nb;
      }
    } else {
      // -------------------------------------------------------------- fetch
      // the rows of a step are named three turns of this warp ahead
      constexpr int NX = (C::ECAP * RW + 31) / 32;
      constexpr int F = C::kFetchWarps;
      const int* hp = reinterpret_cast<const int*>(p.step + t0) + 1;
      struct Turn {
        int er[NX];    // the rows of its values
        int a, n;      // first external row and their number, of the turn after
      };
      auto head = [&](int t, Turn& u) {
        u.a = __ldg(hp + 2 * min(t, T));
        u.n = __ldg(hp + 2 * min(t + 1, T)) - u.a;
      };
      auto name = [&](Turn& u) {
#pragma unroll
        for (int j = 0; j < NX; ++j) {
          const int e = (lane + 32 * j) / RW;
          u.er[j] = e < u.n ? __ldg(p.ext_row + u.a + e) : -1;
        }
      };
      auto one = [&](int t, Turn& u) {
        const int slot = t % kSlots;
        const double* src[NX];
        bool any = false;
#pragma unroll
        for (int j = 0; j < NX; ++j) {
          src[j] = u.er[j] >= 0 ? p.x + (int64_t)u.er[j] * p.xs + (lane + 32 * j) % RW : nullptr;
          any |= u.er[j] >= 0;
        }
        const int who = u.er[0];
        name(u);
        head(t + 2 * 3 * F, u);
        if (__any_sync(0xffffffffu, any)) {
          double v[NX];
          bool pend = false;
#pragma unroll
          for (int j = 0; j < NX; ++j) v[j] = src[j] ? ld_poll(src[j]) : 0.0;
#pragma unroll
          for (int j = 0; j < NX; ++j) pend |= is_sentinel(v[j]);
          unsigned spins = 0;
          while (pend) {
            if (++spins > p.spin_limit) {
              set_status(p.st, BSP_TIMEOUT, who);
              break;
            }
            if ((spins & 255u) == 0u && *reinterpret_cast<volatile int*>(&p.st->code) != 0) break;
            poll_pause(spins);
            pend = false;
#pragma unroll
            for (int j = 0; j < NX; ++j)
              if (is_sentinel(v[j])) v[j] = ld_poll(src[j]);
#pragma unroll
            for (int j = 0; j < NX; ++j) pend |= is_sentinel(v[j]);
          }
          if (lane == 0) mbar_wait(empty(slot), phase(t) ^ 1u, true, p.st);
          __syncwarp();
          double* ex = vec + (size_t)(kRing * W + 1 + kSlots * W + slot * C::ECAP) * LD;
#pragma unroll
          for (int j = 0; j < NX; ++j)
            if (src[j]) ex[(lane + 32 * j) / RW * LD + (lane + 32 * j) % RW] = v[j];
        } else if (lane == 0) {
          mbar_wait(empty(slot), phase(t) ^ 1u, true, p.st);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(full_b(slot));
      };
      const int f = warp - NCW - 2;
      Turn u0, u1, u2;
      head(f, u0);
      head(f + F, u1);
      head(f + 2 * F, u2);
      name(u0);
      name(u1);
      name(u2);
      head(f + 3 * F, u0);
      head(f + 4 * F, u1);
      head(f + 5 * F, u2);
      for (int t = f; t < T; t += 3 * F) {
        one(t, u0);
        if (t + F < T) one(t + F, u1);
        if (t + 2 * F < T) one(t + 2 * F, u2);
      }
    }
    // a slot was used T / kSlots times, the first T % kSlots once more
    par0 ^= ((T / kSlots) & 1 ? (1u << kSlots) - 1u : 0u) ^ ((1u << (T % kSlots)) - 1u);
  }
}

// The arrays of a sweep as the kernel takes them (vectors and ticket aside).
template <typename VT> WaveP<VT> wave_params(bsp_handle_s* h, const WaveSym& S, const WaveVals& V) {
  WaveP<VT> p{};
  p.n_super = S.n_super;
  p.super_step = S.super_step.get();
  p.super_group = S.super_group.get();
  p.step = S.step.get();
  p.rec = S.rec.get();
  p.ext_row = S.ext_row.get();
  p.vals = reinterpret_cast<const VT*>(V.vals.get());
  p.spin_limit = h->spin_limit;
  p.st = h->ws.status.get();
  return p;
}

template <int BS, typename VT, bool HAS_D, int NE, int R>
int wave_launch(bsp_handle_s* h, const WaveP<VT>& p, cudaStream_t stream) {
  using C = WaveCfg<BS, VT, HAS_D, NE, R>;
  static PerDevice ready;
  auto kern = k_wave<BS, VT, HAS_D, NE, R>;
  if (!ready.has(h->device)) {
    BSP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
    ready.set(h->device);
  }
  const int grid = p.n_super < h->num_sms ? (p.n_super < 1 ? 1 : p.n_super) : h->num_sms;
  kern<<<grid, C::kThreads, C::kSmem, stream>>>(p);
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

}  // namespace bsp
