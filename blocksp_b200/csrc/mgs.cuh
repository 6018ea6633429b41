// mgs.cuh — modified Gram-Schmidt of one Arnoldi column in one launch.
//
// one_arnoldi (blocksp_solvers.hpp:109-136):
//   for i = 0..j: H(i, j) = <q_i, v>;  v -= H(i, j) q_i
//   H(j+1, j) = ||v||;  q_{j+1} = v / H(j+1, j) (unless below zero_thresh)
// One CTA per SM, all co-resident (cooperative launch).  Each CTA keeps its
// slice of v in registers for the whole column.  The basis vectors are taken B
// at a time: their slices sit in shared memory together, the products <q_i, v>
// of all of them and <q_k, q_i> (i < k) among them are summed over the grid in
// one step, and the coefficients follow as modified Gram-Schmidt gives them,
//   h_k = <q_k, v> - sum_{i<k} <q_k, q_i> h_i
// (the triangular form of the same recurrence: h_k is the product with v after
// the updates by q_i, i < k), before v takes the B updates in order.  In exact
// arithmetic that is modified Gram-Schmidt; in rounding h_k carries eps ||v|| of
// the block's start where that carries eps ||v|| after the updates before it, up
// to B vectors at a time.  Both lose orthogonality like eps times the condition
// of the columns, and histories of nearly dependent columns are off 80-bit
// arithmetic by as much as plain modified Gram-Schmidt is.  So a
// column costs a grid barrier per B vectors instead of one per vector, and every
// basis vector is still read once.  Steps are separated by a bounded grid
// barrier; every CTA sums the per-CTA partials in index order, so H is
// bit-reproducible.
//
// What bounds it: HBM (one read of the basis) and, for short vectors, the
// barriers (about 4 us each with the sums).  B is what shared memory holds of a
// slice, at most 7 (5 complex ones): the sums of a step then fit one value per
// lane.
#pragma once
#include "per_device.h"
#include "reduce.cuh"
#include "sentinel.cuh"
#include "stage.cuh"

namespace bsp {

struct MgsP {
  int64_t len;             // doubles
  int64_t slice;           // doubles per CTA
  const double* v;         // M^-1 A q_j
  double* const* Q;        // basis table
  int j;                   // column
  double* h;               // h[i * hs] = H(i, j) (complex: h[i * hs], h[i * hs + 1]); the norm at i = j + 1
  int64_t hs;
  const double* zero_thresh;
  double* partials;        // kMgsSums x gridDim.x
  unsigned* bar;           // barrier counter (0 at launch)
  unsigned spin_limit;
  DevStatus* st;
};
constexpr int kMgsSums = 32;  // sums of a step
constexpr int kMgsSmem = 227 * 1024 - 2048;

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier number `gen` (1, 2, ...): bounded spin, BSP_TIMEOUT on expiry.
__device__ __forceinline__ void mgs_barrier(const MgsP& p, unsigned gen) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(p.bar, 1u);
    const unsigned target = gen * gridDim.x;
    unsigned spins = 0;
    while (ld_acquire_u32(p.bar) < target) {
      if (++spins > p.spin_limit) {
        set_status(p.st, BSP_TIMEOUT, -1);
        break;
      }
      poll_pause(spins);
    }
    __threadfence();
  }
  __syncthreads();
}

// Asks L2 to fetch n doubles at src (a hint: nothing is written; a range
// that is not 16-byte aligned is skipped).  Called by warp 0 of the CTA:
// lane k issues the k-th 16 KB piece.
__device__ __forceinline__ void prefetch_l2(const double* src, int64_t n) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(src);
  if (n <= 0 || (a & 15u)) return;
  const int64_t bytes = (n * 8) & ~int64_t(15);
  constexpr int64_t kPiece = 16384;
  for (int64_t o = (int64_t)(threadIdx.x & 31) * kPiece; o < bytes; o += 32 * kPiece) {
    const unsigned sz = (unsigned)(bytes - o < kPiece ? bytes - o : kPiece);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a + o), "r"(sz) : "memory");
  }
}

// Sums of NP (a power of two) values over the warp: halved between lane pairs
// until one is left, so lane l ends with the sum of value l % NP.
template <int NP> __device__ __forceinline__ double warp_sums(double (&s)[NP]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = NP / 2; n >= 1; n >>= 1)
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const bool hi = (lane & n) != 0;
      const double give = hi ? s[k] : s[k + n];
      s[k] = (hi ? s[k + n] : s[k]) + __shfl_xor_sync(0xffffffffu, give, n);
    }
#pragma unroll
  for (int o = NP; o < 32; o <<= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
  return s[0];
}

// Sums of the values over the grid, in CTA order (the same in every CTA): tot[k].
template <int TH, int NP>
__device__ __forceinline__ void grid_sums(const MgsP& p, double (&s)[NP], unsigned gen, double* red, double* tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = TH / 32;
  const double a = warp_sums<NP>(s);
  if (lane < NP) red[warp * NP + lane] = a;
  __syncthreads();
  double* part = p.partials + (size_t)(gen & 1u) * kMgsSums * gridDim.x;
  if (threadIdx.x < NP) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) t += red[w * NP + threadIdx.x];
    __stcg(part + (size_t)threadIdx.x * gridDim.x + blockIdx.x, t);
  }
  mgs_barrier(p, gen);
  for (int k = warp; k < NP; k += NW) {
    double t = 0.0;
    for (int c = lane; c < (int)gridDim.x; c += 32) t += __ldcg(part + (size_t)k * gridDim.x + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) tot[k] = t;
  }
  __syncthreads();
}

// TH (512: more registers a thread) threads of NPT values each; U: values moved at once (2 when the vectors
// are 16-byte aligned); CX: pairs (re, im), <x, y> = sum conj(x) y.
template <int TH, int NPT, int B, int U, bool CX>
__global__ void __launch_bounds__(TH, 1) k_mgs(const MgsP p) {
  static_assert(NPT % U == 0 && (!CX || U == 2), "whole pieces");
  constexpr int NS = (B + B * (B - 1) / 2) * (CX ? 2 : 1);
  constexpr int NP = NS <= 1 ? 1 : NS <= 2 ? 2 : NS <= 4 ? 4 : NS <= 8 ? 8 : NS <= 16 ? 16 : 32;
  static_assert(NS <= kMgsSums, "one value per lane");
  constexpr int SL = TH * NPT;  // doubles of a slice in shared memory
  extern __shared__ __align__(16) double qs[];  // B slices
  __shared__ double red[(TH / 32) * NP], tot[NP < 2 ? 2 : NP];
  const int t = threadIdx.x;
  const int64_t beg = (int64_t)blockIdx.x * p.slice;
  const int64_t left = p.len - beg;
  const int nloc = (int)(left < p.slice ? (left < 0 ? 0 : left) : p.slice);
  const int nv = p.j + 1;  // basis vectors
  if (t < 32)
    for (int i = 0; i < min(B, nv); ++i) prefetch_l2(p.Q[i] + beg, nloc);
  double v[NPT];
#pragma unroll
  for (int k = 0; k < NPT / U; ++k) {
    const int o = (t + k * TH) * U;
    if constexpr (U == 2) {
      const double2 x = o < nloc ? *reinterpret_cast<const double2*>(p.v + beg + o) : make_double2(0.0, 0.0);
      v[2 * k] = x.x;
      v[2 * k + 1] = x.y;
    } else {
      v[k] = o < nloc ? p.v[beg + o] : 0.0;
    }
  }
  unsigned gen = 0;
  for (int i0 = 0; i0 < nv; i0 += B) {
    const int nb = min(B, nv - i0);
    // the slices of this block of vectors (each thread copies and reads only
    // its own entries), one batch of copies in flight at once
    for (int i = 0; i < nb; ++i) {
      const double* qb = p.Q[i0 + i] + beg;
#pragma unroll
      for (int k = 0; k < NPT / U; ++k) {
        const int o = (t + k * TH) * U;
        if (o < nloc) cp_async_small<8 * U>(qs + i * SL + o, qb + o);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    // the next block's slices stream into L2 while the grid meets
    if (t < 32)
      for (int i = i0 + B; i < min(i0 + 2 * B, nv); ++i) prefetch_l2(p.Q[i] + beg, nloc);
    double s[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) s[k] = 0.0;
#pragma unroll
    for (int k = 0; k < NPT / U; ++k) {
      const int o = (t + k * TH) * U;
      if (o >= nloc) continue;
      double q[B][U];
#pragma unroll
      for (int i = 0; i < B; ++i) {
        if constexpr (U == 2) {
          const double2 x = i < nb ? *reinterpret_cast<const double2*>(qs + i * SL + o) : make_double2(0.0, 0.0);
          q[i][0] = x.x;
          q[i][1] = x.y;
        } else {
          q[i][0] = i < nb ? qs[i * SL + o] : 0.0;
        }
      }
      // value (a, b): <q_a, v> (b = B), then <q_a, q_b>, b < a
      auto add = [&](int idx, const double (&x)[U], const double* y) {
        if constexpr (CX) {
          s[2 * idx] = fma(x[0], y[0], fma(x[1], y[1], s[2 * idx]));
          s[2 * idx + 1] = fma(x[0], y[1], fma(-x[1], y[0], s[2 * idx + 1]));
        } else {
#pragma unroll
          for (int u = 0; u < U; ++u) s[idx] = fma(x[u], y[u], s[idx]);
        }
      };
#pragma unroll
      for (int a = 0; a < B; ++a) add(a, q[a], v + k * U);
#pragma unroll
      for (int a = 1; a < B; ++a)
#pragma unroll
        for (int b = 0; b < a; ++b) add(B + a * (a - 1) / 2 + b, q[a], q[b]);
    }
    grid_sums<TH, NP>(p, s, ++gen, red, tot);
    constexpr int CW = CX ? 2 : 1;
    double h[B][CW];
#pragma unroll
    for (int a = 0; a < B; ++a) {
#pragma unroll
      for (int c = 0; c < CW; ++c) h[a][c] = tot[CW * a + c];
#pragma unroll
      for (int b = 0; b < a; ++b) {
        const double* g = tot + CW * (B + a * (a - 1) / 2 + b);
        if constexpr (CX) {
          h[a][0] = fma(-g[0], h[b][0], fma(g[1], h[b][1], h[a][0]));
          h[a][1] = fma(-g[0], h[b][1], fma(-g[1], h[b][0], h[a][1]));
        } else {
          h[a][0] = fma(-g[0], h[b][0], h[a][0]);
        }
      }
    }
    if (blockIdx.x == 0 && t == 0)
#pragma unroll
      for (int a = 0; a < B; ++a)
        if (a < nb)
#pragma unroll
          for (int c = 0; c < CW; ++c) p.h[(int64_t)(i0 + a) * p.hs + c] = h[a][c];
#pragma unroll
    for (int k = 0; k < NPT / U; ++k) {
      const int o = (t + k * TH) * U;
      if (o >= nloc) continue;
#pragma unroll
      for (int a = 0; a < B; ++a) {
        if (a >= nb) continue;
        if constexpr (CX) {
          const double2 x = *reinterpret_cast<const double2*>(qs + a * SL + o);
          v[2 * k] = fma(-h[a][0], x.x, fma(h[a][1], x.y, v[2 * k]));
          v[2 * k + 1] = fma(-h[a][0], x.y, fma(-h[a][1], x.x, v[2 * k + 1]));
        } else if constexpr (U == 2) {
          const double2 x = *reinterpret_cast<const double2*>(qs + a * SL + o);
          v[2 * k] = fma(-h[a][0], x.x, v[2 * k]);
          v[2 * k + 1] = fma(-h[a][0], x.y, v[2 * k + 1]);
        } else {
          v[k] = fma(-h[a][0], qs[a * SL + o], v[k]);
        }
      }
    }
  }
  double nn[1] = {0.0};
#pragma unroll
  for (int k = 0; k < NPT; ++k) nn[0] = fma(v[k], v[k], nn[0]);
  grid_sums<TH, 1>(p, nn, ++gen, red, tot);
  const double nrm = sqrt(fabs(tot[0]));
  if (blockIdx.x == 0 && t == 0) p.h[(int64_t)nv * p.hs] = nrm;
  if (fabs(nrm) < *p.zero_thresh) return;  // breakdown: the basis is not extended
  double* qn = p.Q[nv] + beg;
#pragma unroll
  for (int k = 0; k < NPT / U; ++k) {
    const int o = (t + k * TH) * U;
    if (o >= nloc) continue;
    if constexpr (U == 2) *reinterpret_cast<double2*>(qn + o) = make_double2(v[2 * k] / nrm, v[2 * k + 1] / nrm);
    else qn[o] = v[k] / nrm;
  }
}

// ------------------------------------------------------------------ host
template <int TH, int NPT, int B, int U, bool CX> int launch_mgs_t(bsp_handle_s* h, MgsP& p) {
  constexpr size_t smem = (size_t)B * TH * NPT * sizeof(double);
  static_assert(smem <= kMgsSmem, "the slices of a block of vectors do not fit shared memory");
  static PerDevice ready;
  auto kern = k_mgs<TH, NPT, B, U, CX>;
  if (!ready.has(h->device)) {
    BSP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    BSP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TH, smem));
    if (per_sm < 1) return 1;
    ready.set(h->device);
  }
  p.slice = (int64_t)TH * NPT;
  void* args[] = {&p};
  count_launch();
  BSP_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, h->num_sms, TH, args, smem, h->stream));
  return BSP_OK;
}

// The column's launch when v's slices fit one CTA per SM, else returns 1.  The
// vectors of a block grow fewer as slices grow (on 148 SMs, real: 7 up to
// 303,000 values, 6 up to 606,000, 4 up to 909,000, 3 up to 1.2 million, 2 up to
// 2.1 million, 1 up to 3.6 million).
template <int U, bool CX> int launch_mgs_u(bsp_handle_s* h, MgsP& p) {
  const int64_t per_thread = (p.len + (int64_t)h->num_sms * 512 - 1) / ((int64_t)h->num_sms * 512);
  if (per_thread <= 4) return launch_mgs_t<512, 4, CX ? 5 : 7, U, CX>(h, p);
  if (per_thread <= 8) return launch_mgs_t<512, 8, CX ? 5 : 6, U, CX>(h, p);
  if (per_thread <= 12) return launch_mgs_t<512, 12, 4, U, CX>(h, p);
  if (per_thread <= 16) return launch_mgs_t<512, 16, 3, U, CX>(h, p);
  if (per_thread <= 28) return launch_mgs_t<512, 28, 2, U, CX>(h, p);
  if (per_thread <= 48) return launch_mgs_t<512, 48, 1, U, CX>(h, p);
  return 1;
}

// partials: 2 * kMgsSums * num_sms values.  v and, when len is even, every basis
// vector start on 16 bytes.  hcol, hs, zero_thresh: see MgsP.
template <bool CX>
int launch_mgs(bsp_handle_s* h, int64_t len, const double* v, double* const* Q, int j, double* hcol, int64_t hs,
               const double* zero_thresh, double* partials, unsigned* bar) {
  MgsP p{};
  p.len = len;
  p.v = v;
  p.Q = Q;
  p.j = j;
  p.h = hcol;
  p.hs = hs;
  p.zero_thresh = zero_thresh;
  p.partials = partials;
  p.bar = bar;
  p.spin_limit = h->spin_limit;
  p.st = h->ws.status.get();
  BSP_CUDA_TRY(cudaMemsetAsync(bar, 0, sizeof(unsigned), h->stream));
  if constexpr (CX) return launch_mgs_u<2, true>(h, p);
  else return len % 2 == 0 ? launch_mgs_u<2, false>(h, p) : launch_mgs_u<1, false>(h, p);
}

}  // namespace bsp
