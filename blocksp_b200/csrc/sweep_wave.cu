// sweep_wave.cu — building, filling and launching the lock-step sweeps.
//
// Reference: blocksp_preconditioners.hpp:294-349 (ILU0::invmul: unit-L
// forward substitution, then backward substitution with D_Inv[i] = U_ii^-1)
// and :432-489 (IChol0::invmul: L forward with L_ii^-1, then L^T backward
// through the column structure of L with L_ii^-T).  Natural order is kept.
#include "sweep_wave.cuh"

namespace bsp {

int grid_for(const bsp_handle_s* h, int64_t n, int threads);

// ------------------------------------------------------------------ values
// Stored block b: minus w times factor block blk_src[b] (transposed when
// trans), or what the negative codes of wave_plan.h say.
template <typename VT> __device__ __forceinline__ void store_as(VT* p, double v) {
  if constexpr (sizeof(VT) == 8) *p = v;
  else if constexpr (sizeof(VT) == 4) *p = (float)v;
  else *p = __float2bfloat16_rn((float)v);
}
template <int BS, typename VT>
__global__ void k_wave_gather(int64_t nblk, const int64_t* __restrict__ blk_src, const double* __restrict__ src,
                              int trans, double w, VT* __restrict__ dst) {
  constexpr int B2 = BS * BS;
  const int64_t total = nblk * B2;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / B2;
    const int k = (int)(t - b * B2);
    const int a = WaveDim<BS>::kChunk ? k / BS : k % BS, c = WaveDim<BS>::kChunk ? k % BS : k / BS;
    const int64_t sb = blk_src[b];
    double v = 0.0;
    if (sb >= 0) v = -w * (trans ? src[sb * B2 + c * BS + a] : src[sb * B2 + a * BS + c]);
    else if (sb == kWaveOne) v = a == c ? 1.0 : 0.0;
    store_as(dst + t, v);
  }
}

// The same with the block premultiplied by its row's D.  Every value takes BS
// products, so a CTA brings UB groups of NB blocks and their D to shared memory
// first (rows one value further apart than they are long: both orders are read
// without conflicts), each block read from memory once and in order: 484 us
// for the backward sweep of the 64^3 grid of 8 x 8 blocks, 424 for 44 x 40 x 36
// of 16 x 16 kept in FP32 (a thread a value that read D and the block itself
// took 555 and 986).
constexpr int kGatherThreads = 256;
template <int BS, typename VT>
__global__ void __launch_bounds__(kGatherThreads)
k_wave_gather_d(int64_t nblk, const int64_t* __restrict__ blk_src, const int* __restrict__ blk_row,
                const double* __restrict__ src, const double* __restrict__ dinv, int trans, int trans_d, double w,
                VT* __restrict__ dst) {
  constexpr int B2 = BS * BS, NB = kGatherThreads / B2, UB = 4, LD = BS + 1;
  static_assert(NB >= 1, "a block per group of threads");
  __shared__ double sB[UB][NB][BS * LD], sD[UB][NB][BS * LD];
  const int nb = threadIdx.x / B2, k = threadIdx.x % B2;
  const int kr = k / BS, kc = k % BS;  // this thread's value of the blocks it loads
  const int a = WaveDim<BS>::kChunk ? kr : kc, c = WaveDim<BS>::kChunk ? kc : kr;  // and of those it stores
  const int da = trans_d ? 1 : LD, dm = trans_d ? LD : 1, bm = trans ? 1 : LD, bc = trans ? LD : 1;
  for (int64_t b0 = (int64_t)blockIdx.x * (UB * NB); b0 < nblk; b0 += (int64_t)gridDim.x * (UB * NB)) {
    int64_t sb[UB];
    double vb[UB], vd[UB];
#pragma unroll
    for (int u = 0; u < UB; ++u) {
      const int64_t b = b0 + u * NB + nb;
      sb[u] = kWaveZero;
      vb[u] = vd[u] = 0.0;
      if (nb < NB && b < nblk) {
        sb[u] = __ldg(blk_src + b);
        if (sb[u] >= 0) vb[u] = __ldcs(src + sb[u] * B2 + k);
        if (sb[u] >= 0 || sb[u] == kWaveD) vd[u] = __ldg(dinv + (int64_t)__ldg(blk_row + b) * B2 + k);
      }
    }
    if (nb < NB)
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        sB[u][nb][kr * LD + kc] = vb[u];
        sD[u][nb][kr * LD + kc] = vd[u];
      }
    __syncthreads();
    if (nb < NB)
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int64_t b = b0 + u * NB + nb;
        if (b >= nblk) continue;
        double v = 0.0;
        if (sb[u] >= 0) {
#pragma unroll
          for (int m = 0; m < BS; ++m) v = fma(sD[u][nb][a * da + m * dm], sB[u][nb][m * bm + c * bc], v);
          v = -w * v;
        } else if (sb[u] == kWaveD) {
          v = sD[u][nb][a * da + c * dm];
        } else if (sb[u] == kWaveOne) {
          v = a == c ? 1.0 : 0.0;
        }
        store_as(dst + b * B2 + k, v);
      }
    __syncthreads();
  }
}

template <int BS, typename VT>
static int gather_t(bsp_handle_s* h, const WaveSym& S, const double* fvals, const double* dinv, bool premul, double w,
                    WaveVals& out) {
  VT* dst = reinterpret_cast<VT*>(out.vals.get());
  count_launch();
  if (S.has_d || premul) {
    const int g = grid_for(h, ceil_div(S.n_blk, 4 * (kGatherThreads / (BS * BS))) * kGatherThreads, kGatherThreads);
    k_wave_gather_d<BS, VT><<<g, kGatherThreads, 0, h->stream>>>(S.n_blk, S.blk_src.get(), S.blk_row.get(), fvals, dinv,
                                                                 S.trans_blocks, S.trans_d, w, dst);
  } else {
    const int g = grid_for(h, S.n_blk * BS * BS, 256);
    k_wave_gather<BS, VT><<<g, 256, 0, h->stream>>>(S.n_blk, S.blk_src.get(), fvals, S.trans_blocks, w, dst);
  }
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

static size_t prec_bytes(int prec) { return prec == BSP_PREC_F64 ? 8 : prec == BSP_PREC_F32 ? 4 : 2; }
size_t wave_val_bytes(const WaveSym& S, int prec) {
  // W items past the last one are read (and dropped)
  return (size_t)(S.n_blk + (int64_t)wave_shape(S.bs, 1).W * (S.ne + 1)) * S.bs * S.bs * prec_bytes(prec);
}

int wave_gather(bsp_handle_s* h, const WaveSym& S, int prec, const double* fvals, const double* dinv, WaveVals& out,
                bool premul, double w) {
  const size_t vb = wave_val_bytes(S, prec);
  if (out.vals.n < vb) BSP_TRY(out.vals.alloc(vb));
  if (S.n_blk > 0) {
    int st = BSP_INVALID;
    switch (S.bs) {
#define BSP_WAVE_CASE(B)                                                                      \
  case B:                                                                                     \
    st = prec == BSP_PREC_F64   ? gather_t<B, double>(h, S, fvals, dinv, premul, w, out)                 \
         : prec == BSP_PREC_F32 ? gather_t<B, float>(h, S, fvals, dinv, premul, w, out)                  \
                                : gather_t<B, __nv_bfloat16>(h, S, fvals, dinv, premul, w, out);         \
    break;
      BSP_WAVE_SIZES(BSP_WAVE_CASE)
#undef BSP_WAVE_CASE
      default: break;
    }
    BSP_TRY(st);
  }
  out.valid = true;
  return BSP_OK;
}

// ------------------------------------------------------------------ SOR
// One thread per value of x: the row's product with the old iterate (its
// threads read a block row each), then the inverted diagonal times the CTA's
// residuals in shared memory.  A pass over A at most; 40 x 36 x 44 rows of 4 x 4
// blocks (60 MB, cached in L2): 12 us beside a sweep of 60 us.
constexpr int kSorThreads = 256;
template <int BS, typename VT>
__global__ void __launch_bounds__(kSorThreads)
k_sor_prepare(int n, int forward, const int* __restrict__ row_ptr, const int* __restrict__ col,
              const VT* __restrict__ avals, const VT* __restrict__ dinv, double w, const int* __restrict__ item_of,
              const double* b, const double* __restrict__ xold, double* __restrict__ rp, double* x) {
  constexpr int RPC = kSorThreads / BS, LD = wave_ld_of(BS);
  __shared__ double res[RPC][BS];
  auto val = [](VT v) -> double {
    if constexpr (sizeof(VT) == 2) return (double)__bfloat162float(v);
    else return (double)v;
  };
  const int lr = threadIdx.x / BS, r = threadIdx.x % BS;
  const int i = blockIdx.x * RPC + lr;
  const bool on = lr < RPC && i < n;
  const int64_t k = (int64_t)i * BS + r;
  double old = 0.0;
  if (on) {
    double t = b[k];
    if (xold) {
      old = xold[k];
      for (int e = __ldg(row_ptr + i); e < __ldg(row_ptr + i + 1); ++e) {
        const int j = __ldg(col + e);
        if (forward ? j <= i : j >= i) continue;
        const VT* a = avals + (int64_t)e * (BS * BS) + r * BS;
        const double* xj = xold + (int64_t)j * BS;
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < BS; ++c) s = fma(val(a[c]), xj[c], s);
        t -= s;
      }
    }
    res[lr][r] = t;
  }
  __syncthreads();
  if (on) {
    const VT* d = dinv + (int64_t)i * (BS * BS) + r * BS;
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < BS; ++c) s = fma(val(d[c]), res[lr][c], s);
    rp[(int64_t)__ldg(item_of + i) * LD + r] = old + (-w * old + w * s);
    reinterpret_cast<unsigned long long*>(x)[k] = kSentinel64;
  }
}

int wave_sor_prepare(bsp_handle_s* h, const WaveSym& S, int prec, bool forward, const int* row_ptr, const int* col,
                     const void* avals, const void* dinv, double w, const double* b, const double* xold, double* rp,
                     double* x) {
  auto run = [&](auto bs, auto v) -> int {
    constexpr int BS = decltype(bs)::value;
    using VT = decltype(v);
    const int grid = (int)ceil_div(S.n, kSorThreads / BS);
    count_launch();
    k_sor_prepare<BS, VT><<<grid, kSorThreads, 0, h->stream>>>(
        S.n, forward ? 1 : 0, row_ptr, col, static_cast<const VT*>(avals), static_cast<const VT*>(dinv), w,
        S.item_of.get(), b, xold, rp, x);
    return BSP_OK;
  };
  int st = BSP_INVALID;
  switch (S.bs) {
#define BSP_WAVE_CASE(B)                                                               \
  case B:                                                                              \
    st = prec == BSP_PREC_F64   ? run(std::integral_constant<int, B>{}, double{})      \
         : prec == BSP_PREC_F32 ? run(std::integral_constant<int, B>{}, float{})       \
                                : run(std::integral_constant<int, B>{}, __nv_bfloat16{}); \
    break;
    BSP_WAVE_SIZES(BSP_WAVE_CASE)
#undef BSP_WAVE_CASE
    default: break;
  }
  BSP_TRY(st);
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

// ------------------------------------------------------------------ build
template <typename T, typename H> static int upload_as(DevBuf<T>& d, const std::vector<H>& v) {
  static_assert(sizeof(T) == sizeof(H), "same layout on host and device");
  BSP_TRY(d.alloc(v.empty() ? 1 : v.size()));
  if (!v.empty()) BSP_CUDA_TRY(cudaMemcpy(d.get(), v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
  return BSP_OK;
}

int wave_upload(WavePlan&& P, int bs, bool trans_blocks, bool has_d, bool trans_d, const std::vector<int>* row_item,
                std::vector<int>* item_of, WaveSym& S) {
  const int n = P.n;
  std::vector<int> items(n, 0);
  for (size_t i = 0; i < P.item_row.size(); ++i)
    if (P.item_row[i] >= 0) items[P.item_row[i]] = (int)i;
  BSP_TRY(upload_as(S.item_of, items));
  if (row_item) {
    for (auto& r : P.rec)
      if (r.row >= 0) r.row = (*row_item)[r.row];
    for (int& r : P.ext_row) r = (*row_item)[r];
  }
  S.n = n;
  S.bs = bs;
  S.n_item = (int64_t)P.rec.size();
  S.to_items = row_item != nullptr;
  S.n_super = P.n_super;
  S.n_levels = P.n_levels;
  S.ne = P.ne;
  S.n_blk = (int64_t)P.blk_src.size();
  S.trans_blocks = trans_blocks;
  S.has_d = has_d;
  S.trans_d = trans_d;
  BSP_TRY(upload_as(S.super_step, P.super_step));
  BSP_TRY(upload_as(S.super_group, P.super_group));
  BSP_TRY(upload_as(S.step, P.step));
  BSP_TRY(upload_as(S.rec, P.rec));
  BSP_TRY(upload_as(S.item_row, P.item_row));
  BSP_TRY(upload_as(S.ext_row, P.ext_row));
  BSP_TRY(upload_as(S.blk_src, P.blk_src));
  BSP_TRY(upload_as(S.blk_row, P.blk_row));
  if (item_of) *item_of = std::move(items);
  return BSP_OK;
}

// ------------------------------------------------------------------ sweep
size_t wave_item_values(const WaveSym& S, int nrhs) {
  return (size_t)std::max<int64_t>(S.n_item, 1) * wave_ld_of(nrhs * S.bs);
}

// rp = r in item order and z's sentinel (a row is read and replaced by the same
// thread, so z may alias r); w's sentinel.
template <int BS>
__global__ void k_wave_prepare(int64_t n_item, const int* __restrict__ item_row, const double* r, double* rp,
                               double* z, int64_t n_w, unsigned long long* __restrict__ w) {
  constexpr int LD = wave_ld_of(BS);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t t = t0; t < n_item * BS; t += stride) {
    const int64_t i = t / BS;
    const int c = (int)(t - i * BS), row = __ldg(item_row + i);
    if (row >= 0) {
      const int64_t k = (int64_t)row * BS + c;
      rp[i * LD + c] = r[k];
      reinterpret_cast<unsigned long long*>(z)[k] = kSentinel64;
    }
  }
  for (int64_t t = t0; t < n_w; t += stride) w[t] = kSentinel64;
}

int wave_prepare(bsp_handle_s* h, const WaveSym& lo, const WaveSym& up, const double* r, double* rp, double* w,
                 double* z) {
  const int64_t nw = (int64_t)wave_item_values(up, 1);
  const int g = grid_for(h, std::max(lo.n_item * lo.bs, nw), 256);
  auto* ws = reinterpret_cast<unsigned long long*>(w);
  count_launch();
  switch (lo.bs) {
#define BSP_WAVE_CASE(B)                                                                          \
  case B:                                                                                         \
    k_wave_prepare<B><<<g, 256, 0, h->stream>>>(lo.n_item, lo.item_row.get(), r, rp, z, nw, ws);  \
    break;
    BSP_WAVE_SIZES(BSP_WAVE_CASE)
#undef BSP_WAVE_CASE
    default: return BSP_INVALID;
  }
  BSP_CUDA_TRY(cudaPeekAtLastError());
  return BSP_OK;
}

template <int BS, typename VT>
static int sweep_t(bsp_handle_s* h, const WaveSym& S, const WaveP<VT>& p) {
  count_launch();
  if (S.ne == 2)
    return S.has_d ? wave_launch<BS, VT, true, 2, 1>(h, p, h->stream) : wave_launch<BS, VT, false, 2, 1>(h, p, h->stream);
  return S.has_d ? wave_launch<BS, VT, true, 3, 1>(h, p, h->stream) : wave_launch<BS, VT, false, 3, 1>(h, p, h->stream);
}

template <typename VT>
static int sweep_typed(bsp_handle_s* h, const WaveSym& S, const WaveVals& V, const double* rhs, double* x,
                       unsigned* ticket) {
  WaveP<VT> p = wave_params<VT>(h, S, V);
  p.rhs = rhs;
  p.x = x;
  p.xs = S.to_items ? wave_ld_of(S.bs) : S.bs;
  p.ticket = ticket;
  switch (S.bs) {
#define BSP_WAVE_CASE(B) \
  case B: return sweep_t<B, VT>(h, S, p);
    BSP_WAVE_SIZES(BSP_WAVE_CASE)
#undef BSP_WAVE_CASE
    default: break;
  }
  record_error("triangular sweep: unsupported block size");
  return BSP_INVALID;
}

int wave_sweep(bsp_handle_s* h, const WaveSym& S, int prec, const WaveVals& V, const double* rhs, double* x,
               unsigned* ticket) {
  if (!V.valid) {
    record_error("triangular sweep: values not gathered");
    return BSP_INVALID;
  }
  if (S.n_super == 0) return BSP_OK;
  if (prec == BSP_PREC_F64) return sweep_typed<double>(h, S, V, rhs, x, ticket);
  if (prec == BSP_PREC_F32) return sweep_typed<float>(h, S, V, rhs, x, ticket);
  return sweep_typed<__nv_bfloat16>(h, S, V, rhs, x, ticket);
}

}  // namespace bsp
