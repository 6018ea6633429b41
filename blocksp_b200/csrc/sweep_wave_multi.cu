// sweep_wave_multi.cu — the lock-step sweeps with several right-hand sides per
// row (the batched solver): every block is read once for all of them.
#include "sweep_wave.cuh"

namespace bsp {

template <int BS, int R>
static int multi_t(bsp_handle_s* h, const WaveSym& S, const WaveP<double>& p, cudaStream_t s) {
  return S.ne == 2 ? wave_launch<BS, double, true, 2, R>(h, p, s) : wave_launch<BS, double, true, 3, R>(h, p, s);
}
template <int BS>
static int multi_r(bsp_handle_s* h, const WaveSym& S, const WaveP<double>& p, int nrhs, cudaStream_t s) {
  return nrhs == 1 ? multi_t<BS, 1>(h, S, p, s) : nrhs == 2 ? multi_t<BS, 2>(h, S, p, s) : multi_t<BS, 4>(h, S, p, s);
}

int wave_sweep_multi(bsp_handle_s* h, const WaveSym& S, const WaveVals& V, int nrhs, const double* rhs, double* x,
                     unsigned* ticket, const int* group_active, cudaStream_t stream) {
  if (!V.valid || !S.has_d || (nrhs != 1 && nrhs != 2 && nrhs != 4)) return BSP_INVALID;
  WaveP<double> p = wave_params<double>(h, S, V);
  p.group_active = group_active;
  p.rhs = rhs;
  p.x = x;
  p.xs = S.to_items ? wave_ld_of(S.bs * nrhs) : S.bs * nrhs;
  p.ticket = ticket;
  switch (S.bs) {
    case 4: return multi_r<4>(h, S, p, nrhs, stream);
    case 8: return multi_r<8>(h, S, p, nrhs, stream);
    case 16: return multi_r<16>(h, S, p, nrhs, stream);
    default: return BSP_INVALID;
  }
}

}  // namespace bsp
