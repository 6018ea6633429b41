// bsmv_rows.hpp — products whose blocks are not whole 16-byte chunks.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

struct bsp_matrix_s;

namespace bsp {

// y = alpha op(A) x + beta z for R (1 to 4) right-hand sides; the block rows of
// x, z and y are ld values apart.
template <typename VT, typename AT>
void bsmv_rows(const bsp_matrix_s* A, int R, int64_t ld, bool tr, const VT* vals, const AT* x, AT alpha, AT beta,
               const AT* z, AT* y, cudaStream_t s);

}  // namespace bsp
