// bsmv_rows.cu — block-sparse products for every block size.
//
// One thread per scalar row (block column entry of the transposed form) of the
// output, for up to four right-hand sides at once.  The threads of a warp read
// a contiguous stretch of the matrix between them, so the sectors that one
// load instruction leaves half used are taken from L1 by the next.  What it is
// bound by is loads in flight: the blocks of U stored entries and the entries
// of x that they meet are all requested before the first product, positions
// past the end of the row being read from its last block and left out.  Against
// a thread per value and right-hand side, one block after another (us, floor of
// the matrix bytes in brackets):
//   3 x 3, 250 x 201, 2 rhs          11.9 ->   9.0  (2.8; most of it the call)
//   3 x 3, 110^3, 1 | 2 rhs    207 | 334 -> 164 | 184  (104)
//   5 x 5, 78^3, 1 | 4 rhs     152 | 393 -> 140 | 222  (103)
//   1 x 1, 230^3, 1 | 4 rhs   330 | 1208 -> 230 | 735  (106)
//   transposed 3 x 3, 110^3, 2 rhs    268 -> 222  (104)
#include "bsmv_rows.hpp"
#include "internal.hpp"

namespace bsp {

constexpr int kRowThreads = 256;

template <typename AT, typename VT> __device__ __forceinline__ AT value_of(VT v) { return static_cast<AT>(v); }
template <typename AT> __device__ __forceinline__ AT value_of(__nv_bfloat16 v) {
  return static_cast<AT>(__bfloat162float(v));
}

// BSC: block size, 0 where it is only known at run time.  idx: column of each
// stored block (its row in the transposed form, where blk is its position).
template <int BSC, typename VT, typename AT, int R, bool TR>
__global__ void __launch_bounds__(kRowThreads)
k_bsmv_rows(int n, int bs_, int64_t ld, const int* __restrict__ ptr, const int* __restrict__ idx,
            const int64_t* __restrict__ blk, const VT* __restrict__ vals, const AT* __restrict__ x, AT alpha, AT beta,
            const AT* z, AT* y) {
  const int bs = BSC > 0 ? BSC : bs_;
  const int64_t e = (int64_t)blockIdx.x * kRowThreads + threadIdx.x;
  const int64_t row = e / bs;
  const int t = (int)(e - row * bs);
  if (row >= n) return;
  const int beg = __ldg(ptr + row), end = __ldg(ptr + row + 1);
  AT acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = AT(0);
  if constexpr (BSC > 0) {
    constexpr int kMost = 32 / (BSC * (R + 1));
    constexpr int U = kMost < 1 ? 1 : kMost > 8 ? 8 : kMost;
    for (int j = beg; j < end; j += U) {
      int64_t col[U], b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int q = min(j + u, end - 1);
        col[u] = __ldg(idx + q);
        b[u] = TR ? __ldg(blk + q) : (int64_t)q;
      }
      VT a[U][BSC];
      AT xv[U][R][BSC];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int c = 0; c < BSC; ++c) a[u][c] = __ldg(vals + b[u] * (BSC * BSC) + (TR ? c * BSC + t : t * BSC + c));
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < BSC; ++c) xv[u][r][c] = __ldg(x + col[u] * ld + r * BSC + c);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (j + u < end)
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = 0; c < BSC; ++c) acc[r] = fma(value_of<AT>(a[u][c]), xv[u][r][c], acc[r]);
    }
  } else {
    for (int j = beg; j < end; ++j) {
      const int64_t b = TR ? __ldg(blk + j) : (int64_t)j;
      const VT* a = vals + b * bs * bs + (TR ? t : t * bs);
      const AT* xj = x + (int64_t)__ldg(idx + j) * ld;
#pragma unroll 4
      for (int c = 0; c < bs; ++c) {
        const AT av = value_of<AT>(__ldg(a + (TR ? c * bs : c)));
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = fma(av, __ldg(xj + r * bs + c), acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t o = row * ld + r * bs + t;
    AT out = alpha * acc[r];
    if (beta != AT(0)) out += beta * z[o];
    y[o] = out;
  }
}

template <int BSC, typename VT, typename AT, int R>
static void launch_rows(const bsp_matrix_s* A, int64_t ld, bool tr, const VT* vals, const AT* x, AT alpha, AT beta,
                        const AT* z, AT* y, cudaStream_t s) {
  const int n = tr ? A->n_cols : A->n_rows;
  const int64_t grid = ceil_div((int64_t)n * A->bs, kRowThreads);
  if (grid == 0) return;
  if (tr)
    bsp::count_launch(), k_bsmv_rows<BSC, VT, AT, R, true><<<(unsigned)grid, kRowThreads, 0, s>>>(
        n, A->bs, ld, A->tr_ptr.get(), A->tr_row.get(), A->tr_blk.get(), vals, x, alpha, beta, z, y);
  else
    bsp::count_launch(), k_bsmv_rows<BSC, VT, AT, R, false><<<(unsigned)grid, kRowThreads, 0, s>>>(
        n, A->bs, ld, A->row_ptr.get(), A->col_idx.get(), nullptr, vals, x, alpha, beta, z, y);
}

// Sizes of 16-byte chunks come here for unaligned vectors only, and take the
// run-time form.
template <typename VT, typename AT, int R>
static void rows_of(const bsp_matrix_s* A, int64_t ld, bool tr, const VT* vals, const AT* x, AT alpha, AT beta,
                    const AT* z, AT* y, cudaStream_t s) {
  switch (A->bs) {
#define BSP_ROWS_CASE(BB)                                              \
  case BB:                                                             \
    if constexpr (BB == 6 || BB % Chunk<VT>::V != 0)                   \
      return launch_rows<BB, VT, AT, R>(A, ld, tr, vals, x, alpha, beta, z, y, s); \
    break;
    BSP_ROWS_CASE(1)
    BSP_ROWS_CASE(2)
    BSP_ROWS_CASE(3)
    BSP_ROWS_CASE(4)
    BSP_ROWS_CASE(5)
    BSP_ROWS_CASE(6)
#undef BSP_ROWS_CASE
    default: break;
  }
  launch_rows<0, VT, AT, R>(A, ld, tr, vals, x, alpha, beta, z, y, s);
}

template <typename VT, typename AT>
void bsmv_rows(const bsp_matrix_s* A, int R, int64_t ld, bool tr, const VT* vals, const AT* x, AT alpha, AT beta,
               const AT* z, AT* y, cudaStream_t s) {
  switch (R) {
    case 1: return rows_of<VT, AT, 1>(A, ld, tr, vals, x, alpha, beta, z, y, s);
    case 2: return rows_of<VT, AT, 2>(A, ld, tr, vals, x, alpha, beta, z, y, s);
    case 3: return rows_of<VT, AT, 3>(A, ld, tr, vals, x, alpha, beta, z, y, s);
    default: return rows_of<VT, AT, 4>(A, ld, tr, vals, x, alpha, beta, z, y, s);
  }
}

#define BSP_ROWS_TYPE(VT, AT)                                                                                        \
  template void bsmv_rows<VT, AT>(const bsp_matrix_s*, int, int64_t, bool, const VT*, const AT*, AT, AT, const AT*, \
                                  AT*, cudaStream_t);
BSP_ROWS_TYPE(double, double)
BSP_ROWS_TYPE(float, float)
BSP_ROWS_TYPE(float, double)
BSP_ROWS_TYPE(__nv_bfloat16, float)
BSP_ROWS_TYPE(__nv_bfloat16, double)
#undef BSP_ROWS_TYPE

}  // namespace bsp
