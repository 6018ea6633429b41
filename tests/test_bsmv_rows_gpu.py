"""Products over every block size that is not whole 16-byte chunks, groups of
right-hand sides, and vectors off 16-byte boundaries, against the CPU oracle.

Tolerances: a row of at most 12 blocks of at most 24 values has n <= 288
products; the recursive sum is within n u sum|a||x| of the exact value, so
n * 2**-53 (FP64 accumulation) or n * 2**-24 (FP32) of sum|a||x| bounds the
error entry by entry, twice that between two such sums.
"""
import numpy as np
import pytest

import oracle.blocksp_oracle as O
from blocksp_b200.systems import BSRSystem

pytestmark = pytest.mark.gpu

N = 83


def ragged(bs, seed):
    """Rows of 0 to 12 blocks in shuffled column order."""
    rng = np.random.default_rng(seed)
    rp, ci = [0], []
    for i in range(N):
        ci.extend(rng.permutation(N)[: i % 13].tolist())
        rp.append(len(ci))
    vals = rng.standard_normal((len(ci), bs, bs))
    return BSRSystem(n=N, bs=bs, row_ptr=np.array(rp, np.int32), col_idx=np.array(ci, np.int32), vals=vals,
                     b=np.zeros(N * bs))


CASES = [(bs, "f64", nrhs, 0) for bs in (1, 2, 3, 4, 5, 6, 7, 8, 12, 16, 24) for nrhs in (1, 2, 3, 4, 5, 6, 9)]
CASES += [(bs, dt, nrhs, 0) for dt in ("f32", "bf16") for bs in (1, 2, 3, 4, 6, 8, 12) for nrhs in (1, 4, 7)]
CASES += [(bs, "f64", nrhs, 1) for bs in (2, 4, 8, 16) for nrhs in (1, 5)]


@pytest.mark.parametrize("bs,dtype,nrhs,shift", CASES)
@pytest.mark.parametrize("transpose", [False, True])
def test_every_block_size(handle, torch_cuda, bs, dtype, nrhs, shift, transpose):
    import blocksp_b200 as bsp
    from blocksp_b200 import _lib
    torch = torch_cuda
    s = ragged(bs, 100 * bs + nrhs)
    rng = np.random.default_rng(bs + nrhs)
    x, y0 = rng.uniform(-1, 1, (2, N * bs * nrhs))
    td = torch.float64
    u = 2.0 ** -53
    if dtype != "f64":
        td, u = torch.float32, 2.0 ** -24
        x, y0 = x.astype(np.float32).astype(np.float64), y0.astype(np.float32).astype(np.float64)
    A = bsp.Matrix.from_system(s, handle)
    code, kept = _lib.BSP_F64, s.vals
    if dtype == "f32":
        code, kept = _lib.BSP_F32, s.vals.astype(np.float32).astype(np.float64)
    elif dtype == "bf16":
        code, kept = _lib.BSP_BF16, torch.tensor(s.vals).to(torch.bfloat16).to(torch.float64).numpy()
    if code != _lib.BSP_F64:
        A.make_lowp(code)
    B = O.BSR(N, bs, s.row_ptr, s.col_idx, kept)
    Babs = O.BSR(N, bs, s.row_ptr, s.col_idx, np.abs(kept))
    ref = O.bsmv(B, x, nrhs=nrhs, transpose=transpose)
    size = O.bsmv(Babs, np.abs(x), nrhs=nrhs, transpose=transpose)
    base = torch.zeros(x.size + shift, dtype=td, device="cuda")
    xd = base[shift:]
    xd.copy_(torch.tensor(x, dtype=td))
    # the transposed form has up to N blocks in a column
    n = (N if transpose else 12) * bs + 4
    y = torch.full((x.size,), float("nan"), dtype=td, device="cuda")
    bsp.bsmv_dev(A, xd, y, nrhs=nrhs, transpose=transpose, dtype=code)
    handle.sync()
    assert np.all(np.abs(y.cpu().double().numpy() - ref) <= 2 * n * u * size)
    y = torch.tensor(y0, dtype=td, device="cuda")
    bsp.bsmv_dev(A, xd, y, nrhs=nrhs, alpha=-0.5, beta=2.0, transpose=transpose, dtype=code)
    handle.sync()
    assert np.all(np.abs(y.cpu().double().numpy() - (2.0 * y0 - 0.5 * ref)) <= 2 * n * u * (size + 2 * np.abs(y0)))
