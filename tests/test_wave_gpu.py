"""The lock-step sweeps on the GPU at the sizes where their layout can go wrong:
tiles that do not divide the grid, lines longer and shorter than a tile, one
row, rows cut into segments, external rows past a step's limit, vectors that
are only 8-byte aligned; against the CPU oracle.

Tolerance: 1e-11 of the largest entry, the bound of one preconditioner
application in test_precond_gpu.py (block rows are summed in another order
than the oracle's, and the blocks are premultiplied by the inverted diagonal).
"""
import numpy as np
import pytest

import oracle.blocksp_oracle as O
from blocksp_b200.systems import BSRSystem, grid_system

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1), (1, 40), (3, 150), (140, 5), (37, 33), (5, 6, 7), (33, 9, 4), (4, 3, 35), (2, 18, 17)]


def rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(b).max(), 1e-300)


def band_system(n, bs, w, seed, wide=0):
    """Symmetric, block diagonally dominant: w neighbours on each side and one
    at distance `wide` (0: none)."""
    rng = np.random.default_rng(seed)
    dist = list(range(1, w + 1)) + ([wide] if wide else [])
    rows = [sorted({i} | {i + s * d for d in dist for s in (-1, 1) if 0 <= i + s * d < n}) for i in range(n)]
    off = {(i, j): rng.uniform(-1, 1, (bs, bs)) for i in range(n) for j in rows[i] if j > i}
    rp, ci, va = [0], [], []
    for i in range(n):
        for j in rows[i]:
            ci.append(j)
            va.append(off[(i, j)] if j > i else off[(j, i)].T if j < i else
                      (2.0 * bs * (len(dist) * 2) + 1.0) * np.eye(bs))
        rp.append(len(ci))
    return BSRSystem(n=n, bs=bs, row_ptr=np.array(rp, np.int32), col_idx=np.array(ci, np.int32), vals=np.array(va),
                     b=rng.uniform(-1, 1, n * bs), name="band")


def check(handle, s, kinds=("ILU0", "IChol0")):
    import blocksp_b200 as bsp
    A, Ao = bsp.Matrix.from_system(s, handle), O.BSR.from_system(s)
    r = np.random.default_rng(3).uniform(-1, 1, s.n * s.bs)
    for kind in kinds:
        pc = getattr(bsp, kind)(A)
        ref = getattr(O, kind)(Ao)(r.copy())
        assert rel(pc.apply_host(r), ref) <= 1e-11, kind
        assert rel(pc.apply_host(r), ref) <= 1e-11, kind  # the ticket and the sentinels are back in place
        pc.close()
    A.close()


@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 6, 8, 16])
@pytest.mark.parametrize("dims", GRIDS)
def test_grids(handle, dims, bs):
    check(handle, grid_system(dims, bs, seed=11))


@pytest.mark.parametrize("bs", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("n,w,wide", [(90, 7, 0), (400, 2, 61), (60, 40, 0), (300, 1, 150)])
def test_long_rows_and_far_rows(handle, bs, n, w, wide):
    check(handle, band_system(n, bs, w, 5, wide))


@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 6, 8, 16])
@pytest.mark.parametrize("kind,nu", [(0, 3), (1, 1), (1, 2), (-1, 1), (-1, 2)])
def test_sor(handle, bs, kind, nu):
    """SOR on the same sweeps: one and several, each way and both (in place)."""
    import blocksp_b200 as bsp
    for s in (grid_system((37, 33), bs, seed=6), grid_system((5, 6, 7), bs, seed=6, skew=0.3),
              band_system(60, bs, 9, 2), grid_system((1, 1), bs, seed=6)):
        A, Ao = bsp.Matrix.from_system(s, handle), O.BSR.from_system(s)
        r = np.random.default_rng(8).uniform(-1, 1, s.n * bs)
        pc = bsp.SOR(A, 1.3, nu, kind)
        assert rel(pc.apply_host(r), O.SOR(Ao, 1.3, nu, kind)(r.copy())) <= 1e-11
        pc.close()
        A.close()


@pytest.mark.parametrize("bs", [4, 8])
def test_vectors_aligned_to_one_value(handle, torch_cuda, bs):
    import blocksp_b200 as bsp
    s = grid_system((7, 6, 5), bs, seed=4)
    pc = bsp.ILU0(bsp.Matrix.from_system(s, handle))
    n = s.n * bs
    buf = torch_cuda.zeros(n + 1, dtype=torch_cuda.float64, device="cuda")
    r = buf[1:]
    r.copy_(torch_cuda.from_numpy(s.b))
    assert r.data_ptr() % 16 == 8
    pc(r)
    ref = O.ILU0(O.BSR.from_system(s))(s.b.copy())
    assert rel(r.cpu().numpy(), ref) <= 1e-11
