"""Preconditioner applications on rows in every kind of order: grids, renumbered
grids, random and coloured rows, meshes, long rows, several super-tasks or
levels of each, whichever kernel takes them; against the CPU oracle, 1e-11 of
the largest entry as in test_precond_gpu.py.  And with too little memory for
the copies in sweep order, where the level-ordered kernels take the sweeps.
"""
import numpy as np
import pytest

import oracle.blocksp_oracle as O
from blocksp_b200.systems import BSRSystem
from test_device_memory_gpu import MB, Filled
from test_sweep_choice import band, by_distance, coloured, graph, grid, randomly

pytestmark = pytest.mark.gpu

ORDERS = {"grid": grid((70, 66)), "random": randomly(grid((70, 66)), 5), "rcm": by_distance(grid((70, 66))),
          "rcm3d": by_distance(grid((17, 16, 17))), "graph": graph(4100, 3), "coloured": coloured((65, 66)),
          "box27": randomly(grid((16, 16, 17), wide=True), 7), "band": band(4200, [1, 2, 3, 1500])}


def system(pattern, bs, seed=0):
    """Symmetric and block diagonally dominant: I (1 + sum |w|) on the diagonal,
    w S off it with one symmetric S of norm 1."""
    n, e = pattern
    rng = np.random.default_rng(seed)
    e = np.concatenate([e, np.stack([np.arange(n)] * 2, 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    key = np.minimum(e[:, 0], e[:, 1]) * n + np.maximum(e[:, 0], e[:, 1])
    _, inv = np.unique(key, return_inverse=True)
    w = rng.uniform(-1, 1, inv.max() + 1)[inv]
    on = e[:, 0] == e[:, 1]
    w[on] = 0.0
    diag = 1.0 + np.bincount(e[:, 0], np.abs(w), minlength=n)
    S = rng.uniform(-1, 1, (bs, bs))
    S = (S + S.T) / np.linalg.norm(S + S.T, 2)
    vals = w[:, None, None] * S
    vals[on] = diag[:, None, None] * (np.eye(bs) + 0.2 * S)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]).astype(np.int32)
    return BSRSystem(n=n, bs=bs, row_ptr=ptr, col_idx=e[:, 1].astype(np.int32), vals=vals,
                     b=rng.uniform(-1, 1, n * bs), name="order")


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 6, 8, 16])
@pytest.mark.parametrize("order", ORDERS)
def test_orders(handle, order, bs):
    import blocksp_b200 as bsp
    s = system(ORDERS[order], bs)
    A, Ao = bsp.Matrix.from_system(s, handle), O.BSR.from_system(s)
    for name, make, ref in (("ILU0", bsp.ILU0, O.ILU0), ("IChol0", bsp.IChol0, O.IChol0),
                            ("SOR", lambda a: bsp.SOR(a, 1.2, 2, 0), lambda a: O.SOR(a, 1.2, 2, 0))):
        pc = make(A)
        want = ref(Ao)(s.b.copy())
        for _ in range(2):
            assert rel(pc.apply_host(s.b), want) <= 1e-11, name
        pc.close()
    A.close()


@pytest.mark.parametrize("order", ["grid", "random"])
@pytest.mark.parametrize("kind", ["ILU0", "IChol0", "SOR"])
def test_without_memory_for_the_copies(torch_cuda, order, kind):
    """8x8 blocks whose copies take 200 MB and more, with 150 MB left."""
    import blocksp_b200 as bsp
    h = bsp.Handle(0)
    pattern = grid((60, 60, 40))
    s = system(pattern if order == "grid" else randomly(pattern), 8)

    def make(A):
        return bsp.SOR(A, 1.2, 1, 0) if kind == "SOR" else getattr(bsp, kind)(A)

    A = bsp.Matrix.from_system(s, h)
    pc = make(A)
    want = pc.apply_host(s.b)
    pc.close()
    A.close()  # a matrix keeps the memory of its preconditioners
    A = bsp.Matrix.from_system(s, h)
    pc = make(A)
    r = torch_cuda.from_numpy(s.b).cuda()
    with Filled(torch_cuda, 150 * MB):
        pc(r)
        torch_cuda.cuda.synchronize()
    assert rel(r.cpu().numpy(), want) <= 1e-11
    pc.close()
    A.close()
    h.close()
