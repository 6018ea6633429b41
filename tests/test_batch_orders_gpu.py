"""Batched solves whose systems have rows in several orders, so that groups run
through the lock-step or the level-ordered sweeps, with the number of
right-hand sides changing on one object; against the oracle per pair.  The
systems are diagonally dominant (condition below 10), so the solution at
tolerance 1e-10 agrees to 1e-8 as in test_batch_gpu.py and the iteration
counts to one.
"""
import numpy as np
import pytest

import oracle.blocksp_oracle as O
from test_apply_orders_gpu import rel, system
from test_sweep_choice import by_distance, coloured, graph, grid, randomly

pytestmark = pytest.mark.gpu

SETS = {
    "grids": [grid((31, 33)), grid((9, 70)), grid((6, 7, 8))],
    "random": [randomly(grid((60, 59)), 2), graph(2100, 4), randomly(grid((14, 13, 12)), 3)],
    "mixed": [by_distance(grid((50, 41))), coloured((40, 41)), grid((1, 1)), graph(1500, 2)],
}


@pytest.mark.parametrize("bs", [4, 8, 16])
@pytest.mark.parametrize("name", SETS)
def test_orders(handle, name, bs):
    import blocksp_b200 as bsp
    sl = [system(p, bs, k) for k, p in enumerate(SETS[name])]
    B = bsp.Batch(sl, handle)
    ref = {}
    for nrhs in (1, 4, 2, 1):
        rng = np.random.default_rng(9)
        cols = [[rng.uniform(-1, 1, (s.n, s.bs)) for _ in range(4)][:nrhs] for s in sl]
        b = np.concatenate([np.stack(c, 1).ravel() for c in cols])
        x, info = B.pcg(b, nrhs, 1e-10, 500)
        assert info["status"] == 0
        its, off = B.results()["iters"], B.offsets(nrhs)
        for k, s in enumerate(sl):
            got = x[off[k]:off[k + 1]].reshape(s.n, nrhs, s.bs)
            Ao = O.BSR.from_system(s)
            for r in range(nrhs):
                if (k, r) not in ref:
                    ref[k, r] = O.pcg(Ao, cols[k][r].ravel(), 1e-10, O.IChol0(Ao), 500)
                o = ref[k, r]
                assert abs(int(its[k, r]) - o.iters) <= 1
                assert rel(got[:, r].ravel(), o.x) <= 1e-8
    B.close()


def test_a_group_swept_by_levels_gives_up_its_waits(handle):
    """The bounded waits of the level-ordered sweeps: one re-poll, a status, and
    the object computes again."""
    import blocksp_b200 as bsp
    s = system(randomly(grid((30, 30, 30)), 4), 8)
    B = bsp.Batch([s], handle)
    x, info = B.pcg(s.b, 1, 1e-10, 500)
    assert info["status"] == 0
    handle.set_spin_limit(1)
    try:
        with pytest.raises(Exception) as ei:
            B.pcg(s.b, 1, 1e-10, 500, retune=False, hist_cap=3)
        assert getattr(ei.value, "status", None) == 6
    finally:
        handle.set_spin_limit()
    again, info = B.pcg(s.b, 1, 1e-10, 500)
    assert info["status"] == 0 and np.array_equal(x, again)
    B.close()


@pytest.mark.parametrize("batch_first", [True, False])
def test_batch_and_preconditioner_share_a_pattern(handle, batch_first):
    """A batch of one system has the pattern of the system's own matrix, whose
    analysis it shares without the layout of the sweeps: whichever comes first,
    the preconditioner applies as the oracle's and the batch solves."""
    import blocksp_b200 as bsp
    s = system(grid((41, 37)), 8, 11)
    Ao = O.BSR.from_system(s)
    want = O.IChol0(Ao)(s.b.copy())

    def batch():
        B = bsp.Batch([s], handle)
        x, info = B.pcg(s.b, 1, 1e-10, 500)
        assert info["status"] == 0 and rel(x, O.pcg(Ao, s.b, 1e-10, O.IChol0(Ao), 500).x) <= 1e-8
        B.close()

    def precond():
        A = bsp.Matrix.from_system(s, handle)
        pc = bsp.IChol0(A)
        assert rel(pc.apply_host(s.b), want) <= 1e-11
        pc.close()
        A.close()

    for f in ((batch, precond, precond, batch) if batch_first else (precond, batch, batch, precond)):
        f()
