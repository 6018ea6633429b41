"""A Batch object keeps its launch graphs from one call to the next; what
belongs to one call (its tolerance and iteration limit) must not stay in them.
A call after one with another limit returns what a fresh object returns, bit
for bit (the same kernels on the same inputs; reductions in a fixed order).
"""
import numpy as np
import pytest

from blocksp_b200 import systems

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("limits", [(3, 2000), (2000, 3, 2000), (0, 7)])
def test_iteration_limit_of_this_call(handle, mode, limits):
    import blocksp_b200 as bsp
    sl = [systems.batch_system(side, bs, seed, nrhs=2) for side, bs, seed in ((12, 4, 1), (9, 8, 2), (7, 4, 3))]
    b = np.concatenate([s.b for s in sl])
    B = bsp.Batch(sl, handle)
    for limit in limits:
        x, info = B.pcg(b, 2, TOL, limit, mode=mode)
    kept = B.results()
    B.close()
    F = bsp.Batch(sl, handle)
    xf, fresh_info = F.pcg(b, 2, TOL, limits[-1], mode=mode)
    fresh = F.results()
    F.close()
    assert info["status"] == fresh_info["status"] == (0 if limits[-1] == 2000 else 4)
    assert np.array_equal(kept["iters"], fresh["iters"]) and np.array_equal(kept["state"], fresh["state"])
    assert np.array_equal(x, xf)
