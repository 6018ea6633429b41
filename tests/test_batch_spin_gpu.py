"""The bound of the device waits that holds for a batched solve is the handle's
at the time of the call, also when the object has kept a graph from a call
under another bound: one re-poll makes the waits run out (the kernels return a
status), the default bound solves again."""
import numpy as np
import pytest

from test_apply_orders_gpu import system
from test_sweep_choice import grid, randomly

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "random"])
def test_bound_of_this_call(handle, order):
    import blocksp_b200 as bsp
    pattern = grid((40, 40, 40))
    s = system(pattern if order == "grid" else randomly(pattern, 4), 8)
    B = bsp.Batch([s], handle)
    x, info = B.pcg(s.b, 1, 1e-10, 500)
    assert info["status"] == 0
    handle.set_spin_limit(1)
    try:
        with pytest.raises(Exception) as ei:
            B.pcg(s.b, 1, 1e-10, 500)
        assert getattr(ei.value, "status", None) == 6
    finally:
        handle.set_spin_limit()
    again, info = B.pcg(s.b, 1, 1e-10, 500)
    assert info["status"] == 0 and np.array_equal(x, again)
    B.close()
