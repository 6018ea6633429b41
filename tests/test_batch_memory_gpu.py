"""A batched solve that runs out of memory while it makes its state for another
number of right-hand sides leaves the object usable: the next call makes the
state again instead of running a kept graph on buffers that are gone."""
import ctypes as C

import numpy as np
import pytest

from test_apply_orders_gpu import system
from test_device_memory_gpu import MB, Filled
from test_sweep_choice import grid, randomly

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "random"])
def test_out_of_memory_between_two_solves(torch_cuda, order):
    import blocksp_b200 as bsp
    from blocksp_b200 import _lib
    torch = torch_cuda
    h = bsp.Handle(0)
    pattern = grid((60, 60, 60))
    s = system(pattern if order == "grid" else randomly(pattern), 8)  # 13.8 MB a vector and right-hand side
    B = bsp.Batch([s], h)
    b1 = torch.from_numpy(s.b).cuda()
    b4, x4 = b1.repeat(4), torch.empty(4 * s.b.size, dtype=torch.float64, device="cuda")

    def solve(nrhs):
        opts, info = _lib.BatchOpts(1e-10, 200, 0, 8, 0, 0), _lib.BatchInfo()
        return h.lib.bsp_batch_pcg_dev(h.h, B.b, nrhs, C.c_void_p(b4.data_ptr()), C.c_void_p(x4.data_ptr()),
                                       C.byref(opts), C.byref(info))

    x1, info = B.pcg(b1, 1, 1e-10, 200)
    assert info["status"] == 0
    for fail in (4, 2):
        with Filled(torch, 48 * MB):  # a few vectors of one right-hand side at most
            assert solve(fail) == 10
        again, info = B.pcg(b1, 1, 1e-10, 200)
        assert info["status"] == 0
        assert torch.equal(x1, again)
    assert solve(4) == 0 and np.isfinite(x4.cpu().numpy()).all()
    B.close()
    h.close()
