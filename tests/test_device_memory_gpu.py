"""Calls near the end of the device's memory: an allocation that a solve only
asks for ahead of its need may fail without ending the solve, and a call that
does run out leaves its objects usable.  The rest of the memory is held by one
(untouched) torch allocation.
"""
import numpy as np
import pytest

from blocksp_b200 import systems

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Filled:
    """All but `leave` bytes of the device's free memory, held."""

    def __init__(self, torch, leave):
        from blocksp_b200 import _lib
        self.torch, self.leave, self.lib = torch, leave, _lib.load()

    def __enter__(self):
        self.torch.cuda.synchronize()
        self.lib.bsp_release_cached_memory(0)
        free, _ = self.torch.cuda.mem_get_info()
        self.block = self.torch.empty(free - self.leave, dtype=self.torch.uint8, device="cuda")
        left, _ = self.torch.cuda.mem_get_info()
        assert abs(left - self.leave) <= 32 * MB
        return self

    def __exit__(self, *a):
        del self.block
        self.torch.cuda.empty_cache()


def diagonal(bsp, handle, n, eigenvalues, cplx):
    """A diagonal matrix with few distinct eigenvalues: GMRES takes as many steps."""
    d = np.resize(np.asarray(eigenvalues, complex if cplx else float), n)
    rp, ci = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    vals = d.reshape(n, 1, 1)
    A = bsp.Matrix.from_complex(rp, ci, vals, handle=handle) if cplx else bsp.Matrix(rp, ci, vals, 1, handle=handle)
    return A, d


def test_complex_basis_asked_for_ahead(torch_cuda):
    """Three steps need four basis vectors; up to nine are asked for."""
    import blocksp_b200 as bsp
    h = bsp.Handle(0)
    n = 1 << 21  # 32 MiB a vector
    A, d = diagonal(bsp, h, n, [1.0, 2.0 + 1j, 3.0], True)
    rng = np.random.default_rng(1)
    b = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    bsp.pGMRES(A, b, 1e-10, None, 0)  # what does not grow with the steps, and two vectors
    with Filled(torch_cuda, 5 * 32 * MB):
        x, info, _ = bsp.pGMRES(A, b, 1e-10, None, 20, return_info=True)
    assert info["status"] == 0 and info["iters"] <= 4
    # |x - b / d| <= tol ||b|| / min |d| = 1e-10 x 1200
    assert np.abs(x - b / d).max() <= 1e-6
    A.close()
    h.close()


def test_real_basis_asked_for_ahead(torch_cuda):
    """Sixteen vectors are there, which fifteen steps need; the next sixteen do
    not fit."""
    import blocksp_b200 as bsp
    h = bsp.Handle(0)
    n = 1 << 21  # 16 MiB a vector
    A, d = diagonal(bsp, h, n, np.linspace(1.0, 30.0, 15), False)
    b = np.random.default_rng(2).uniform(-1, 1, n)
    _, first, _ = bsp.pGMRES(A, b, 1e-9, None, 13, return_info=True)
    assert first["status"] == 4
    with Filled(torch_cuda, 100 * MB):
        x, info, _ = bsp.pGMRES(A, b, 1e-9, None, 40, return_info=True)
    assert info["status"] == 0 and info["iters"] <= 15
    assert np.abs(x - b / d).max() <= 1e-5  # tol ||b|| / min |d| = 1e-9 x 840
    A.close()
    h.close()
