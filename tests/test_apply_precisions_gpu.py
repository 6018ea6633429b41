"""Factors and inner operators stored in FP32 and BF16 on rows in every kind of
order, so through the lock-step, the streamed and the level-ordered sweeps:
solves to an FP64 true residual of 1e-10 by refinement, from the same
right-hand side as the FP64 solve.  The solution is within cond * 1e-10 of the
oracle's (cond below 10: 1e-8 with room)."""
import numpy as np
import pytest

import oracle.blocksp_oracle as O
from test_apply_orders_gpu import ORDERS, rel, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [2, 4, 8, 16])
@pytest.mark.parametrize("order", ["grid", "random", "rcm3d", "coloured"])
@pytest.mark.parametrize("precision", ["F32", "BF16"])
def test_refined_solve(handle, order, bs, precision):
    import blocksp_b200 as bsp
    from blocksp_b200 import _lib
    s = system(ORDERS[order], bs, 6)
    A, Ao = bsp.Matrix.from_system(s, handle), O.BSR.from_system(s)
    want = None
    for kind, solve in (("ILU0", bsp.pGMRES), ("IChol0", bsp.pCG)):
        pc = getattr(bsp, kind)(A)
        x, info, _ = solve(A, s.b, 1e-10, pc, 500, return_info=True, precision=getattr(_lib, "PREC_" + precision))
        assert info["status"] == 0
        assert O.true_rel_residual(Ao, s.b, x) <= 1.1e-10
        if want is None:
            want = O.pcg(Ao, s.b, 1e-13, O.IChol0(Ao), 500).x
        assert rel(x, want) <= 1e-8
        pc.close()
    A.close()
