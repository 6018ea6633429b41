"""Infinities and NaN in the right-hand side of an application: the rows that
depend on them are not finite, as in the oracle, and every other row is what it
is without them.  Two systems that do not meet share the rows (even and odd),
so rows of both lie in the same steps of a sweep; rows of many entries are cut
into segments, and absent entries read a row of zeros.
"""
import numpy as np
import pytest

import oracle.blocksp_oracle as O
from test_apply_orders_gpu import rel, system
from test_sweep_choice import band, grid

pytestmark = pytest.mark.gpu


def twice(pattern):
    n, e = pattern
    return 2 * n, np.concatenate([2 * e, 2 * e + 1])


PATTERNS = {"band": band(300, range(2, 18, 2)), "grid": twice(grid((30, 21))), "grid3d": twice(grid((9, 8, 7)))}


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 8, 16])
def test_contained(handle, bad, pattern, bs):
    import blocksp_b200 as bsp
    s = system(PATTERNS[pattern], bs, 4)
    r = s.b.copy()
    row = s.n // 2 // 2 * 2  # an even one in the middle
    r[row * bs + bs // 2] = bad
    A, Ao = bsp.Matrix.from_system(s, handle), O.BSR.from_system(s)
    for make, ref in ((bsp.ILU0, O.ILU0), (bsp.IChol0, O.IChol0),
                      (lambda a: bsp.SOR(a, 1.2, 1, 1), lambda a: O.SOR(a, 1.2, 1, 1))):
        pc = make(A)
        got = pc.apply_host(r)
        with np.errstate(all="ignore"):
            want = ref(Ao)(r.copy())
        fin = np.isfinite(want).reshape(s.n, bs).all(1)
        assert fin[1::2].all() and not fin.all()
        assert np.array_equal(np.isfinite(got).reshape(s.n, bs).all(1), fin)
        keep = np.repeat(fin, bs)
        assert rel(got[keep], want[keep]) <= 1e-11
        # and the next application starts clean
        assert rel(pc.apply_host(s.b), ref(Ao)(s.b.copy())) <= 1e-11
        pc.close()
    A.close()
