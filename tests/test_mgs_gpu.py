"""The one-launch Gram-Schmidt at every length where it takes another form
(basis vectors per grid barrier 7 to 1, then one pass per vector), real with
even and odd lengths and complex, against numpy.

A block diagonal matrix keeps the operator exact to a few eps, so the residual
history of unpreconditioned GMRES tests the orthogonalisation alone.  Both
sides run modified Gram-Schmidt; the history entries are relative to the first
residual and differ by rounding of sums over up to 4e6 products (about
sqrt(n) eps = 5e-13 in each coefficient): 1e-10, as for the solver tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ITERS = 17  # more than two blocks of seven vectors


def gmres_history(apply, b, iters):
    beta = np.sqrt(np.vdot(b, b).real)
    Q, H, hist = [b / beta], np.zeros((iters + 1, iters), b.dtype), [1.0]
    for j in range(iters):
        v = apply(Q[j])
        for i in range(j + 1):
            H[i, j] = np.vdot(Q[i], v)
            v = v - H[i, j] * Q[i]
        H[j + 1, j] = np.sqrt(np.vdot(v, v).real)
        Q.append(v / H[j + 1, j])
        rhs = np.zeros(j + 2, b.dtype)
        rhs[0] = 1.0
        y = np.linalg.lstsq(H[:j + 2, :j + 1], rhs, rcond=None)[0]
        hist.append(np.linalg.norm(rhs - H[:j + 2, :j + 1] @ y))
    return np.array(hist)


def run(handle, n, bs, cplx):
    import blocksp_b200 as bsp
    rng = np.random.default_rng(n)
    d = rng.uniform(0.5, 4.0, (n, bs))
    if cplx:
        d = d * np.exp(1j * rng.uniform(-0.5, 0.5, (n, bs)))
    vals = np.zeros((n, bs, bs), d.dtype)
    vals[:, np.arange(bs), np.arange(bs)] = d
    rp, ci = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    A = bsp.Matrix.from_complex(rp, ci, vals, handle=handle) if cplx else bsp.Matrix(rp, ci, vals, bs, handle=handle)
    b = rng.uniform(-1, 1, n * bs) + (1j * rng.uniform(-1, 1, n * bs) if cplx else 0.0)
    x, info, hist = bsp.pGMRES(A, b, 1e-30, None, ITERS - 1, return_info=True)
    A.close()
    ref = gmres_history(lambda q: d.reshape(-1) * q, b, ITERS)
    # the space of a very short vector is exhausted early: nothing is defined after that
    n = int(np.argmax(ref <= 1e-14)) if (ref <= 1e-14).any() else len(ref)
    assert len(hist) >= n and (n < len(ref) or len(hist) == n)
    assert np.abs(hist[:n] / hist[0] - ref[:n]).max() <= 1e-10


@pytest.mark.parametrize("values", [5, 1000, 303000, 303200, 606300, 909400, 1212500, 2121800, 3637300])
@pytest.mark.parametrize("odd", [False, True])
def test_real(handle, values, odd):
    run(handle, values | 1 if odd else values // 2, 1 if odd else 2, False)


@pytest.mark.parametrize("values", [2, 500, 151600, 303200, 454700, 606300, 1060900, 1818700])
def test_complex(handle, values):
    run(handle, values, 1, True)
