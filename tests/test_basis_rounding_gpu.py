"""Gram-Schmidt where the new column nearly vanishes: A = I + s D with small s,
so A q_j is q_j up to s and its orthogonal part comes out of a cancellation.

The one-launch kernel takes a coefficient from the products with the column as
it was before the block of (up to seven) vectors it belongs to, corrected by
the products among them, so it carries eps ||v|| of the block's start; plain
modified Gram-Schmidt carries eps ||v|| after the vectors before it.  Both lose
orthogonality like eps times the condition of the Krylov vectors, which grows
as the residuals fall.  So the measure is plain modified Gram-Schmidt itself:
against 80-bit arithmetic the history is off by at most ten times what that
method is off by in double precision (the largest over four orders of the
rows, which change its rounding only; ten as in test_solvers_gpu.py) and a few
eps an entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.3e-16


def history(d, b, iters, real=np.longdouble):
    """Unpreconditioned GMRES of diag(d) by modified Gram-Schmidt, relative residuals."""
    num = (np.clongdouble if real is np.longdouble else np.complex128) if np.iscomplexobj(d) else real
    d, b = d.astype(num), b.astype(num)
    Q, g, rots, out = [b / np.sqrt(np.vdot(b, b).real)], [num(1)], [], [1.0]
    for j in range(iters):
        v, h = d * Q[j], []
        for q in Q:
            h.append(np.vdot(q, v))
            v = v - h[-1] * q
        nrm = np.sqrt(np.vdot(v, v).real)
        Q.append(v / nrm)
        for k, (c, s) in enumerate(rots):
            h[k], h[k + 1] = np.conj(c) * h[k] + np.conj(s) * h[k + 1], -s * h[k] + c * h[k + 1]
        r = np.sqrt(abs(h[j]) ** 2 + nrm ** 2)
        c, s = h[j] / r, nrm / r
        rots.append((c, s))
        g.append(-s * g[j])
        out.append(float(abs(g[-1])))
    return np.array(out)


@pytest.mark.parametrize("n", [37, 20000, 20001, 700001])
@pytest.mark.parametrize("s", [1e-2, 1e-4, 1e-6])
@pytest.mark.parametrize("cplx", [False, True])
def test_nearly_dependent_columns(handle, n, s, cplx):
    import blocksp_b200 as bsp
    rng = np.random.default_rng(n)
    d = 1.0 + s * rng.uniform(-1, 1, n)
    b = rng.uniform(-1, 1, n)
    if cplx:
        d, b = d + 1j * s * rng.uniform(-1, 1, n), b + 1j * rng.uniform(-1, 1, n)
    rp, ci, vals = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d.reshape(n, 1, 1)
    A = bsp.Matrix.from_complex(rp, ci, vals, handle=handle) if cplx else bsp.Matrix(rp, ci, vals, 1, handle=handle)
    _, _, hist = bsp.pGMRES(A, b, 1e-13, None, 12, return_info=True)
    A.close()
    ref = history(d, b, 8)
    k = int(np.sum(ref > 1e-12))  # falling, so these are the first ones
    assert 2 <= k <= len(ref) and len(hist) >= k
    off = np.zeros(k)
    for t in range(4):
        order = np.random.default_rng(t).permutation(n)
        off = np.maximum(off, np.abs(history(d[order], b[order], k, np.float64)[:k] - ref[:k]))
    assert np.all(np.abs(hist[:k] / hist[0] - ref[:k]) <= 10 * off + 4 * EPS * np.arange(1, k + 1))
