"""The lock-step sweep plan (csrc/wave_plan.h), run on the host.

The harness executes a plan as the kernel does and checks every limit (items
and external rows per step, the ring of recent results, publication order);
its result is compared with a row-by-row sweep in natural order.  Tolerance:
both sum the same products of a row in another order, so they differ by
rounding carried through the sweep; the blocks are scaled so that a row's
off-diagonal blocks sum to at most 1/2 in norm, which bounds the growth, and
1e-13 of the largest entry is over 100 eps for the longest row (40 blocks).
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent

# (items per step, external rows, ring, slots) the kernel uses per block size
SHAPES = {1: (256, 64, 8, 8), 2: (128, 64, 8, 8), 3: (64, 32, 8, 8), 4: (64, 32, 8, 8), 5: (32, 16, 8, 8),
          8: (16, 16, 8, 8), 16: (8, 8, 8, 8)}


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("wave") / "wave_plan.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out),
                    str(HERE / "native" / "wave_plan_harness.cpp")], check=True)
    return C.CDLL(str(out))


def grid(dims, wide=False):
    """Neighbours of every grid row: 5- / 7-point, or with all diagonals."""
    n, nd = int(np.prod(dims)), len(dims)
    strides = np.cumprod([1, *dims[:-1]])
    deps = [[] for _ in range(n)]
    shifts = [s for s in np.ndindex(*(3,) * nd)]
    for i in range(n):
        co = [(i // strides[a]) % dims[a] for a in range(nd)]
        for s in shifts:
            d = [k - 1 for k in s]
            if not any(d) or (not wide and sum(map(abs, d)) > 1):
                continue
            c = [co[a] + d[a] for a in range(nd)]
            if all(0 <= c[a] < dims[a] for a in range(nd)):
                deps[i].append(int(sum(c[a] * strides[a] for a in range(nd))))
    return n, deps


def banded(n, w):
    return n, [[j for j in range(max(0, i - w), min(n, i + w + 1)) if j != i] for i in range(n)]


def random_rows(n, k, seed):
    rng = np.random.default_rng(seed)
    return n, [sorted(set(map(int, rng.integers(0, n, k))) - {i}) for i in range(n)]


PATTERNS = {
    "one_row": (1, [[]]), "no_entries": (700, [[] for _ in range(700)]), "line": banded(130, 1),
    "grid2d": grid((23, 19)), "grid2d_long": grid((150, 9)), "grid2d_tall": grid((5, 140)),
    "grid3d": grid((9, 11, 10)), "grid3d_flat": grid((12, 3, 14)), "grid3d_wide": grid((7, 6, 5), wide=True),
    "grid2d_wide": grid((20, 17), wide=True), "band40": banded(160, 40), "random": random_rows(600, 9, 1),
    "random_sparse": random_rows(900, 2, 2),
}


def run(lib, n, deps, bs, ascending, has_d, shape, groups=()):
    rng = np.random.default_rng(n + bs)
    rows = [[j for j in d if (j < i if ascending else j > i)] for i, d in enumerate(deps)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.array([j for r in rows for j in r] or [0], np.int32)
    vals = rng.uniform(-1, 1, (max(1, ptr[-1]), bs, bs)) / bs
    for i in range(n):
        vals[ptr[i]:ptr[i + 1]] *= 0.5 / max(1, ptr[i + 1] - ptr[i])
    dinv = rng.uniform(-1, 1, (n, bs, bs)) / bs + np.eye(bs)
    rhs = rng.uniform(-1, 1, (n, bs))
    x, stats = np.full((n, bs), np.nan), np.zeros(6, np.int32)
    gb = np.array(groups, np.int32)

    def p(a):
        return a.ctypes.data_as(C.c_void_p)

    rc = lib.wave_plan_run(n, int(ascending), bs, *shape, int(has_d), int(bs >= 4), p(ptr), p(col), p(vals), p(dinv), p(rhs),
                           len(gb), p(gb), p(x), p(stats))
    ref = np.zeros((n, bs))
    for i in (range(n) if ascending else reversed(range(n))):
        t = rhs[i].copy()
        for e in range(ptr[i], ptr[i + 1]):
            t -= vals[e] @ ref[col[e]]
        ref[i] = dinv[i] @ t if has_d else t
    return rc, x, ref, stats


@pytest.mark.parametrize("name", PATTERNS)
@pytest.mark.parametrize("bs", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("ascending,has_d", [(True, False), (False, True)])
def test_plan_runs_the_sweep(lib, name, bs, ascending, has_d):
    n, deps = PATTERNS[name]
    rc, x, ref, stats = run(lib, n, deps, bs, ascending, has_d, SHAPES[bs])
    assert rc == 0
    assert np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()
    assert stats[0] >= 1


def test_groups_are_kept_apart(lib):
    parts = [grid((9, 8)), grid((20, 31)), (3, [[], [], []]), grid((6, 6, 5))]
    deps, beg = [], [0]
    for n, d in parts:
        deps += [[j + beg[-1] for j in r] for r in d]
        beg.append(beg[-1] + n)
    for asc in (True, False):
        rc, x, ref, _ = run(lib, beg[-1], deps, 4, asc, True, SHAPES[4], beg)
        assert rc == 0 and np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()


def test_steps_follow_the_wavefront(lib):
    """A grid's super-task takes a step per diagonal of its rows: 4 x 4 chains
    of 64 rows in 64 + 6 steps, one CTA for a 2D system of 64 lines."""
    n, deps = grid((64, 8, 8))
    rc, _, _, stats = run(lib, n, deps, 8, True, False, SHAPES[8])
    assert rc == 0 and stats[0] == 4 and stats[1] == 4 * 70
    n, deps = grid((64, 64))
    rc, _, _, stats = run(lib, n, deps, 4, True, False, SHAPES[4])
    assert rc == 0 and stats[0] == 1 and stats[1] == 127


@pytest.mark.parametrize("dims,supers", [((80, 80), 10), ((20, 40), 5), ((6, 90), 1), ((9, 8), 1)])
def test_super_tasks_of_a_2d_grid(lib, dims, supers):
    """W = 8: long lines 8 to a super-task, a line's step after the one before;
    short lines as many as reach 1024 rows."""
    n, deps = grid(dims)
    rc, x, ref, stats = run(lib, n, deps, 16, True, True, SHAPES[16])
    assert rc == 0 and np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()
    assert stats[0] == supers
    if supers > 1:
        assert stats[1] == supers * (dims[0] + 7)


def test_not_triangular_is_refused(lib):
    ptr, col = np.array([0, 1, 1], np.int32), np.array([1], np.int32)
    one = np.zeros(16)
    st = np.zeros(6, np.int32)

    def p(a):
        return a.ctypes.data_as(C.c_void_p)

    assert lib.wave_plan_run(2, 1, 1, 16, 16, 8, 8, 0, 0, p(ptr), p(col), p(one), p(one), p(one), 0, p(ptr), p(one), p(st)) == 1
