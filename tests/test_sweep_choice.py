"""Which kernel runs a triangular sweep, and the lock-step plan on irregular
rows of several super-tasks, on the CPU.

The choice (csrc/sweep_cost.h) is checked where one side was measured more than
1.5 times as fast as the other.  The plans are run as the kernel runs them
(native/wave_plan_harness.cpp) in the shapes that the kernel has
(csrc/wave_shape.h), on rows of a random graph, a renumbered grid and long rows;
tolerance as in test_wave_plan.py: rounding carried through the sweep, 1e-13.
"""
import ctypes as C
import subprocess
import time
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


def build(tmp, name):
    out = tmp / f"{name}.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out), str(HERE / "native" / f"{name}.cpp")],
                   check=True)
    return C.CDLL(str(out))


@pytest.fixture(scope="module")
def choice(tmp_path_factory):
    return build(tmp_path_factory.mktemp("choice"), "sweep_choice_harness")


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    return build(tmp_path_factory.mktemp("plans"), "wave_plan_harness")


def p(a):
    return a.ctypes.data_as(C.c_void_p)


def grid(dims, wide=False):
    """Neighbour pairs of a grid in grid order: 5- / 7-point, or all around."""
    n, idx = int(np.prod(dims)), np.arange(int(np.prod(dims))).reshape(dims[::-1])
    out = []
    for s in np.ndindex(*(3,) * len(dims)):
        d = [k - 1 for k in s]
        if not any(d) or (not wide and sum(map(abs, d)) > 1):
            continue
        a = tuple(slice(max(0, -x), min(m, m - x)) for x, m in zip(d, idx.shape))
        b = tuple(slice(max(0, x), min(m, m + x)) for x, m in zip(d, idx.shape))
        out.append(np.stack([idx[a].ravel(), idx[b].ravel()], 1))
    return n, np.concatenate(out)


def renumbered(pattern, order):
    n, e = pattern
    new = np.empty(n, np.int64)
    new[order] = np.arange(n)
    return n, new[e]


def randomly(pattern, seed=1):
    return renumbered(pattern, np.random.default_rng(seed).permutation(pattern[0]))


def by_distance(pattern):
    """Rows by their distance from row 0, last first (as reverse Cuthill-McKee
    numbers them)."""
    n, e = pattern
    nb = [[] for _ in range(n)]
    for i, j in e:
        nb[i].append(int(j))
    seen, order = {0}, [0]
    for i in order:
        for j in nb[i]:
            if j not in seen:
                seen.add(j)
                order.append(j)
    return renumbered(pattern, np.array(order[::-1]))


def coloured(dims):
    n, e = grid(dims)
    return renumbered((n, e), np.argsort(np.indices(dims[::-1]).sum(0).ravel() % 2, kind="stable"))


def graph(n, k, seed=3):
    r = np.random.default_rng(seed)
    i, j = np.repeat(np.arange(n), k), r.integers(0, n, n * k)
    e = np.unique(np.stack([i, j], 1)[i != j], axis=0)
    return n, np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)


def band(n, dist):
    e = np.concatenate([np.stack([np.arange(n - d), np.arange(d, n)], 1) for d in dist])
    return n, np.concatenate([e, e[:, ::-1]])


def csr(pattern, ascending):
    n, e = pattern
    e = e[e[:, 1] < e[:, 0]] if ascending else e[e[:, 1] > e[:, 0]]
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]).astype(np.int32)
    return n, ptr, np.ascontiguousarray(e[:, 1], np.int32) if len(e) else np.zeros(1, np.int32)


def choose(lib, pattern, bs, ascending, streamed, limited=1):
    n, ptr, col = csr(pattern, ascending)
    o = np.zeros(5)
    took = lib.sweep_choice(n, int(ascending), bs, 1, int(streamed), limited, p(ptr), p(col), 0, None, p(o))
    return bool(took), o


BIG = {
    "grid3d": grid((40, 40, 40)), "grid2d": grid((200, 180)), "line": band(8000, [1]), "band8": band(6000, range(1, 9)),
    "rcm3d": by_distance(grid((40, 40, 40))), "random3d": randomly(grid((40, 40, 40))),
    "random2d": randomly(grid((200, 180))), "graph12": graph(40000, 12), "box27": grid((26, 26, 26), wide=True),
    "box27_random": randomly(grid((26, 26, 26), wide=True)),
}


@pytest.mark.parametrize("name,bs,lock_step", [
    *[("grid3d", b, True) for b in (1, 2, 3, 4, 5, 6)], *[("grid2d", b, True) for b in (1, 2, 3, 4, 5, 6, 8, 16)],
    *[("line", b, True) for b in (1, 2, 3, 4, 5, 6)], *[("band8", b, True) for b in (1, 2, 3, 4, 5, 6, 8, 16)],
    *[(s, b, False) for s in ("random3d", "random2d", "graph12", "box27_random") for b in (1, 2, 3, 4, 5, 6, 8, 16)],
    *[("rcm3d", b, False) for b in (3, 4, 5, 6, 8, 16)], *[("box27", b, False) for b in (3, 4, 5, 6, 8, 16)]])
def test_the_faster_kernel_is_chosen(choice, name, bs, lock_step):
    took = [choose(choice, BIG[name], bs, asc, bs >= 8)[0] for asc in (True, False)]
    assert took == [lock_step] * 2


def together(patterns):
    beg = np.concatenate([[0], np.cumsum([n for n, _ in patterns])])
    return (int(beg[-1]), np.concatenate([e + b for (_, e), b in zip(patterns, beg)])), beg.astype(np.int32)


@pytest.mark.parametrize("bs", [4, 8, 16])
@pytest.mark.parametrize("nrhs", [1, 4])
@pytest.mark.parametrize("name,lock_step", [("grid2d", True), ("grid3d", True), ("random2d", False), ("random3d", False),
                                            ("graph", False)])
def test_the_faster_kernel_is_chosen_in_a_batch(choice, name, lock_step, bs, nrhs):
    parts = {"grid2d": [grid((100 + 3 * i, 90)) for i in range(6)], "grid3d": [grid((20, 20, 12 + i)) for i in range(6)],
             "random2d": [randomly(grid((100 + 3 * i, 90)), i) for i in range(6)],
             "random3d": [randomly(grid((20, 20, 12 + i)), i) for i in range(6)],
             "graph": [graph(9000 + 100 * i, 3, i) for i in range(6)]}[name]
    pattern, beg = together(parts)
    for asc in (True, False):
        n, ptr, col = csr(pattern, asc)
        o = np.zeros(5)
        took = choice.sweep_choice(n, int(asc), bs, nrhs, 2, 1, p(ptr), p(col), len(parts), p(beg), p(o))
        assert bool(took) == lock_step, o


@pytest.mark.parametrize("bs", [4, 8])
def test_a_plan_that_is_too_slow_is_given_up_early(choice, bs):
    """The estimate grows with the super-tasks planned: a random order is left
    after a small part of it."""
    _, full = choose(choice, BIG["random3d"], bs, True, bs >= 8, limited=0)
    took, part = choose(choice, BIG["random3d"], bs, True, bs >= 8)
    assert not took and part[0] > 0.9 * part[1] and part[4] < 0.2 * full[4]


def test_planning_random_rows_takes_little_time(choice):
    """Under 0.5 us a row with the estimate (it took 4 us a row to plan them)."""
    pattern = csr(randomly(grid((64, 64, 64))), True)
    n, ptr, col = pattern
    o, best = np.zeros(5), 1e9
    for _ in range(3):
        t = time.process_time()
        choice.sweep_choice(n, 1, 4, 1, 0, 1, p(ptr), p(col), 0, None, p(o))
        best = min(best, time.process_time() - t)
    assert best <= 2.0 * 0.5e-6 * n  # twice that on a slow machine


IRREGULAR = {"random2d": randomly(grid((70, 66)), 5), "rcm3d": by_distance(grid((17, 16, 17))), "graph": graph(4100, 4),
             "box27": randomly(grid((16, 16, 17), wide=True), 7), "coloured": coloured((65, 66)),
             "band": band(4200, [1, 2, 3, 4, 5, 1500])}


@pytest.mark.parametrize("name", IRREGULAR)
@pytest.mark.parametrize("bs,nrhs", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 1), (6, 1), (8, 1), (16, 1), (4, 2), (8, 4),
                                     (16, 4)])
@pytest.mark.parametrize("ascending,has_d", [(True, False), (False, True)])
def test_plan_of_irregular_rows(choice, plans, name, bs, nrhs, ascending, has_d):
    s = np.zeros(6, np.int32)
    choice.sweep_shape(bs, nrhs, p(s))
    W, ecap, ring, slots, item_major, _ = map(int, s)
    n, ptr, col = csr(IRREGULAR[name], ascending)
    b = min(bs, 3)  # the plan does not depend on the values: small blocks keep the check short
    rng = np.random.default_rng(n + bs)
    vals = rng.uniform(-1, 1, (max(1, ptr[-1]), b, b)) / b
    rows = np.repeat(np.arange(n), np.diff(ptr))
    vals[:len(rows)] *= (0.5 / np.maximum(1, np.diff(ptr)))[rows][:, None, None]
    dinv, rhs = rng.uniform(-1, 1, (n, b, b)) / b + np.eye(b), rng.uniform(-1, 1, (n, b))
    x, st = np.full((n, b), np.nan), np.zeros(6, np.int32)
    rc = plans.wave_plan_run(n, int(ascending), b, W, ecap, ring, slots, int(has_d), item_major, p(ptr), p(col), p(vals),
                             p(dinv), p(rhs), 0, p(np.zeros(1, np.int32)), p(x), p(st))
    ref = np.zeros((n, b))
    for i in (range(n) if ascending else range(n - 1, -1, -1)):
        t = rhs[i] - sum((vals[e] @ ref[col[e]] for e in range(ptr[i], ptr[i + 1])), np.zeros(b))
        ref[i] = dinv[i] @ t if has_d else t
    assert rc == 0 and np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()
    # a band is one chain, and so one super-task
    assert st[0] == 1 if name == "band" else st[0] > 1


def test_shapes_of_the_kernel(choice):
    s = np.zeros(6, np.int32)
    for bs, nrhs, want in ((4, 1, (32, 16)), (4, 4, (32, 12)), (6, 1, (32, 16)), (8, 1, (16, 16)), (8, 2, (16, 8)),
                           (16, 1, (8, 8)), (16, 4, (4, 8)), (7, 1, (0, 0))):
        choice.sweep_shape(bs, nrhs, p(s))
        assert tuple(s[:2]) == want, bs
