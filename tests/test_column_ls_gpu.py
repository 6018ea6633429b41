"""The least-squares update of the first columns of a GMRES cycle: the lanes of
a warp bring the column to shared memory and one of them rotates it, with no
older rotations in between on the first column of a solve and of every plain
restart.  Short cycles (mostly first columns) and columns past the 32 lanes,
against the CPU oracle; tolerances of test_solvers_gpu.py.
"""
import re
from pathlib import Path

import numpy as np
import pytest

import oracle.blocksp_oracle as O
from blocksp_b200.systems import grid_system

CSRC = Path(__file__).resolve().parents[1] / "blocksp_b200" / "csrc"


def test_column_is_complete_before_it_is_rotated():
    """Between the lanes' stores of the column and the first read by one lane
    the warp meets on every path, also where the loop over rotations is empty."""
    src = (CSRC / "krylov.cu").read_text()
    fill = src.index("col[i] = g.H[i * g.m + j];")
    loop = src.index("for (int t0 = 0; t0 < nrot", fill)
    assert re.search(r"__syncwarp\(\);", src[fill:loop])


@pytest.mark.gpu
@pytest.mark.parametrize("restart,k", [(1, 0), (2, 0), (3, 0), (35, 0), (40, 3), (-1, -1)])
@pytest.mark.parametrize("dims,bs", [((6, 6, 6), 4), ((9, 8), 3)])
def test_short_and_long_cycles(handle, dims, bs, restart, k):
    import blocksp_b200 as bsp
    s = grid_system(dims, bs, seed=31, skew=0.3)
    A, Ao = bsp.Matrix.from_system(s, handle), O.BSR.from_system(s)
    pc = bsp.ILU0(A)
    limit = 60 if 0 < restart < 4 else 2000
    x, info, hist = bsp.pGMRES(A, s.b, 1e-10, pc, limit, restart, k, return_info=True)
    ref = O.pgmres(Ao, s.b, 1e-10, O.ILU0(Ao), limit, restart, k)
    n = min(len(hist), len(ref.hist))
    assert abs(len(hist) - len(ref.hist)) <= 2 and n >= 3
    h, r = np.asarray(hist[:n]) / hist[0], np.asarray(ref.hist[:n]) / ref.hist[0]
    assert np.abs(h - r).max() <= 1e-10
    assert np.abs(x - ref.x).max() <= 1e-8 * np.abs(ref.x).max()
    pc.close()
    A.close()
