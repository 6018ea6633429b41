"""The workloads whose speed is followed, through the package's public calls.

A case is a dict of plain values; its "op" is the call it stands for:

* ``bsmv``   one block-sparse product ``y = op(A) x (+ z)`` on device tensors;
* ``apply``  one preconditioner application in place (what every Krylov
  iteration does twice or more);
* ``solve``  one solver object of the reference's kind, built and used: set-up
  of the preconditioner on a new matrix plus the whole Krylov solve;
* ``batch``  one batched block-IChol0 pCG over many systems and 4 right-hand
  sides.

The matrices are 5-point / 7-point block stencils on 2D / 3D grids, the shape
of every configuration, test and benchmark of this repository: a grid edge
(p, q) adds K = G G^T + 0.1 I to A_pp and A_qq and -K to A_pq and A_qp, and
0.01 I is added to every diagonal block; ``skew`` adds c (S - S^T) to A_pq and
A_qp.  They are drawn on the GPU (the sizes take seconds on the host) and
handed to the package as the host arrays its containers are packed from.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

import blocksp_b200 as bsp
from blocksp_b200 import _lib

DEV = "cuda"
DTYPES = {"f64": _lib.BSP_F64, "f32": _lib.BSP_F32, "bf16": _lib.BSP_BF16}
VALUE_BYTES = {"f64": 8, "f32": 4, "bf16": 2}
PRECISIONS = {"f64": _lib.PREC_F64, "f32": _lib.PREC_F32, "bf16": _lib.PREC_BF16}


def listed() -> list[dict]:
    return [
        # the smallest solve: a coarse 2D problem with B = 2, D = 1, the block
        # size the reference's notes call the fastest; launches and latency
        {"name": "solve_pcg_2d_24x20_bs2", "op": "solve", "method": "pcg", "nx": 24, "ny": 20, "nz": 1, "bs": 2,
         "skew": 0.0, "tol": 1e-10, "precision": "f64"},
        # 2D SPD diffusion, 4x4 blocks: IChol0_pCG at the size of the first configuration
        {"name": "solve_pcg_2d_64x64_bs4", "op": "solve", "method": "pcg", "nx": 64, "ny": 64, "nz": 1, "bs": 4,
         "skew": 0.0, "tol": 1e-10, "precision": "f64"},
        # 3D nonsymmetric, 8x8 blocks: ILU0_pGMRES(30, k = 10), the benchmark's headline solve
        {"name": "solve_gmres_3d_64_bs8", "op": "solve", "method": "gmres", "nx": 64, "ny": 64, "nz": 64, "bs": 8,
         "skew": 0.3, "tol": 1e-10, "precision": "f64"},
        # 16x16 blocks, factors and inner operator stored in FP32 inside FP64 refinement, uneven sides
        {"name": "solve_gmres_f32_3d_44x40x36_bs16", "op": "solve", "method": "gmres", "nx": 44, "ny": 40, "nz": 36,
         "bs": 16, "skew": 0.3, "tol": 1e-10, "precision": "f32"},
        # T = std::complex<double>: ILU0_pGMRES(30, k = 10) on complex 4x4 blocks
        {"name": "solve_complex_3d_32_bs4", "op": "solve", "method": "complex", "nx": 32, "ny": 32, "nz": 32, "bs": 4,
         "skew": 0.3, "tol": 1e-10, "precision": "f64"},
        # many small SPD systems at once: uneven 2D sides, 4x4 and 8x8 blocks, 4 right-hand sides
        {"name": "batch_16_systems_4rhs", "op": "batch", "count": 16, "lo": 32, "hi": 160, "nrhs": 4, "tol": 1e-10},
        # the two triangular sweeps of an ILU0 application at the headline size
        {"name": "apply_ilu0_3d_64_bs8", "op": "apply", "kind": "ilu0", "nx": 64, "ny": 64, "nz": 64, "bs": 8,
         "skew": 0.3},
        # block IChol0 on a long thin wavefront (2D, odd side)
        {"name": "apply_ichol0_2d_300x257_bs4", "op": "apply", "kind": "ichol0", "nx": 300, "ny": 257, "nz": 1,
         "bs": 4, "skew": 0.0},
        # symmetric block SOR with the packaged defaults (w = 1.6, nu = 3): six sweeps
        {"name": "apply_sor_3d_40x36x44_bs4", "op": "apply", "kind": "sor", "nx": 40, "ny": 36, "nz": 44, "bs": 4,
         "skew": 0.0},
        # the matrix product of the headline size
        {"name": "bsmv_3d_64_bs8", "op": "bsmv", "nx": 64, "ny": 64, "nz": 64, "bs": 8, "skew": 0.3, "nrhs": 1,
         "dtype": "f64", "transpose": False, "accumulate": False},
        # an odd block size (linear triangles), two right-hand sides, accumulating into b
        {"name": "bsmv_2d_250x201_bs3_2rhs", "op": "bsmv", "nx": 250, "ny": 201, "nz": 1, "bs": 3, "skew": 0.0,
         "nrhs": 2, "dtype": "f64", "transpose": False, "accumulate": True},
        # the transposed product in FP32, 4 right-hand sides, 16x16 blocks
        {"name": "bsmv_t_f32_3d_28_bs16_4rhs", "op": "bsmv", "nx": 28, "ny": 28, "nz": 28, "bs": 16, "skew": 0.3,
         "nrhs": 4, "dtype": "f32", "transpose": True, "accumulate": False},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, bs: int, max_values: int, flat: bool, max_side: int = 1000) -> dict:
    """Uneven sides, 2D or 3D, with at most max_values stored values."""
    nd = 2 if flat else 3
    most = max_values / (bs * bs * (2 * nd + 1))
    hi = min(max_side, max(6, int(most ** (1.0 / nd))))
    lo = 4 if nd == 3 else 8
    mid = _log_int(rng, min(lo, hi), hi)
    side = [max(3, min(hi, int(round(mid * rng.uniform(0.75, 1.25))))) for _ in range(nd)]
    return {"nx": side[0], "ny": side[1], "nz": side[2] if nd == 3 else 1}


def draw(rng) -> dict:
    op = rng.choice(["solve", "solve", "apply", "apply", "bsmv", "bsmv", "batch"])
    if op == "bsmv":
        dtype = rng.choice(["f64", "f64", "f32", "bf16"])
        bs = rng.choice([1, 2, 3, 4, 5, 8, 16, 32] if dtype == "f64" else [4, 8, 16])
        flat = rng.random() < 0.5
        return {"op": op, **_grid(rng, bs, 90_000_000, flat), "bs": bs, "skew": 0.0 if flat else 0.3,
                "nrhs": rng.choice([1, 1, 2, 3, 4, 5]), "dtype": dtype, "transpose": rng.random() < 0.3,
                "accumulate": rng.random() < 0.4}
    if op == "apply":
        kind = rng.choice(["ilu0", "ilu0", "ichol0", "sor", "diag"])
        bs = rng.choice([1, 2, 3, 4, 4, 8, 8, 16])
        flat = rng.random() < 0.5
        most = 90_000_000 if bs > 3 else 4_000_000
        return {"op": op, "kind": kind, **_grid(rng, bs, most, flat), "bs": bs,
                "skew": 0.3 if kind == "ilu0" and not flat else 0.0}
    if op == "batch":
        lo = rng.choice([16, 32])
        return {"op": op, "count": _log_int(rng, 2, 16), "lo": lo, "hi": _log_int(rng, 2 * lo, 144),
                "nrhs": rng.choice([1, 2, 4]), "tol": 1e-10}
    method = rng.choice(["pcg", "pcg", "gmres", "gmres", "complex"])
    if method == "pcg":
        bs, flat = rng.choice([2, 3, 4, 8]), rng.random() < 0.7
        return {"op": op, "method": method, **_grid(rng, bs, 1_500_000, flat, 90), "bs": bs, "skew": 0.0,
                "tol": 1e-10, "precision": "f64"}
    if method == "complex":
        bs = rng.choice([1, 2, 4])
        return {"op": op, "method": method, **_grid(rng, bs, 3_000_000, False), "bs": bs, "skew": 0.3, "tol": 1e-10,
                "precision": "f64"}
    bs = rng.choice([4, 8, 8, 16])
    return {"op": op, "method": method, **_grid(rng, bs, 60_000_000, False), "bs": bs, "skew": 0.3, "tol": 1e-10,
            "precision": rng.choice(["f64", "f64", "f32"])}


# ---------------------------------------------------------------- systems

def _dims(case) -> tuple[int, ...]:
    return (case["nx"], case["ny"]) if case["nz"] == 1 else (case["nx"], case["ny"], case["nz"])


def _structure(dims):
    """Block CSR structure of the stencil, columns ascending in a row: row_ptr,
    col_idx, the position of every (row, slot) (-1: none) and the coordinates.
    Slots: -axis for the last axis to the first, the row itself, +axis for the
    first to the last."""
    nd, n = len(dims), math.prod(dims)
    idx = torch.arange(n, device=DEV)
    coords, stride, s = [], [], 1
    for d in dims:
        coords.append((idx // s) % d)
        stride.append(s)
        s *= d
    cols, mask = [], []
    for ax in reversed(range(nd)):
        cols.append(idx - stride[ax])
        mask.append(coords[ax] > 0)
    cols.append(idx)
    mask.append(torch.ones_like(mask[0]))
    for ax in range(nd):
        cols.append(idx + stride[ax])
        mask.append(coords[ax] < dims[ax] - 1)
    cols, mask = torch.stack(cols, 1), torch.stack(mask, 1)
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row_ptr[1:] = mask.sum(1).cumsum(0)
    pos = torch.where(mask, row_ptr[:-1, None] + mask.cumsum(1) - 1, -1)
    return row_ptr, cols[mask], pos, coords, stride


def _system(dims, bs: int, seed: int, skew: float, nrhs: int = 1):
    """Device arrays of one seeded system: row_ptr, col_idx, vals, b, pos, coords, stride."""
    nd, n = len(dims), math.prod(dims)
    gen = torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))
    row_ptr, col_idx, pos, coords, stride = _structure(dims)
    vals = torch.empty(col_idx.numel(), bs, bs, dtype=torch.float64, device=DEV)
    eye = torch.eye(bs, dtype=torch.float64, device=DEV)
    diag = (0.01 * eye).expand(n, bs, bs).clone()
    for ax in range(nd):
        p = torch.nonzero(coords[ax] < dims[ax] - 1).flatten()
        q = p + stride[ax]
        g = torch.randn(p.numel(), bs, bs, dtype=torch.float64, device=DEV, generator=gen)
        k = g @ g.transpose(1, 2) + 0.1 * eye
        off = -k
        if skew:
            w = torch.randn(p.numel(), bs, bs, dtype=torch.float64, device=DEV, generator=gen)
            off = off + skew * (w - w.transpose(1, 2))
        diag[p] += k
        diag[q] += k
        vals[pos[p, nd + 1 + ax]] = off
        vals[pos[q, nd - 1 - ax]] = off
    vals[pos[:, nd]] = diag
    b = 2.0 * torch.rand(n * nrhs * bs, dtype=torch.float64, device=DEV, generator=gen) - 1.0
    return SimpleNamespace(dims=dims, bs=bs, n=n, row_ptr=row_ptr, col_idx=col_idx, vals=vals, b=b, pos=pos,
                           coords=coords, stride=stride)


def _complex_system(dims, bs: int, seed: int, skew: float):
    re, im = _system(dims, bs, seed, skew), _system(dims, bs, seed + 7919, skew)
    re.vals = torch.complex(re.vals, 0.3 * im.vals)
    re.b = torch.complex(re.b, im.b)
    return re


def _batch_specs(case, seed: int):
    """(side, bs, seed) per system: sides spread evenly over the logarithm of
    [lo, hi], block sizes 4 and 8 in turn, so that every seed is the same work."""
    m = case["count"]
    return [(int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / m))), 8 if i % 3 == 2 else 4,
             seed * 1009 + i) for i in range(m)]


def _host(t, dtype=None):
    t = t if dtype is None else t.to(dtype)
    return t.cpu().numpy()


def _matrix(s):
    args = (_host(s.row_ptr, torch.int32), _host(s.col_idx, torch.int32), _host(s.vals))
    return bsp.Matrix.from_complex(*args) if s.vals.is_complex() else bsp.Matrix(*args, bs=s.bs)


# ---------------------------------------------------------------- the four calls

def prepare(case, seed: int) -> dict:
    op = case["op"]
    if op == "batch":
        sys_, bs_ = [], []
        for side, bs, sd in _batch_specs(case, seed):
            s = _system((side, side), bs, sd, 0.0, case["nrhs"])
            sys_.append(SimpleNamespace(row_ptr=_host(s.row_ptr, torch.int32), col_idx=_host(s.col_idx, torch.int32),
                                        vals=_host(s.vals), bs=bs))
            bs_.append(s.b)
        return {"case": case, "batch": bsp.Batch(sys_), "b": torch.cat(bs_)}
    if op == "solve" and case["method"] == "complex":
        s = _complex_system(_dims(case), case["bs"], seed, case["skew"])
        return {"case": case, "A": _matrix(s), "b": torch.view_as_real(s.b).reshape(-1).contiguous()}
    s = _system(_dims(case), case["bs"], seed, case["skew"], case.get("nrhs", 1))
    state = {"case": case, "A": _matrix(s), "b": s.b}
    if op == "apply":
        A, kind = state["A"], case["kind"]
        state["pc"] = {"ilu0": bsp.ILU0, "ichol0": bsp.IChol0, "diag": bsp.Diag}[kind](A) if kind != "sor" \
            else bsp.SOR(A, 1.6, 3, 0)
        state["r"] = torch.empty_like(s.b)
    elif op == "bsmv":
        if case["dtype"] != "f64":
            state["A"].make_lowp(DTYPES[case["dtype"]])
            state["b"] = s.b.float()
        state["y"] = torch.empty_like(state["b"])
        state["z"] = state["b"].flip(0).contiguous() if case["accumulate"] else None
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "bsmv":
        bsp.bsmv_dev(state["A"], state["b"], state["y"], nrhs=case["nrhs"], transpose=case["transpose"],
                     beta=1.0 if case["accumulate"] else 0.0, z=state["z"], dtype=DTYPES[case["dtype"]])
        return state["y"]
    if op == "apply":
        r = state["r"].copy_(state["b"])
        state["pc"](r)
        return r
    if op == "batch":
        x, _ = state["batch"].pcg(state["b"], case["nrhs"], tol=case["tol"])
        return x
    A, b, tol = state["A"], state["b"], case["tol"]
    if case["method"] == "pcg":
        return bsp.IChol0_pCG(A, tol).solve(A, b)
    if case["precision"] == "f64":
        return bsp.ILU0_pGMRES(A, tol, 5000, 30, 10).solve(A, b)
    return bsp.pGMRES(A, b, tol, bsp.ILU0(A), 5000, 30, 10, stop_rule=_lib.STOP_TRUE_RESIDUAL,
                      precision=PRECISIONS[case["precision"]])


# ---------------------------------------------------------------- work

def _counts(dims):
    n = math.prod(dims)
    return n, n + sum(2 * n // d * (d - 1) for d in dims)


def _apply_work(n, nnzb, bs, kind, rhs: int = 1, value_bytes: int = 8):
    """Bytes and flops of one application: the swept blocks once per use of
    them, the inverted diagonal blocks, r read and z written."""
    b2, off = bs * bs, nnzb - n
    blocks = {"ilu0": off + n, "ichol0": off / 2 + n, "sor": off + n, "diag": n}[kind]
    muls = {"ilu0": off + n, "ichol0": off + 2 * n, "sor": 6 * (off + n), "diag": n}[kind]
    return blocks * b2 * value_bytes + 16.0 * n * bs * rhs, 2.0 * muls * b2 * rhs


def _pcg_iterations(side, bs):
    """Iterations that the 2D systems take to 1e-10, fitted to sides of 24 to 152."""
    return (140 + 0.5 * side) * math.sqrt(bs / 4)


def work(case) -> dict:
    """One pass over what is read and written.  A solve reads the matrix and the
    preconditioner's factors once in every iteration (the larger ones exceed
    the caches), with the number of iterations that these systems take."""
    op = case["op"]
    if op == "batch":
        by = fl = 0.0
        for side, bs, _ in _batch_specs(case, 0):
            n, nnzb = _counts((side, side))
            pb, pf = _apply_work(n, nnzb, bs, "ichol0", case["nrhs"])
            its = _pcg_iterations(side, bs)
            by += its * (pb + nnzb * (bs * bs * 8 + 4) + 72.0 * n * bs * case["nrhs"])
            fl += its * (pf + 2.0 * nnzb * bs * bs * case["nrhs"] + 12.0 * n * bs * case["nrhs"])
        return {"bytes": by, "flops": fl}
    dims, bs = _dims(case), case["bs"]
    n, nnzb = _counts(dims)
    if op == "bsmv":
        vb, xb = VALUE_BYTES[case["dtype"]], 8 if case["dtype"] == "f64" else 4
        vecs = 3 if case["accumulate"] else 2
        return {"bytes": nnzb * (bs * bs * vb + 4.0) + 4.0 * n + vecs * float(n * bs * case["nrhs"]) * xb,
                "flops": 2.0 * nnzb * bs * bs * case["nrhs"]}
    if op == "apply":
        by, fl = _apply_work(n, nnzb, bs, case["kind"])
        return {"bytes": by, "flops": fl}
    cplx = case["method"] == "complex"
    vb, mul = (16, 4) if cplx else (VALUE_BYTES[case["precision"]], 1)
    if case["method"] == "pcg":
        its, kind, vecs = _pcg_iterations(max(dims), bs), "ichol0", 9
    else:
        its, kind, vecs = 23.0 * math.sqrt(2 * bs if cplx else bs), "ilu0", 20  # the basis so far, on average
    pb, pf = _apply_work(n, nnzb, bs, kind, 1, vb)
    xb = 16.0 if cplx else 8.0
    return {"bytes": its * (pb + nnzb * (bs * bs * vb + 4.0) + vecs * n * bs * xb),
            "flops": mul * its * (pf + 2.0 * nnzb * bs * bs + 2.0 * vecs * n * bs)}


# ---------------------------------------------------------------- exact values

def _levels(s):
    """Rows grouped by the sum of their coordinates: a row's neighbours are in
    the level before or after, so natural order visits the levels in turn."""
    lev = sum(s.coords)
    order = torch.argsort(lev, stable=True)
    return torch.split(order, torch.bincount(lev).tolist())


def _neighbours(s, rows, sign: int):
    """(rows that have it, the neighbour, the block position) per axis."""
    nd = len(s.dims)
    for ax in range(nd):
        p = s.pos[rows, nd + 1 + ax if sign > 0 else nd - 1 - ax]
        has = p >= 0
        if bool(has.any()):
            r = rows[has]
            yield r, r + sign * s.stride[ax], p[has]


def _mv(blocks, x):
    return torch.bmm(blocks, x.unsqueeze(2)).squeeze(2)


def _exact_apply(s, kind: str):
    nd, bs = len(s.dims), s.bs
    b = s.b.view(s.n, bs)
    d = s.vals[s.pos[:, nd]].clone()
    if kind == "diag":
        return torch.linalg.solve(d, b.unsqueeze(2)).reshape(-1)
    levels = _levels(s)
    if kind == "sor":
        x = torch.zeros_like(b)
        for sweep in range(6):
            for rows in (levels if sweep < 3 else reversed(levels)):
                t = b[rows].clone()
                at = torch.empty(s.n, dtype=torch.int64, device=DEV)
                at[rows] = torch.arange(rows.numel(), device=DEV)
                for sign in (-1, 1):
                    for r, j, p in _neighbours(s, rows, sign):
                        t[at[r]] -= _mv(s.vals[p], x[j])
                new = torch.linalg.solve(d[rows], t.unsqueeze(2)).squeeze(2)
                x[rows] += 1.6 * (new - x[rows])
        return x.reshape(-1)
    # block ILU(0) (and IChol0, the same operator on a symmetric matrix) of a
    # stencil without triangles: only the diagonal blocks change
    dinv = torch.empty_like(d)
    y, u = b.clone(), torch.empty_like(b)
    for rows in levels:
        for r, j, p in _neighbours(s, rows, -1):
            # block (j, r) of the row below: its + slot along the same axis
            ax = s.stride.index(int(r[0] - j[0]))
            d[r] -= s.vals[p] @ dinv[j] @ s.vals[s.pos[j, nd + 1 + ax]]
            y[r] -= _mv(s.vals[p], u[j])
        dinv[rows] = torch.linalg.inv(d[rows])
        u[rows] = _mv(dinv[rows], y[rows])
    z = torch.zeros_like(b)
    for rows in reversed(levels):
        t = y[rows].clone()
        at = torch.empty(s.n, dtype=torch.int64, device=DEV)
        at[rows] = torch.arange(rows.numel(), device=DEV)
        for r, j, p in _neighbours(s, rows, 1):
            t[at[r]] -= _mv(s.vals[p], z[j])
        z[rows] = _mv(dinv[rows], t)
    return z.reshape(-1)


def _exact_bsmv(s, case):
    bs, nrhs = s.bs, case["nrhs"]
    rows = torch.repeat_interleave(torch.arange(s.n, device=DEV), s.row_ptr.diff())
    src, dst, blocks = s.col_idx, rows, s.vals
    if case["transpose"]:
        src, dst, blocks = rows, s.col_idx, s.vals.transpose(1, 2)
    x = s.b.view(s.n, nrhs, bs)
    y = torch.zeros_like(x)
    step = max(1, (1 << 26) // (bs * bs))
    for k in range(0, src.numel(), step):
        t = torch.bmm(x[src[k:k + step]], blocks[k:k + step].transpose(1, 2))
        y.index_add_(0, dst[k:k + step], t)
    y = y.reshape(-1)
    return y + s.b.flip(0) if case["accumulate"] else y


def _exact_2d(s, nrhs: int = 1):
    """A x = b on a 2D grid by block elimination over the grid lines."""
    (nx, ny), bs = s.dims, s.bs
    m = nx * bs
    b = s.b.view(s.n, nrhs, bs).transpose(1, 2).reshape(ny, m, nrhs)

    def line(j, slots):
        out = torch.zeros(nx, bs, nx, bs, dtype=s.vals.dtype, device=DEV)
        rows = torch.arange(nx, device=DEV) + j * nx
        for slot, shift in slots:
            p = s.pos[rows, slot]
            i = torch.nonzero(p >= 0).flatten()
            out[i, :, i + shift, :] = s.vals[p[i]]
        return out.view(m, m)

    kept, c = [], b.clone()
    for j in range(ny):
        d = line(j, ((1, -1), (2, 0), (3, 1)))
        if j:
            low, up = line(j, ((0, 0),)), line(j - 1, ((4, 0),))
            t = torch.linalg.lu_solve(*kept[-1], torch.cat([up, c[j - 1]], 1))
            d -= low @ t[:, :m]
            c[j] -= low @ t[:, m:]
        kept.append(torch.linalg.lu_factor(d))
    x = torch.empty_like(c)
    for j in reversed(range(ny)):
        t = c[j] if j == ny - 1 else c[j] - line(j, ((4, 0),)) @ x[j + 1]
        x[j] = torch.linalg.lu_solve(*kept[j], t)
    return x.view(s.n, bs, nrhs).transpose(1, 2).reshape(-1)


def _exact_dense(s):
    bs = s.bs
    a = torch.zeros(s.n, s.n, bs, bs, dtype=s.vals.dtype, device=DEV)
    rows = torch.repeat_interleave(torch.arange(s.n, device=DEV), s.row_ptr.diff())
    a[rows, s.col_idx] = s.vals
    return torch.linalg.solve(a.transpose(1, 2).reshape(s.n * bs, s.n * bs), s.b)


def exact(case, seed: int):
    op = case["op"]
    if op == "batch":
        return torch.cat([_exact_2d(_system((side, side), bs, sd, 0.0, case["nrhs"]), case["nrhs"])
                          for side, bs, sd in _batch_specs(case, seed)])
    dims, bs = _dims(case), case["bs"]
    if op == "solve":
        if case["nz"] > 1 and math.prod(dims) * bs > 10_000:
            return None  # no direct solve in reasonable time
        if case["method"] == "complex":
            return torch.view_as_real(_exact_dense(_complex_system(dims, bs, seed, case["skew"]))).reshape(-1)
        s = _system(dims, bs, seed, case["skew"])
        return _exact_2d(s) if len(dims) == 2 else _exact_dense(s)
    s = _system(dims, bs, seed, case["skew"], case.get("nrhs", 1))
    return _exact_bsmv(s, case) if op == "bsmv" else _exact_apply(s, case["kind"])
