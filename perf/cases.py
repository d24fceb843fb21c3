"""Measured cases of the numeric factorize + solve phase.

Each case is a sparse symmetric system of one of the five workload families
(sylver_gb300/workloads.py) that a program analyses once and then factorizes
and solves again and again with new values and right-hand sides: a time step,
a Newton or interior-point iteration, a parameter sweep.  One pass is either

  op = "factor"  new values: one numeric factorization and one solve;
  op = "solve"   one more solve with a factorization that is already there.

prec "fp64" is the reference's only precision and the default of
spldlt_factorize (no refinement); "fp32" is FP32 factors with FP64 iterative
refinement to a scaled backward error of 1e-14.  device = True passes values
and right-hand sides that are already in HBM (spldlt_factorize_device /
spldlt_solve_device); otherwise host arrays go through the C-ABI, as in the
reference.

Right-hand sides are b = A x_true with a random x_true, so exact() knows the
solution without solving anything.
"""
import ctypes
import math

import numpy as np
import torch

import sylver_gb300 as sg
from sylver_gb300 import workloads as w


def _case(name, family, dims, prec, nrhs, op="factor", device=False):
    d = {"family": family, "nx": dims[0], "ny": dims[1], "nz": dims[2], "prec": prec,
         "nrhs": nrhs, "op": op, "device": device}
    return dict(d, name=name) if name else d


def listed():
    return [
        # the smallest call: the 12 x 12 grid of the golden tests, where launches and latency count
        _case("grid2d_12_fp64", "grid2d", (12, 12, 1), "fp64", 1),
        # 2D 5-point SPD 100 x 100, one right-hand side: the reference user's default call
        _case("grid2d_100_fp64", "grid2d", (100, 100, 1), "fp64", 1),
        # a larger 2D problem with odd sides in mixed precision
        _case("grid2d_401x333_fp32", "grid2d", (401, 333, 1), "fp32", 1),
        # an ordinary 3D problem with ragged sides and a few right-hand sides
        _case("box3d_33x29x31_fp64", "box3d", (33, 29, 31), "fp64", 3),
        # a large 3D problem in the reference's precision, inputs in HBM
        _case("box3d_56_fp64", "box3d", (56, 56, 56), "fp64", 1, device=True),
        # the headline benchmark: 27-point log-normal 80^3, 16 right-hand sides
        _case("box3d_80_fp32", "box3d", (80, 80, 80), "fp32", 16, device=True),
        # many solves per factorization: one refined right-hand side at a time
        _case("box3d_64_fp32_solve", "box3d", (64, 64, 64), "fp32", 1, op="solve", device=True),
        # a block of right-hand sides (not a multiple of a tile) in FP64
        _case("box3d_40_fp64_solve", "box3d", (40, 40, 40), "fp64", 17, op="solve"),
        # indefinite 7-point 48^3 - sigma I, 4 right-hand sides (Helmholtz-like), mixed precision
        _case("shift3d_48_fp32", "shift3d", (48, 48, 48), "fp32", 4, device=True),
        # indefinite with ragged sides in the reference's precision
        _case("shift3d_27x24x21_fp64", "shift3d", (27, 24, 21), "fp64", 1),
        # many small independent systems in one call (nx: instances, sides 8..64)
        _case("batch2d_500_fp32", "batch2d", (500, 1, 1), "fp32", 1),
        # saddle point with the matching-based ordering and its scaling, delayed pivots
        _case("kkt_14_fp64", "kkt", (14, 14, 14), "fp64", 1),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["grid2d", "grid2d", "box3d", "box3d", "box3d", "shift3d", "shift3d",
                         "batch2d", "kkt"])
    prec = rng.choice(["fp64", "fp32"])
    nrhs = logint(1, 24)
    op = rng.choice(["factor", "factor", "solve"])
    device = rng.random() < 0.5
    if family == "batch2d":
        return _case(None, family, (logint(20, 500), 1, 1), prec, 1, op, device)
    if family == "kkt":
        k = logint(5, 14)
        return _case(None, family, (k, k, k), prec, min(nrhs, 4), op, device)
    if family == "grid2d":
        s = logint(8, 360)
        return _case(None, family, (s, max(4, int(s * rng.uniform(0.6, 1.2))), 1), prec, nrhs, op,
                     device)
    top = {("box3d", "fp32"): 72, ("box3d", "fp64"): 50, ("shift3d", "fp32"): 44,
           ("shift3d", "fp64"): 34}[family, prec]
    s = logint(8, top)
    dims = tuple(max(5, int(round(s * rng.uniform(0.85, 1.1)))) for _ in range(3))
    return _case(None, family, dims, prec, nrhs, op, device)


# ---------------------------------------------------------------------------
# matrices: lower triangle by columns, rows increasing; a column's first
# entry is its diagonal

class _Grid:
    """Pattern of a grid stencil: the edge from node j to node j + stride[o]
    exists where mask[j, o]; edges are numbered by (j, o)."""

    def __init__(self, dims, box):
        nx, ny, nz = dims
        offs = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
                if (dz, dy, dx) > (0, 0, 0) and (box or abs(dx) + abs(dy) + abs(dz) == 1)]
        self.offs = offs
        self.dims = dims
        n = nx * ny * nz
        ix = np.arange(n) % nx
        iy = np.arange(n) // nx % ny
        iz = np.arange(n) // (nx * ny)
        self.mask = np.stack([(ix + dx >= 0) & (ix + dx < nx) & (iy + dy >= 0) & (iy + dy < ny) &
                              (iz + dz >= 0) & (iz + dz < nz) for dx, dy, dz in offs], axis=1)
        self.stride = np.array([dx + nx * (dy + ny * dz) for dx, dy, dz in offs])
        self.n = n
        src, o = np.nonzero(self.mask)
        self.src, self.dst = src, src + self.stride[o]
        cnt = self.mask.sum(axis=1)
        self.ptr = np.concatenate([[0], np.cumsum(cnt + 1)]).astype(np.int64)
        self.epos = np.arange(src.size) + src + 1
        row = np.empty(self.ptr[-1], dtype=np.int32)
        row[self.ptr[:-1]] = np.arange(n)
        row[self.epos] = self.dst
        self.row = row
        full = 26 if box else 2 * sum(d > 1 for d in dims)
        self.missing = full - (cnt + np.bincount(self.dst, minlength=n))

    def laplacian(self, weights, shift):
        """Weighted Laplacian (weights None: ones), ghost edges of weight 1,
        plus shift * I; the diagonal and the values by column."""
        wt = np.ones(self.src.size) if weights is None else weights
        diag = (np.bincount(self.src, wt, self.n) + np.bincount(self.dst, wt, self.n) +
                self.missing)
        diag = diag + (shift(diag) if callable(shift) else shift)
        val = np.empty(self.row.size)
        val[self.ptr[:-1]] = diag
        val[self.epos] = -wt
        return val


def _times(n, ptr, row, val, x):
    """A x in a fixed order of additions (x: n x nrhs)."""
    col = np.repeat(np.arange(n), np.diff(ptr))
    off = row != col
    r, c, v = row[off], col[off], val[off]
    y = val[ptr[:-1], None] * x
    for q in range(x.shape[1]):
        y[:, q] += np.bincount(r, v * x[c, q], n) + np.bincount(c, v * x[r, q], n)
    return y


class _Pattern:
    """What a program keeps over all factorizations of one sparsity pattern:
    the pattern and its analysis."""

    def __init__(self, case):
        fam = case["family"]
        dims = (case["nx"], case["ny"], case["nz"])
        self.options = sg.default_options()
        val0 = None
        if fam == "batch2d":
            sides = np.random.default_rng(4).integers(8, 65, size=dims[0])
            self.grids = [_Grid((int(s), int(s), 1), False) for s in sides]
            base = np.concatenate([[0], np.cumsum([g.n for g in self.grids])])
            nnz = np.concatenate([[0], np.cumsum([g.row.size for g in self.grids])])
            self.n = int(base[-1])
            self.ptr = np.concatenate([g.ptr[:-1] + nnz[i] for i, g in enumerate(self.grids)] +
                                      [nnz[-1:]])
            self.row = np.concatenate([g.row + base[i] for i, g in enumerate(self.grids)])
            order = np.concatenate([w.grid_nested_dissection((int(s), int(s))) + base[i]
                                    for i, s in enumerate(sides)])
        elif fam == "kkt":
            g = self.grid = _Grid(dims, False)
            m = g.n // 4
            rng = np.random.default_rng(5)
            cols = np.stack([rng.choice(g.n, size=4, replace=False) for _ in range(m)])
            self.m, self.n = m, g.n + m
            # column j: H's entries, then the rows of B that hold column j
            brow, bcol = np.repeat(np.arange(m), 4) + g.n, cols.ravel()
            r = np.concatenate([g.row, brow, np.arange(g.n, self.n)])
            c = np.concatenate([np.repeat(np.arange(g.n), np.diff(g.ptr)), bcol,
                                np.arange(g.n, self.n)])
            self.perm = np.lexsort((r, c))
            self.row = r[self.perm].astype(np.int32)
            self.ptr = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=self.n))])
            order = None
            self.options.ordering = 2
            self.options.scaling = 3
            val0 = self.values(case, np.random.default_rng(6))
        else:
            g = self.grid = _Grid(dims, fam == "box3d")
            self.n, self.ptr, self.row = g.n, g.ptr, g.row
            order = w.grid_nested_dissection(dims if dims[2] > 1 else dims[:2])
            if fam == "shift3d":
                e = [2.0 - 2.0 * np.cos(np.arange(1, k + 1) * np.pi / (k + 1)) for k in dims]
                lam = np.sort((e[0][:, None, None] + e[1][None, :, None] + e[2]).ravel())
                # the widest gap of the spectrum near its 5 % quantile
                lo, hi = int(0.04 * lam.size), max(int(0.06 * lam.size), int(0.04 * lam.size) + 2)
                k = lo + int(np.argmax(lam[lo + 1:hi + 1] - lam[lo:hi]))
                self.gap = (lam[k], lam[k + 1])
        self.analysis = sg.Analysis(self.n, self.ptr + 1, self.row.astype(np.int32) + 1,
                                    order=order, options=self.options, val=val0)
        assert self.analysis.flag >= 0, self.analysis.flag

    def values(self, case, rng):
        fam = case["family"]
        if fam == "box3d":  # log-normal edge weights, a small diagonal shift
            g = self.grid
            return g.laplacian(np.exp(rng.standard_normal(g.src.size)), lambda d: 1e-3 * d.min())
        if fam == "grid2d":  # implicit time step: Laplacian plus a mass term
            return self.grid.laplacian(None, rng.uniform(0.1, 1.0))
        if fam == "shift3d":
            return self.grid.laplacian(None, -(self.gap[0] + rng.uniform(0.4, 0.6) *
                                               (self.gap[1] - self.gap[0])))
        if fam == "batch2d":
            return np.concatenate([g.laplacian(None, rng.uniform(0.1, 1.0)) for g in self.grids])
        v = np.concatenate([self.grid.laplacian(None, 0.0), rng.standard_normal(4 * self.m),
                            np.full(self.m, -1e-8)])
        return v[self.perm]


_patterns = {}


def _pattern(case):
    # one pattern at a time: a program works on its own, not on every case's
    key = (case["family"], case["nx"], case["ny"], case["nz"])
    if key not in _patterns:
        _patterns.clear()
        _patterns[key] = _Pattern(case)
    return _patterns[key]


def _x_true(case, n, seed):
    return np.random.default_rng([seed, 1]).uniform(-1.0, 1.0, size=(n, case["nrhs"]))


def prepare(case, seed):
    pat = _pattern(case)
    posdef = case["family"] in ("grid2d", "box3d", "batch2d")
    val = pat.values(case, np.random.default_rng([seed, 0]))
    b = _times(pat.n, pat.ptr, pat.row, val, _x_true(case, pat.n, seed))
    s = {"case": case, "pat": pat, "posdef": posdef, "val": val, "b": np.asfortranarray(b)}
    s["prec"], s["maxit"] = (sg.FP32, 20) if case["prec"] == "fp32" else (sg.FP64, 0)
    # the handle a program holds from its first factorization on
    s["factor"] = sg.Factor(pat.analysis, posdef, val, precision=s["prec"], ir_tol=1e-14,
                            ir_max_iter=s["maxit"], options=pat.options)
    assert s["factor"].flag >= 0, s["factor"].flag
    if case["device"]:
        s["stream"] = torch.cuda.ExternalStream(sg.load().sylver_gb300_stream())
        s["val_d"] = torch.from_numpy(val).cuda()
        s["b_d"] = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()  # column-major n x nrhs
        s["x_d"] = torch.empty_like(s["b_d"])
    return s


def run(s):
    f, pat = s["factor"], s["pat"]
    out = {}
    if s["case"]["device"]:
        lib, P = sg.load(), ctypes.c_void_p
        if s["case"]["op"] == "factor":
            lib.spldlt_factorize_device(s["posdef"], P(s["val_d"].data_ptr()), pat.analysis.akeep,
                                        ctypes.byref(f.fkeep), ctypes.byref(pat.options),
                                        ctypes.byref(f.inform), s["prec"], 1e-14, s["maxit"])
        inf = sg.Inform()
        with torch.cuda.stream(s["stream"]):
            s["x_d"].copy_(s["b_d"])
        lib.spldlt_solve_device(0, s["case"]["nrhs"], P(s["x_d"].data_ptr()), pat.n,
                                pat.analysis.akeep, f.fkeep, ctypes.byref(pat.options),
                                ctypes.byref(inf))
        out["x"], out["solve_flag"] = s["x_d"], inf.flag
    else:
        if s["case"]["op"] == "factor":
            f.refactor(s["val"], precision=s["prec"], ir_tol=1e-14, ir_max_iter=s["maxit"])
        out["x"] = f.solve(s["b"])
        out["solve_flag"] = f.solve_inform.flag
    if s["case"]["op"] == "factor":
        out["flag"], out["rank"], out["num_neg"] = (f.inform.flag, f.inform.matrix_rank,
                                                    f.inform.num_neg)
    return out


def work(case):
    """Factor flops (mul + add, from the analysis), the solve's two sweeps, the
    values, the right-hand sides and solution, and the factor moved once."""
    an = _pattern(case).analysis
    nnz, lnz, n, r = _pattern(case).row.size, an.inform.num_factor, _pattern(case).n, case["nrhs"]
    e = 4 if case["prec"] == "fp32" else 8
    factor = case["op"] == "factor"
    return {"bytes": e * lnz + 16 * n * r + (8 * nnz if factor else 0),
            "flops": 4.0 * lnz * r + (float(an.inform.num_flops) if factor else 0.0)}


def exact(case, seed):
    x = _x_true(case, _pattern_rows(case), seed)
    return {"x": np.ascontiguousarray(x.T) if case["device"] else np.asfortranarray(x),
            "solve_flag": None, "flag": None, "rank": None, "num_neg": None}


def _pattern_rows(case):
    if case["family"] == "batch2d":
        return int((np.random.default_rng(4).integers(8, 65, size=case["nx"]) ** 2).sum())
    n = case["nx"] * case["ny"] * case["nz"]
    return n + n // 4 if case["family"] == "kkt" else n
