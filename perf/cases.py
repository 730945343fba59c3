"""The solves this library is used for, as cases that can be timed and compared.

A case is one call of a public entry point: the reference's drop-in functions on device or
host arrays, the split set-up / start handle, DIA and DDM input, the mixed-precision,
double-double and learned solvers.  Every case solves A x = b to a tolerance, as a user's
program does, and returns the whole solution (and the residual history where the entry
point fills a caller's buffer).  Right-hand sides are N(0, 1); the matrices are the finite
difference stencils and the banded matrix of parcel_b.problems on any grid.

The library runs on the stream the inputs are made on (parcel_b_set_stream), so no pass has
to wait for the host between making x0 and solving.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parcel-legacy_b200"))

from parcel_b import _lib, api, ddm  # noqa: E402

SOLVERS = {"cg": 1, "bicgstab": 2, "gmres": 3, "cagmres": 4}
ITRMAX = 5000
PECLET, VELOCITY = 10.0, (1.0, 0.5, 0.25)
ANISO = (1.0, 1.0e-2, 1.0e-4)
BAND, BAND_NNZ, BAND_DIAG = 64, 9, 1.2
COARSEN, COARSE_STEPS = 8, 2


# ---- the cases ------------------------------------------------------------------------------
def _case(name, form, problem, solver, nx, ny, nz, rtol, precon=2, ilu=0, blocks=1, m=30, gs=1):
    return {"name": name, "form": form, "problem": problem, "solver": solver, "nx": nx, "ny": ny, "nz": nz,
            "rtol": rtol, "precon": precon, "ilu": ilu, "blocks": blocks, "m": m, "gs": gs}


def listed():
    return [
        # the smallest call: a C program relinked to the host-array shim on a toy grid
        _case("cg_host_16", "host", "poisson", "cg", 16, 16, 16, 1e-9, blocks=4),
        # a 2D Poisson solve: hundreds of short iterations, where launches and latency count
        _case("cg_jacobi_2d_256", "device", "poisson", "cg", 256, 256, 1, 1e-8, precon=1),
        # an implicit time step on a mid-sized odd grid: the factors kept, one new b per call
        _case("gmres_start_61x53x47", "handle", "convdiff", "gmres", 61, 53, 47, 1e-10, blocks=16),
        # the benchmark's solve: GMRES(30), block-Jacobi ILU(0) over 64 blocks
        _case("gmres_128", "device", "convdiff", "gmres", 128, 128, 128, 1e-10, blocks=64),
        # DIA input on a ragged grid, BiCGStab with D-ILU
        _case("bicgstab_dia_97x89x83", "dia", "convdiff", "bicgstab", 97, 89, 83, 1e-9, ilu=1, blocks=48),
        # the reference's CRS example: 160^3 Poisson, CG, D-ILU over 80 blocks (the largest)
        _case("cg_dilu_160", "device", "poisson", "cg", 160, 160, 160, 1e-9, ilu=1, blocks=80),
        # single-precision CG in a refinement loop to an FP64 residual of 1e-12
        _case("cg_mixed_aniso_128", "mixed", "aniso", "cg", 128, 128, 128, 1e-12, blocks=64),
        # communication-avoiding GMRES(8 x 8), Newton basis and TSQR, on 4M banded rows
        _case("cagmres_banded_4m", "device", "banded", "cagmres", 4000000, 1, 1, 1e-10, precon=1, m=64),
        # the reference's stencil-format example as its CUDA build runs it: 4^3 boxes
        _case("ddm_cubes_160", "ddm", "poisson", "cg", 160, 160, 160, 1e-9, ilu=1),
        # double-double CG and GMRES with D-ILU: solves whose residual double cannot resolve
        _case("ddcg_dilu_80", "dd", "poisson", "cg", 80, 80, 80, 1e-9, ilu=1, blocks=40),
        _case("ddgmres_64", "dd", "convdiff", "gmres", 64, 64, 64, 1e-10, ilu=1, blocks=32),
        # the two-level stage with the network in mixed-precision flexible GMRES
        _case("learned_vardiff_128", "learned", "vardiff", "gmres", 128, 128, 128, 1e-10, blocks=64, m=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(("host", "device", "device", "device", "handle", "handle", "dia", "mixed", "ddm", "dd", "dd"))
    if form == "device" and rng.random() < 0.25:
        n = _log(rng, 20000, 2000000) | 1
        return _drawn(rng, form, "banded", "cagmres", n, 1, 1, 1e-10, 1)
    if form in ("host", "device") and rng.random() < 0.3:
        nx, ny = _log(rng, 24, 400), _log(rng, 24, 400) | 1
        return _drawn(rng, form, "poisson", "cg", nx, ny, 1, 1e-8, rng.choice((0, 1)))
    top = {"host": 40, "device": 120, "handle": 100, "dia": 110, "mixed": 110, "ddm": 120, "dd": 56}[form]
    side = _log(rng, 12, top)
    nx, ny, nz = (max(8, int(side * rng.uniform(0.75, 1.0))) for _ in range(3))
    nx = nx | 1 if rng.random() < 0.5 else nx
    solver = rng.choice(("cg", "gmres") if form in ("mixed", "ddm") else ("cg", "bicgstab", "gmres"))
    if form == "ddm":
        problem = "poisson"
    elif solver == "cg":
        problem = rng.choice(("poisson", "aniso") if form != "dd" else ("poisson",))
    else:
        problem = "convdiff"
    rtol = 1e-12 if form == "mixed" else 1e-9
    precon = 1 if form in ("host", "device", "handle", "dia") and rng.random() < 0.25 else 2
    return _drawn(rng, form, problem, solver, nx, ny, nz, rtol, precon)


def _drawn(rng, form, problem, solver, nx, ny, nz, rtol, precon):
    n = nx * ny * nz
    blocks = max(2, min(96, n // rng.randint(2000, 20000) + 1))
    ilu = 1 if form in ("ddm", "dd") else rng.choice((0, 1))
    m = 64 if solver == "cagmres" else rng.choice((10, 20, 30, 40))
    gs = 2 if solver == "gmres" and rng.random() < 0.25 else 1
    c = _case("", form, problem, solver, nx, ny, nz, rtol, precon, ilu, blocks, m, gs)
    del c["name"]
    return c


# ---- the matrices -----------------------------------------------------------------------------
def _axes(case):
    """Per axis of a constant-coefficient stencil: (lower neighbour, half-diagonal, upper neighbour, cells)."""
    sizes = [case["nx"], case["ny"], case["nz"]]
    dims = 2 if sizes[2] == 1 else 3
    out = []
    for d in range(dims):
        if case["problem"] == "convdiff":
            c = PECLET * VELOCITY[d] / (max(sizes) + 1)
            out.append((-1.0 - c, 2.0 + c, -1.0, sizes[d]))
        else:
            k = ANISO[d] if case["problem"] == "aniso" else 1.0
            out.append((-k, 2.0 * k, -k, sizes[d]))
    return out


def _neighbours(case):
    """(offset, 1-based axis, direction) of the stencil points in column order, the centre among them."""
    nx, ny = case["nx"], case["ny"]
    dims = 2 if case["nz"] == 1 else 3
    step = [1, nx, nx * ny]
    return [(-step[d], d, -1) for d in reversed(range(dims))] + [(0, 0, 0)] + [(step[d], d, 1) for d in range(dims)]


def _faces(case, seed):
    """vardiff: the face coefficient towards every stencil neighbour, [z, y, x] per neighbour; k = exp(smooth noise)."""
    shape = (case["nz"], case["ny"], case["nx"])
    g = torch.Generator(device="cuda").manual_seed(1000 + seed)
    w = torch.fft.rfftn(torch.randn(shape, dtype=torch.float64, device="cuda", generator=g))
    kz, ky = (torch.fft.fftfreq(s, dtype=torch.float64, device="cuda") for s in shape[:2])
    kx = torch.fft.rfftfreq(shape[2], dtype=torch.float64, device="cuda")
    k2 = kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2
    f = torch.fft.irfftn(w * torch.exp(-((math.pi * 8.0) ** 2) * k2), s=shape)
    f = (f - f.mean()) * (math.sqrt(2.0) / f.std())
    k = torch.exp(f)
    p = torch.nn.functional.pad(k[None, None], (1,) * 6, mode="replicate")[0, 0]
    h = 1.0 / max(shape)
    out = {}
    for off, d, s in _neighbours(case):
        if s:
            sl = [slice(1, 1 + n) for n in shape]
            sl[2 - d] = slice(1 + s, 1 + s + shape[2 - d])
            out[off] = -h / (0.5 * (1.0 / k + 1.0 / p[tuple(sl)]))
    return out


def _stencil(case, seed):
    """[(offset, values over all cells, mask of the cells that have the neighbour)] in column order."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    i = torch.arange(n, device="cuda")
    at = [i % nx, (i // nx) % ny, i // (nx * ny)]
    size = [nx, ny, nz]
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    if case["problem"] == "vardiff":
        faces = _faces(case, seed)
        diag = -sum(f.reshape(-1) for f in faces.values())
    else:
        ax = _axes(case)
        diag = one * sum(a[1] for a in ax)
    out = []
    for off, d, s in _neighbours(case):
        if s == 0:
            out.append((0, diag, torch.ones(n, dtype=torch.bool, device="cuda")))
            continue
        mask = at[d] > 0 if s < 0 else at[d] < size[d] - 1
        v = faces[off].reshape(-1) if case["problem"] == "vardiff" else one * ax[d][0 if s < 0 else 2]
        out.append((off, v, mask))
    return out


def _banded(case, seed):
    """Random nonsymmetric band: the diagonal and 8 distinct offsets within +-64 per row, diagonal 1.2 x the row's absolute sum."""
    n, k = case["nx"], BAND_NNZ - 1
    g = torch.Generator(device="cuda").manual_seed(2000 + seed)
    # 8 distinct strata of the 128 offsets -64..-1, 1..64, one drawn from each, mirrored at the ends
    o = torch.randint(0, 2 * BAND // k, (n, k), device="cuda", generator=g)
    o += torch.arange(k, device="cuda") * (2 * BAND // k) - BAND
    o += o >= 0
    i = torch.arange(n, device="cuda")[:, None]
    c = i + o
    c = torch.where(c < 0, i - o + BAND, torch.where(c >= n, i - o - BAND, c))
    v = 2.0 * torch.rand((n, k), dtype=torch.float64, device="cuda", generator=g) - 1.0
    c = torch.cat([c, i], 1)
    v = torch.cat([v, BAND_DIAG * v.abs().sum(1, keepdim=True)], 1)
    c, order = c.sort(dim=1, stable=True)
    v = torch.gather(v, 1, order)
    rowptr = torch.arange(n + 1, device="cuda") * BAND_NNZ + 1
    return rowptr.int(), (c.reshape(-1) + 1).int(), v.reshape(-1).contiguous()


def _crs(case, seed):
    if case["problem"] == "banded":
        return _banded(case, seed)
    st = _stencil(case, seed)
    n = case["nx"] * case["ny"] * case["nz"]
    mask = torch.stack([m for _, _, m in st], 1)
    col = torch.arange(1, n + 1, device="cuda")[:, None] + torch.tensor([o for o, _, _ in st], device="cuda")
    val = torch.stack([v for _, v, _ in st], 1)
    rowptr = torch.ones(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] += mask.sum(1).cumsum(0)
    return rowptr.int(), col[mask].int(), val[mask]


def _dia(case, seed):
    st = _stencil(case, seed)
    val = torch.cat([torch.where(m, v, torch.zeros_like(v)) for _, v, m in st])
    return val, torch.tensor([o for o, _, _ in st], dtype=torch.int32, device="cuda")


def _ddm(case, seed):
    """The padded box (margin 1) of the 7-point stencil: values, offsets and offsets per axis."""
    size = [case["nx"], case["ny"], case["nz"]]
    pad = [s + 2 for s in size]
    step = [1, pad[0], pad[0] * pad[1]]
    val, off, per_axis = [], [], []
    for (_, v, m), (_, d, s) in zip(_stencil(case, seed), _neighbours(case)):
        box = torch.zeros(pad[::-1], dtype=torch.float64, device="cuda")
        box[1:-1, 1:-1, 1:-1] = torch.where(m, v, torch.zeros_like(v)).reshape(size[::-1])
        val.append(box.reshape(-1))
        off.append(s * step[d])
        per_axis.append([s if a == d else 0 for a in range(3)])
    od = np.ascontiguousarray(np.array(per_axis, np.int32).T.reshape(-1))
    return torch.cat(val), torch.tensor(off, dtype=torch.int32, device="cuda"), od


def _rhs(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


def _to_box(case, v):
    box = torch.zeros([case["nz"] + 2, case["ny"] + 2, case["nx"] + 2], dtype=torch.float64, device="cuda")
    box[1:-1, 1:-1, 1:-1] = v.reshape(case["nz"], case["ny"], case["nx"])
    return box.reshape(-1)


# ---- the calls ----------------------------------------------------------------------------------
class Handle:
    """parcel_b_setup's matrix layout and preconditioner, released with the object."""

    def __init__(self, options, crs):
        self.lib, self.h = _lib.load(), C.c_void_p()
        if self.lib.parcel_b_setup(C.byref(options), C.byref(crs), C.byref(self.h)) < 0:
            raise RuntimeError(_lib.last_error())

    def __del__(self):
        self.lib.parcel_b_release(self.h)


_stream = None


def _use_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
        if _lib.load().parcel_b_set_stream(_stream.cuda_stream) != 0:
            raise RuntimeError(_lib.last_error())
    _stream.wait_stream(torch.cuda.default_stream())
    return torch.cuda.stream(_stream)


def _options(case):
    o = dict(solver=SOLVERS[case["solver"]], ipreflag=case["precon"], ILU_method=case["ilu"],
             precon_thblock=case["blocks"], itrmax=ITRMAX, rtolmax=case["rtol"], GMRES_m=case["m"],
             GMRES_GSflag=case["gs"])
    if case["solver"] == "cagmres":
        o.update(CAGMRES_sstep=8, CAGMRES_tstep=8, CAGMRES_basis=1, CAGMRES_QRflag=3)
    if case["form"] in ("mixed", "learned"):
        o.update(inner_precision=1, inner_rtol=1e-4, max_refine=80)
    if case["form"] == "mixed":
        o.update(residual_dd=1)
    return o


class Shape:
    """What api.solve and its siblings read of a matrix besides the arrays: its order."""

    def __init__(self, n):
        self.n = n


def prepare(case, seed):
    with _use_stream():
        s = {"case": case, "n": case["nx"] * case["ny"] * case["nz"], "b": _rhs(case, seed)}
        if case["form"] == "dia":
            s["val"], s["offset"] = _dia(case, seed)
        elif case["form"] == "ddm":
            s["val"], s["offset"], s["offset_dim"] = _ddm(case, seed)
            s["b"] = _to_box(case, s["b"])
        else:
            s["rowptr"], s["col"], s["val"] = _crs(case, seed)
        if case["form"] == "host":
            for k in ("b", "rowptr", "col", "val"):
                s[k] = s[k].cpu().numpy()
        elif case["form"] == "handle":
            s["crs"] = api.crs_struct(Shape(s["n"]), s["rowptr"], s["col"], s["val"])
            s["handle"] = Handle(_lib.new_input(**_options(case)), s["crs"])
        elif case["form"] == "learned":
            s["net"] = api.Learned(case["nx"], case["ny"], case["nz"], COARSEN, seed=1)
            s["net"].set_stage(COARSE_STEPS, True)
    return s


def _wrapper(s):
    """The reference's argument list (parcel_dcg and its siblings) on device or host arrays."""
    c, n = s["case"], s["n"]
    x = np.zeros(n) if c["form"] == "host" else torch.zeros_like(s["b"])
    hist = np.zeros(ITRMAX)
    fn = {"cg": api.parcel_dcg, "bicgstab": api.parcel_dbicgstab, "gmres": api.parcel_dgmres,
          "cagmres": api.parcel_dcagmres}[c["solver"]]
    more = {}
    if c["solver"] == "gmres":
        more = dict(GMRES_m=c["m"], GMRES_GSflag=c["gs"])
    elif c["solver"] == "cagmres":
        more = dict(CAGMRES_sstep=8, CAGMRES_tstep=8, CAGMRES_basis=1, CAGMRES_QRflag=3)
    fn(x, s["b"], n, n, int(s["col"].shape[0]), 1, s["val"], s["rowptr"], s["col"], c["precon"], c["ilu"], 0, 1,
       ITRMAX, c["rtol"], hist, precon_thblock=c["blocks"], **more)
    return {"x": x, "hist": hist}


def run(s):
    c = s["case"]
    with torch.cuda.stream(_stream):
        if c["form"] in ("host", "device"):
            return _wrapper(s)
        o = _options(c)
        if c["form"] == "handle":
            x, hist = torch.zeros_like(s["b"]), np.zeros(ITRMAX)
            niter, iret = C.c_int(0), C.c_int(0)
            _lib.load().parcel_b_start(s["handle"].h, s["b"].data_ptr(), x.data_ptr(), hist.ctypes.data,
                                       C.byref(niter), C.byref(iret))
            return {"x": x, "hist": hist}
        if c["form"] == "dia":
            return {"x": api.solve_dia(s["val"], s["offset"], s["b"], **o)["x"]}
        if c["form"] == "ddm":
            size = [c["nx"], c["ny"], c["nz"]]
            return {"x": ddm.solve(s["val"], s["offset"], s["offset_dim"], size, s["b"], boxes=ddm.BOXES_CUBES,
                                   **o)["x"]}
        arrays = dict(rowptr=s["rowptr"], col=s["col"], val=s["val"])
        if c["form"] == "mixed":
            return {"x": api.solve(Shape(s["n"]), s["b"], **arrays, **o)["x"]}
        if c["form"] == "dd":
            r = api.ddcg(Shape(s["n"]), s["b"], **arrays, **o)
            return {"x_hi": r["x_hi"], "x_lo": r["x_lo"]}
        x = torch.zeros_like(s["b"])
        niter, iret = C.c_int(0), C.c_int(0)
        crs = api.crs_struct(Shape(s["n"]), s["rowptr"], s["col"], s["val"])
        _lib.load().parcel_b_solve_learned_many(C.byref(_lib.new_input(**o)), C.byref(crs), s["net"].handle, 1,
                                                s["b"].data_ptr(), x.data_ptr(), C.byref(niter), C.byref(iret))
        return {"x": x}


# ---- what a pass cannot do without ----------------------------------------------------------------
def _nnz(case):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["problem"] == "banded":
        return BAND_NNZ * n
    size = [s for s in (case["nx"], case["ny"], case["nz"]) if s > 1]
    return n + sum(2 * (n - n // s) for s in size)


def _iterations(case):
    """Iterations to the tolerance, from solves of each family (a model, within about 20 %)."""
    side = max(case["nx"], case["ny"], case["nz"])
    if case["solver"] == "cagmres":
        return 24
    if case["form"] == "learned":
        return 74
    decades = -math.log10(case["rtol"])
    per = {"cg": 0.19, "bicgstab": 0.12, "gmres": 0.23}[case["solver"]]
    if case["problem"] == "aniso":
        per *= 0.4
    if case["form"] == "ddm":
        per *= 1.2
    if case["precon"] < 2:
        per *= 1.8
    return max(5, int(per * side * decades))


def work(case):
    """Bytes and operations of the iteration: the matrix, the factors and the vectors once per use and iteration."""
    n, nnz, it = case["nx"] * case["ny"] * case["nz"], _nnz(case), _iterations(case)
    v = {"dd": 16, "mixed": 4, "learned": 4}.get(case["form"], 8)      # bytes of a vector entry
    a = 4 if v == 4 else 8                                             # of a matrix value
    spmv = (a + 4) * nnz + 4 * n + 2 * v * n
    precon = {0: 0, 1: 3 * v * n, 2: (a + 4) * nnz + 3 * v * n}[case["precon"]]
    if case["solver"] == "cg":
        per = spmv + precon + 8 * v * n
    elif case["solver"] == "bicgstab":
        per = 2 * spmv + 2 * precon + 12 * v * n
    elif case["solver"] == "gmres":
        per = spmv + precon + (case["m"] // 2 + 3) * v * n
    else:
        per = spmv + precon + 14 * v * n
    flops = 2 * nnz * (1 + (case["precon"] == 2)) * (2 if case["solver"] == "bicgstab" else 1) + 10 * n
    if case["solver"] in ("gmres", "cagmres"):
        flops += 4 * n * (case["m"] // 2)
    return {"bytes": it * per, "flops": it * flops * (20 if case["form"] == "dd" else 1)}


# Largest relative error of a converged solve, as a multiple of its stopping tolerance: how much
# a residual of that size is amplified into x on the grids above, four times the largest
# measured against exact() (CG 35, BiCGStab 150, GMRES 260, CA-GMRES on the banded matrix 1; a
# refinement loop ends anywhere below its tolerance, so at most what its inner solver shows).
# The histories differ by less.  The double-double solvers fix the order of
# every operation, so their results are the same bits.
def tolerance(case):
    if case["form"] == "dd":
        return "exact"
    amplify = {"cg": 140.0, "bicgstab": 600.0, "gmres": 1000.0, "cagmres": 4.0}[case["solver"]]
    return {"rel": amplify * case["rtol"]}


# ---- the answers in 64 bits ------------------------------------------------------------------------
def _separable(case, b):
    """A constant-coefficient stencil is a sum of one tridiagonal operator per axis: transform each axis to its eigenvectors."""
    ax = _axes(case)
    shape = [a[3] for a in reversed(ax)]
    scale, vec, lam = [], [], []
    for lo, diag, hi, n in ax:
        off = torch.full((n - 1,), -math.sqrt(lo * hi), dtype=torch.float64, device="cuda")
        t = torch.diag(torch.full((n,), diag, dtype=torch.float64, device="cuda"))
        t = t + torch.diag(off, 1) + torch.diag(off, -1)
        w, q = torch.linalg.eigh(t)
        lam.append(w)
        vec.append(q)
        scale.append((lo / hi) ** (0.5 * torch.arange(n, dtype=torch.float64, device="cuda")))

    def along(v, op, d):
        return torch.movedim(torch.tensordot(op, v, dims=([1], [len(ax) - 1 - d])), 0, len(ax) - 1 - d)

    def view(v, d):
        return v.reshape([-1 if e == len(ax) - 1 - d else 1 for e in range(len(ax))])

    denom = sum(view(lam[d], d) for d in range(len(ax)))

    def apply(x):
        y = torch.zeros_like(x)
        for d, (lo, diag, hi, n) in enumerate(ax):
            e = len(ax) - 1 - d
            y += diag * x
            y.narrow(e, 1, n - 1).add_(x.narrow(e, 0, n - 1), alpha=lo)
            y.narrow(e, 0, n - 1).add_(x.narrow(e, 1, n - 1), alpha=hi)
        return y

    def solve(r):
        for d in range(len(ax)):
            r = along(r / view(scale[d], d), vec[d].T.contiguous(), d)
        r = r / denom
        for d in range(len(ax)):
            r = along(r, vec[d], d) * view(scale[d], d)
        return r

    b = b.reshape(shape)
    x = solve(b)
    for _ in range(2):
        x = x + solve(b - apply(x))
    return x.reshape(-1)


def _richardson(case, seed, b):
    """The banded matrix is diagonally dominant: point Jacobi steps until they no longer change x."""
    _, col, val = _banded(case, seed)
    n = case["nx"]
    col, val = (col.long() - 1).reshape(n, BAND_NNZ), val.reshape(n, BAND_NNZ)
    diag = val[col == torch.arange(n, device="cuda")[:, None]]
    x = torch.zeros_like(b)
    for _ in range(300):
        step = (b - (val * x[col]).sum(1)) / diag
        x = x + step
        if step.norm() <= 1e-16 * x.norm():
            break
    return x


def _conjugate(case, seed, b):
    """Jacobi-preconditioned CG on the variable-coefficient stencil."""
    st = _stencil(case, seed)
    diag = st[len(st) // 2][1]
    parts = [(o, torch.where(m, v, torch.zeros_like(v))) for o, v, m in st if o]
    n = b.numel()

    def apply(x):
        y = diag * x
        for o, v in parts:
            if o < 0:
                y[-o:] += v[-o:] * x[:o]
            else:
                y[:n - o] += v[:n - o] * x[o:]
        return y

    x = torch.zeros_like(b)
    for _ in range(2):
        r = b - apply(x)
        z = r / diag
        p, rz, d = z.clone(), r @ z, torch.zeros_like(b)
        for i in range(3000):
            q = apply(p)
            alpha = rz / (p @ q)
            d += alpha * p
            r -= alpha * q
            if i % 50 == 49 and r.norm() < 1e-13 * b.norm():
                break
            z = r / diag
            new = r @ z
            p = z + (new / rz) * p
            rz = new
        x = x + d
    return x


def exact(case, seed):
    b = _rhs(case, seed)
    if case["problem"] == "banded":
        x = _richardson(case, seed, b)
    elif case["problem"] == "vardiff":
        x = _conjugate(case, seed, b)
    else:
        x = _separable(case, b)
    if case["form"] == "dd":
        return {"x_hi": x, "x_lo": None}
    if case["form"] == "ddm":
        return {"x": _to_box(case, x)}
    if case["form"] == "host":
        return {"x": x.cpu().numpy(), "hist": None}
    return {"x": x, "hist": None} if case["form"] in ("device", "handle") else {"x": x}
