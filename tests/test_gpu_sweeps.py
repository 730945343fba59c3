"""Block-Jacobi sweeps at the sizes where their layout changes: blocks that start inside a
grid plane (levels tightened before the layout is made), blocks whose level gaps are so long
that the shared-memory ring holds the whole block by position, levels wider than one chunk,
levels narrower than a warp, and every supported coupling count.

Tolerance: the sweeps evaluate the oracle's expressions with fused multiply-adds; 1e-11 of
the largest entry, as the other preconditioner tests.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
from parcel_b import _lib, api, problems

pytestmark = pytest.mark.gpu


def _apply_both(A, **pre):
    r = np.random.default_rng(11).standard_normal(A.n)
    s_ref = oracle.precon_apply(A, r, **pre)
    s = np.zeros(A.n)
    p = _lib.new_input(**pre)
    rc = _lib.load().parcel_b_precon_apply(C.byref(p), C.byref(api.crs_struct(A)), r.ctypes.data, s.ctypes.data)
    assert rc == 0, _lib.last_error()
    return np.abs(s - s_ref).max() / np.abs(s_ref).max()


def _symmetric_pattern(n, links, seed):
    """A diagonally dominant matrix with the given number of long-range links per row (and
    their transposes), nonsymmetric values."""
    rng = np.random.default_rng(seed)
    cols = [set((i,)) for i in range(n)]
    for k in range(links):
        p = rng.permutation(n)
        for i in range(n):
            cols[i].add(int(p[i]))
            cols[int(p[i])].add(i)
    rp, ci, va = [1], [], []
    for i in range(n):
        c = sorted(cols[i])
        ci += [j + 1 for j in c]
        va += [4.0 * len(c) if j == i else float(rng.uniform(-1, 1)) for j in c]
        rp.append(len(ci) + 1)
    return problems.CRS(n=n, rowptr=np.array(rp, np.int32), col=np.array(ci, np.int32), val=np.array(va))


@pytest.mark.parametrize("ilu", [0, 1])
@pytest.mark.parametrize("N,blocks", [(31, 1), (31, 7), (41, 3), (47, 5)])
def test_blocks_that_start_inside_a_plane(N, blocks, ilu):
    A = problems.convdiff3d_upwind(N)
    assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=blocks) < 1e-11


@pytest.mark.parametrize("n,blocks", [(700, 1), (6001, 3), (9000, 1)])
def test_long_level_gaps(n, blocks):
    """One link per row: at most four couplings; the blocks of 700, 2,000 and 9,000 rows keep
    their whole solution, or too long a ring for 64 KB, which takes the general sweep."""
    A = _symmetric_pattern(n, 1, n)
    for ilu in (0, 1):
        assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=blocks) < 1e-11


@pytest.mark.parametrize("links", [1, 2, 3, 4])
def test_coupling_counts(links):
    """Up to eight couplings per row and sweep in the records, more in the general sweep."""
    A = _symmetric_pattern(1500, links, 90 + links)
    for ilu in (0, 1):
        assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=2) < 1e-11


@pytest.mark.parametrize("nx,ny", [(3, 900), (20, 20), (600, 600)])
def test_level_widths(nx, ny):
    """2D grids: levels of at most 3 rows, of 20, and of more than one 512-row chunk."""
    A = problems.poisson2d_5pt(nx, ny)
    for ilu in (0, 1):
        assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=1) < 1e-11


def _lattice(nx, ny, diagonals):
    """nx x ny grid, five-point links plus the first `diagonals` of the two diagonal directions."""
    i = np.arange(nx * ny).reshape(ny, nx)
    pairs = [(i[:, :-1], i[:, 1:]), (i[:-1], i[1:]), (i[:-1, :-1], i[1:, 1:]), (i[:-1, 1:], i[1:, :-1])][:2 + diagonals]
    r = np.concatenate([i.ravel()] + [np.concatenate([a.ravel(), b.ravel()]) for a, b in pairs])
    c = np.concatenate([i.ravel()] + [np.concatenate([b.ravel(), a.ravel()]) for a, b in pairs])
    v = np.random.default_rng(nx).uniform(-1, 1, r.size)
    v[:nx * ny] = 9.0
    o = np.lexsort((c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=nx * ny))]) + 1
    return problems.CRS(n=nx * ny, rowptr=rp.astype(np.int32), col=(c[o] + 1).astype(np.int32), val=v[o])


@pytest.mark.parametrize("ilu", [0, 1])
@pytest.mark.parametrize("nx,ny,diagonals,blocks", [(40, 30, 1, 1), (40, 30, 2, 3), (700, 700, 0, 1), (700, 700, 1, 2)])
def test_factor_recurrences(nx, ny, diagonals, blocks, ilu):
    """Three and four couplings; levels wider than the recurrence's CTA; triangles, which send
    ILU(0) to the general elimination but not D-ILU."""
    assert _apply_both(_lattice(nx, ny, diagonals), ipreflag=2, ILU_method=ilu, precon_thblock=blocks) < 1e-11


# ---- many small blocks: plan on the device, CG's step fused into the sweep --------------------
def _dense_blocks(nb, rows, seed):
    """nb blocks of `rows` fully coupled rows each, linked to the next block by one entry."""
    rng = np.random.default_rng(seed)
    n = nb * rows
    i = np.arange(n)
    base = i // rows * rows
    col = base[:, None] + np.arange(rows)[None, :]
    val = rng.uniform(-1, 1, (n, rows))
    val[i, i - base] = 2.0 * rows
    col = np.concatenate([col, np.minimum(base + rows, n - 1)[:, None]], 1)
    val = np.concatenate([val, np.full((n, 1), 0.5)], 1)
    keep = np.ones_like(col, bool)
    keep[:, -1] = base + rows < n
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]) + 1
    return problems.CRS(n=n, rowptr=rp.astype(np.int32), col=(col[keep] + 1).astype(np.int32), val=val[keep])


@pytest.mark.parametrize("ilu", [0, 1, 2])
@pytest.mark.parametrize("nb,rows", [(1300, 1), (1300, 3), (1400, 9), (1200, 12)])
def test_small_dense_blocks(nb, rows, ilu):
    """One-row blocks, one coupling count after the other, and more couplings than the records
    hold (the general plan and the general sweep)."""
    A = _dense_blocks(nb, rows, rows)
    assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=nb) < 1e-11


@pytest.mark.parametrize("ilu", [0, 1])
@pytest.mark.parametrize("N,blocks", [(24, 1200), (24, 2000), (24, 5000), (61, 1500), (30, 27000)])
def test_small_blocks_cg(N, blocks, ilu):
    """CG through the fused sweep: 8, 16 and 32 lanes per block, staged and (61^3: 151 rows a
    block) long stretches, one row per block; iterations and x against the oracle's."""
    A = problems.poisson3d_reference(N, N, N)[0]
    b = problems.rhs_normal(A.n, N)
    kw = dict(solver=1, itrmax=60 if N > 40 else 400, rtolmax=1e-10, ipreflag=2, ILU_method=ilu,
              precon_thblock=blocks)
    xo, ho, no, io = oracle.solve(A, b, **kw)
    res = api.solve(A, b, **kw)
    assert abs(res["niter"] - no) <= 1
    k = min(len(ho), len(res["reshistory"]))
    assert (np.abs(res["reshistory"][:k] - ho[:k]) / ho[:k]).max() < 1e-6
    assert np.abs(res["x"] - xo).max() < 1e-7 * np.abs(xo).max()


def test_small_blocks_mixed_precision_cg():
    A = problems.poisson3d_reference(24, 24, 24)[0]
    b = problems.rhs_normal(A.n, 2)
    res = api.solve(A, b, solver=1, itrmax=2000, rtolmax=1e-12, ipreflag=2, ILU_method=1, precon_thblock=2000,
                    inner_precision=1, inner_rtol=1e-4, residual_dd=1, max_refine=50)
    assert res["iret"] == 0 and res["stats"]["true_relres"] < 1e-12


def test_small_blocks_missing_diagonal_is_an_error():
    A = _dense_blocks(1300, 3, 1)
    A.col[A.rowptr[700] - 1:A.rowptr[701] - 1][...] = np.clip(
        A.col[A.rowptr[700] - 1:A.rowptr[701] - 1], 1, A.n)
    row = slice(A.rowptr[700] - 1, A.rowptr[701] - 1)
    keep = A.col[row] != 701
    B = problems.CRS(n=A.n, rowptr=A.rowptr.copy(), col=np.delete(A.col, np.flatnonzero(~keep) + row.start),
                     val=np.delete(A.val, np.flatnonzero(~keep) + row.start))
    B.rowptr[701:] -= 1
    with pytest.raises(RuntimeError, match="block 233 has a row without an in-block diagonal"):
        api.solve(B, np.ones(B.n), solver=3, ipreflag=2, ILU_method=0, precon_thblock=1300)


# ---- CG of short vectors in one launch -----------------------------------------------------------
@pytest.mark.parametrize("ipreflag", [0, 1])
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 2), (32, 16), (33, 16), (270, 281), (280, 271), (389, 390), (551, 550)])
def test_short_vector_cg(nx, ny, ipreflag):
    """One CTA, a partial one, and the row counts either side of 1, 2 and 4 rows per thread (151,552
    and 303,104 rows on 148 SMs); past the last the separate kernels run."""
    A = problems.poisson2d_5pt(nx, ny)
    b = problems.rhs_normal(A.n, 1 + nx)
    kw = dict(solver=1, itrmax=40, rtolmax=1e-10, ipreflag=ipreflag)
    xo, ho, no, io = oracle.solve(A, b, **kw)
    res = api.solve(A, b, **kw)
    assert res["niter"] == no and res["iret"] == io
    assert (np.abs(res["reshistory"][:no] - ho[:no]) / ho[:no]).max() < 1e-6
    assert np.abs(res["x"] - xo).max() < 1e-7 * np.abs(xo).max()


@pytest.mark.parametrize("ipreflag", [0, 1])
@pytest.mark.parametrize("nx,ny", [(551, 551), (673, 677)])
def test_cg_step(nx, ny, ipreflag):
    """The smallest vector past the one-launch CG, and one with elements over in the last step of
    a thread (a step takes three elements of each of 151,552 threads)."""
    A = problems.poisson2d_5pt(nx, ny)
    b = problems.rhs_normal(A.n, nx)
    kw = dict(solver=1, itrmax=40, rtolmax=1e-10, ipreflag=ipreflag)
    xo, ho, no, io = oracle.solve(A, b, **kw)
    res = api.solve(A, b, **kw)
    assert res["niter"] == no and res["iret"] == io
    assert (np.abs(res["reshistory"][:no] - ho[:no]) / ho[:no]).max() < 1e-6
    assert np.abs(res["x"] - xo).max() < 1e-7 * np.abs(xo).max()


def test_short_vector_cg_without_a_diagonal_copy_and_past_one_launch():
    """A matrix that has no diagonal copy (sliced ELLPACK), and more iterations than one launch
    runs (4,096), ended by the iteration limit."""
    A = _symmetric_pattern(900, 3, 4)
    S = A.to_scipy()
    S = (S + S.T).tocsr()
    S.sort_indices()
    B = problems.CRS(n=900, rowptr=(S.indptr + 1).astype(np.int32), col=(S.indices + 1).astype(np.int32),
                     val=S.data.copy())
    b = problems.rhs_normal(900, 5)
    xo, ho, no, io = oracle.solve(B, b, solver=1, itrmax=300, rtolmax=1e-10, ipreflag=1)
    res = api.solve(B, b, solver=1, itrmax=300, rtolmax=1e-10, ipreflag=1)
    assert res["niter"] == no and res["iret"] == io and res["stats"]["spmv_diagonals"] == 0
    assert np.abs(res["x"] - xo).max() < 1e-9 * np.abs(xo).max()
    P = problems.poisson2d_5pt(300, 301)
    res = api.solve(P, problems.rhs_normal(P.n, 5), solver=1, itrmax=5000, rtolmax=0.0, ipreflag=1)
    # the true residual stagnates at the order of eps cond(A) = 2e-16 * 4e4
    assert res["niter"] == 5000 and res["iret"] == 1 and res["stats"]["true_relres"] < 1e-11


# ---- double-double: bit for bit ----------------------------------------------------------------
def _dd_both(A, b, **kw):
    g = api.ddcg(A, b, **kw)
    xh, xl, h, niter, _ = oracle.ddcg(A, b, **kw)
    assert g["niter"] == niter
    assert np.array_equal(g["reshistory"], h, equal_nan=True)
    assert np.array_equal(g["x_hi"], xh, equal_nan=True) and np.array_equal(g["x_lo"], xl, equal_nan=True)


@pytest.mark.parametrize("solver", [1, 2, 3])
@pytest.mark.parametrize("N,blocks", [(21, 3), (13, 1), (24, 2000)])
def test_dd_blocks(N, blocks, solver):
    """Ragged blocks, one block, and so many that the sweep without staged records runs."""
    A = problems.poisson3d_reference(N, N, N)[0] if solver == 1 else problems.convdiff3d_upwind(N)
    _dd_both(A, problems.rhs_normal(A.n, N), solver=solver, itrmax=25, rtolmax=1e-13, GMRES_m=7, ipreflag=2,
             ILU_method=1, precon_thblock=blocks)


@pytest.mark.parametrize("links", [1, 2, 3, 4])
def test_dd_coupling_counts(links):
    """Up to six couplings per row and sweep in the records, more in the sweep without them."""
    A = _symmetric_pattern(1500, links, 90 + links)
    for ilu in (1, 2):
        _dd_both(A, problems.rhs_normal(A.n, 5), solver=3, itrmax=12, rtolmax=1e-25, GMRES_m=5, ipreflag=2,
                 ILU_method=ilu, precon_thblock=2)


@pytest.mark.parametrize("exponent", [-520, -300, 0, 300, 505])
def test_dd_products_near_the_ends_of_the_range(exponent):
    """Right-hand sides scaled so far that products and their rounding errors leave the range in
    which a fused multiply-subtract equals the split product."""
    A = problems.poisson3d_reference(12, 12, 12)[0]
    b = problems.rhs_normal(A.n, 3) * 2.0 ** exponent
    _dd_both(A, b, solver=1, itrmax=20, rtolmax=1e-13, ipreflag=2, ILU_method=1, precon_thblock=3)


@pytest.mark.parametrize("n,m,itrmax", [(524288, 3, 5), (524289, 3, 5), (700001, 4, 6), (1000, 700, 12), (3, 5, 4)])
def test_dd_mgs_column_sizes(n, m, itrmax):
    """Basis vectors at and past the register-resident length, a restart length whose rotations
    do not fit shared memory, and fewer rows than a CTA has threads."""
    i = np.arange(n)
    cols, vals = [i - 1, i, i + 1], [-1.1, 4.0 + (i % 7) * 0.25, -0.9]
    mask = [i > 0, i >= 0, i < n - 1]
    C3 = np.stack(cols, 1)
    V3 = np.stack([np.broadcast_to(v, n) for v in vals], 1)
    M3 = np.stack(mask, 1)
    rp = np.concatenate([[0], np.cumsum(M3.sum(1))]) + 1
    A = problems.CRS(n=n, rowptr=rp.astype(np.int32), col=(C3[M3] + 1).astype(np.int32), val=V3[M3].astype(float))
    _dd_both(A, problems.rhs_normal(n, 8), solver=3, itrmax=itrmax, rtolmax=1e-28, GMRES_m=m, GMRES_GSflag=1,
             ipreflag=1)


# ---- times that a launch shape decides ------------------------------------------------------------
def _spread_rows(n, k, seed):
    """n rows of k entries spread over a quarter of the columns, the diagonal among them."""
    rng = np.random.default_rng(seed)
    w = max(n // 4, k)
    c = (np.arange(n)[:, None] + np.arange(k) * (w // k) + rng.integers(0, max(1, w // k), (n, k))) % n
    c[:, 0] = np.arange(n)
    c.sort(1)
    v = -rng.random((n, k))
    v[c == np.arange(n)[:, None]] = 1.2 * k
    keep = np.ones_like(c, bool)
    keep[:, 1:] = c[:, 1:] != c[:, :-1]
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]) + 1
    return problems.CRS(n=n, rowptr=rp.astype(np.int32), col=(c[keep] + 1).astype(np.int32), val=v[keep])


def _spmv_ms(A):
    import time
    import torch
    L = _lib.load()
    rp, ci, va, x = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.rowptr, A.col, A.val, np.ones(A.n)))
    y = torch.empty_like(x)
    S = api.crs_struct(A, rp, ci, va)
    best = np.inf
    torch.cuda.synchronize()
    for _ in range(8):
        t = time.perf_counter()
        for _ in range(20):
            assert L.parcel_b_spmv(C.byref(S), x.data_ptr(), y.data_ptr()) == 0, _lib.last_error()
        torch.cuda.synchronize()
        best = min(best, (time.perf_counter() - t) / 20)
    assert np.abs(y.cpu().numpy() - A.to_scipy() @ np.ones(A.n)).max() < 1e-11 * np.abs(A.val).max()
    return best


def test_product_of_few_long_rows_fills_the_chip():
    """Rows of 400 entries are split over a warp each, so 2,000 of them need 250 CTAs; with a CTA for
    256 rows (8 CTAs) their product took five times as long as the call, which the same number of
    short rows measures."""
    assert _spmv_ms(_spread_rows(2000, 400, 1)) < 2.0 * _spmv_ms(_spread_rows(2000, 9, 1))


@pytest.mark.parametrize("n,k,one_launch", [(20000, 100, True), (20400, 100, False), (180000, 11, True), (180000, 14, False)])
def test_short_vector_cg_is_for_few_entries(n, k, one_launch):
    """Either side of two million entries, and of twelve a row past that: the launch count tells which
    kernels ran (the separate ones are three an iteration)."""
    A = _spread_rows(n, k, 3)
    b = problems.rhs_normal(A.n, 4)
    kw = dict(solver=1, itrmax=30, rtolmax=1e-200, ipreflag=1)
    xo, _, no, _ = oracle.solve(A, b, **kw)
    res = api.solve(A, b, **kw)
    assert res["niter"] == no == 30
    assert (res["stats"]["kernel_launches"] < 20) == one_launch
    assert np.abs(res["x"] - xo).max() < 1e-9 * np.abs(xo).max()


def test_dd_setup_of_many_small_blocks():
    """4,096 lines of 64 rows, each row its own level: the set-up makes no table of the sweep with staged
    records, which these blocks do not take (with it 1.5 applications' time, without 0.9)."""
    import torch
    A = problems.poisson3d_reference(64, 64, 64)[0]
    rp, ci, va, b = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.rowptr, A.col, A.val, np.ones(A.n)))
    torch.cuda.synchronize()
    st = [api.ddcg(A, b, rowptr=rp, col=ci, val=va, itrmax=8, rtolmax=1e-30, ipreflag=2, ILU_method=1,
                   precon_thblock=4096)["stats"] for _ in range(5)]
    assert min(s["setup_s"] for s in st) < 1.25 * min(s["solve_s"] for s in st) / 8


# ---- the wavefront plan -----------------------------------------------------------------------------
def _from_pairs(n, r, c, seed):
    """A diagonally dominant matrix with the given entries (r, c) and the diagonal, pattern as given."""
    rng = np.random.default_rng(seed)
    key = np.unique(np.concatenate([np.arange(n, dtype=np.int64) * (n + 1), np.asarray(r, np.int64) * n + np.asarray(c, np.int64)]))
    r, c = key // n, key % n
    v = rng.uniform(-1, 1, r.size)
    cnt = np.bincount(r, minlength=n)
    v[r == c] = 2.0 * cnt + np.bincount(c, minlength=n)
    rp = np.concatenate([[0], np.cumsum(cnt)]) + 1
    return problems.CRS(n=n, rowptr=rp.astype(np.int32), col=(c + 1).astype(np.int32), val=v)


def _chain(n):
    i = np.arange(n - 1)
    return np.concatenate([i, i + 1]), np.concatenate([i + 1, i])


@pytest.mark.parametrize("ilu", [0, 1])
@pytest.mark.parametrize("n,blocks", [(130, 1), (1024, 1), (5000, 1), (5000, 3), (4000, 900)])
def test_plan_of_chains(n, blocks, ilu):
    """Tridiagonal blocks: every row its own level, more rounds than a chunk of rows is given."""
    assert _apply_both(_from_pairs(n, *_chain(n), 1), ipreflag=2, ILU_method=ilu, precon_thblock=blocks) < 1e-11


@pytest.mark.parametrize("chain", [False, True])
@pytest.mark.parametrize("n,blocks", [(700, 1), (3000, 1), (6000, 4), (9000, 600), (60000, 1300)])
def test_plan_of_one_sided_couplings(n, blocks, chain):
    """Entries whose transposes are missing, near (same chunk of rows) and far, with and without a
    chain through all rows; some rows with more near couplings than are listed."""
    rng = np.random.default_rng(n)
    r = rng.integers(0, n, 2 * n)
    c = np.clip(r + rng.integers(-90, 91, 2 * n), 0, n - 1)
    r2, c2 = rng.integers(0, n, n // 4), rng.integers(0, n, n // 4)
    dense = rng.choice(n, max(1, n // 200), replace=False)
    r3 = np.repeat(dense, 41)
    c3 = np.clip(r3 + np.tile(np.arange(-20, 21), dense.size), 0, n - 1)
    r, c = np.concatenate([r, r2, r3]), np.concatenate([c, c2, c3])
    if chain:
        a, b = _chain(n)
        r, c = np.concatenate([r, a]), np.concatenate([c, b])
    A = _from_pairs(n, r, c, 2)
    for ilu in (0, 1):
        assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=blocks) < 1e-11


@pytest.mark.parametrize("ilu", [0, 1])
def test_plan_moves_levels_along_a_chain(ilu):
    """A chain of 6,000 rows and 3,000 rows between that could start at once but are coupled to its end:
    late levels over chunks that need a round per row."""
    n = 9000
    link = np.concatenate([np.arange(3000), np.arange(6000, 9000)])
    single = np.arange(3000, 6000)
    end = 8999 - np.arange(3000) % 1500
    r = np.concatenate([link[:-1], link[1:], single, end])
    c = np.concatenate([link[1:], link[:-1], end, single])
    assert _apply_both(_from_pairs(n, r, c, 3), ipreflag=2, ILU_method=ilu, precon_thblock=1) < 1e-11


_TRACE = """
import sys, numpy as np, torch
sys.path[:0] = %r
import test_gpu_sweeps as t
from parcel_b import api, problems
A = t._from_pairs(100000, *t._chain(100000), 1) if sys.argv[1] == "chain" else problems.poisson3d_reference(100, 100, 120)[0]
rp, ci, va, b = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.rowptr, A.col, A.val, np.ones(A.n)))
torch.cuda.synchronize()
for _ in range(3):
    api.solve(A, b, rowptr=rp, col=ci, val=va, solver=3, ipreflag=2, ILU_method=0, precon_thblock=int(sys.argv[2]), itrmax=1, rtolmax=1e-30)
"""


@pytest.mark.parametrize("matrix,blocks", [("chain", 1), ("grid", 1200)])
def test_plan_takes_less_than_the_factorisation(matrix, blocks):
    """One long chain, and 1,200 blocks of 1,000 rows: plans that took 1.4 and five times as long as
    the factorisation when a round went to every row or a thread to every block."""
    import os
    import re
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    path = [here, os.path.join(here, "..", "parcel-legacy_b200"), os.path.join(here, "..", "oracle")]
    out = subprocess.run([sys.executable, "-c", _TRACE % path, matrix, str(blocks)], capture_output=True, text=True,
                         timeout=300, env=dict(os.environ, PARCEL_B_TRACE="1"))
    assert out.returncode == 0, out.stderr[-2000:]
    ms = lambda label: min(float(x) for x in re.findall(re.escape(label) + r"\s+([\d.]+) ms", out.stderr))
    assert ms("setup: wavefront plan") < ms("ilu: factor" if blocks == 1 else "setup: ILU factor + pack")


# ---- BiCGStab on a sweep in another order than its vectors' --------------------------------------------
@pytest.mark.parametrize("inner", [0, 1])
@pytest.mark.parametrize("ilu", [0, 1])
@pytest.mark.parametrize("N,blocks", [(31, 7), (41, 3), (33, 1)])
def test_bicgstab_on_ragged_blocks(N, blocks, ilu, inner):
    """Blocks of more than 2,048 rows that start inside a plane: their levels are moved for the sweep,
    the vectors keep the early levels' order (33^3 in one block: nothing to move)."""
    A = problems.convdiff3d_upwind(N)
    pre = dict(ipreflag=2, ILU_method=ilu, precon_thblock=blocks)
    b = problems.rhs_normal(A.n, N)
    if inner:
        res = api.solve(A, b, solver=2, itrmax=500, rtolmax=1e-11, inner_precision=1, inner_rtol=1e-4, max_refine=40, **pre)
        xo, _, _, _ = oracle.solve(A, b, solver=2, itrmax=500, rtolmax=1e-12, **pre)
        assert res["iret"] == 0 and res["stats"]["true_relres"] < 1e-11
        # 1.1e-11 cond(A), cond(A) as below
        assert np.linalg.norm(res["x"] - xo) < 1.1e-11 * 0.41 * (N + 1) ** 2 * np.linalg.norm(xo)
        return
    assert _apply_both(A, solver=2, **pre) < 1e-11
    kw = dict(solver=2, itrmax=400, rtolmax=1e-9, **pre)
    xo, ho, no, io = oracle.solve(A, b, **kw)
    res = api.solve(A, b, **kw)
    assert abs(res["niter"] - no) <= 1 and res["iret"] == io
    k = min(5, len(ho))   # its recurrences amplify rounding: the first steps agree closely, then x does
    assert (np.abs(res["reshistory"][:k] - ho[:k]) / ho[:k]).max() < 1e-9
    # both residuals are below 1e-9 |b|, so x differs by at most 2e-9 cond(A), 4 (N + 1)^2 / pi^2
    assert np.linalg.norm(res["x"] - xo) < 2e-9 * 0.41 * (N + 1) ** 2 * np.linalg.norm(xo)


def test_bicgstab_sets_up_one_order_where_levels_do_not_move():
    """One block of whole planes: its levels cannot move, so BiCGStab plans and factors once, as GMRES."""
    import torch
    A = problems.convdiff3d_upwind(64)
    rp, ci, va, b = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.rowptr, A.col, A.val, np.ones(A.n)))
    torch.cuda.synchronize()
    t = {}
    for solver in (2, 3):
        kw = dict(solver=solver, ipreflag=2, ILU_method=1, precon_thblock=1, itrmax=1, rtolmax=1e-30)
        t[solver] = min(api.solve(A, b, rowptr=rp, col=ci, val=va, **kw)["stats"]["setup_s"] for _ in range(6))
    assert t[2] < 1.35 * t[3]


# ---- records of many couplings on wide levels, and of one -----------------------------------------------
def _stencil15(nx, ny, nz, corners=4):
    """The 7-point stencil and the first `corners` pairs of cube corners: 3 + corners couplings each way."""
    i = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    sh = [(0, 0, 1), (0, 1, 0), (1, 0, 0)] + [(1, 1, 1), (1, 1, -1), (1, -1, 1), (1, -1, -1)][4 - corners:]
    cut = lambda d, n, up: slice(max(d, 0), n + min(d, 0)) if up else slice(max(-d, 0), n + min(-d, 0))
    r = np.concatenate([i[cut(a, nz, 0), cut(b, ny, 0), cut(c, nx, 0)].ravel() for a, b, c in sh])
    c = np.concatenate([i[cut(a, nz, 1), cut(b, ny, 1), cut(c, nx, 1)].ravel() for a, b, c in sh])
    return _from_pairs(nx * ny * nz, np.concatenate([r, c]), np.concatenate([c, r]), 7)


@pytest.mark.parametrize("dims,blocks,corners", [((96, 96, 8), 2, 4), ((140, 140, 4), 1, 4), ((140, 140, 4), 1, 2),
                                                 ((200, 180, 5), 1, 4)])
def test_many_couplings_on_wide_levels(dims, blocks, corners):
    """Five to seven couplings on levels of 372 rows and of more than one chunk (480 rows of seven
    couplings, 512 of fewer; in double-double 352 of five and six)."""
    A = _stencil15(*dims, corners=corners)
    pre = dict(ipreflag=2, precon_thblock=blocks)
    for ilu in (0, 1):
        assert _apply_both(A, ILU_method=ilu, **pre) < 1e-11
    if corners == 2:
        _dd_both(A, problems.rhs_normal(A.n, 5), solver=1, itrmax=6, rtolmax=1e-25, ILU_method=1, **pre)


def _apply_ms(A, **pre):
    import torch
    rp, ci, va = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.rowptr, A.col, A.val))
    torch.cuda.synchronize()
    p, S, a, b = _lib.new_input(**pre), api.crs_struct(A, rp, ci, va), C.c_double(), C.c_double()
    best = np.inf
    for _ in range(5):
        assert _lib.load().parcel_b_bench_kernels(C.byref(p), C.byref(S), 20, C.byref(a), C.byref(b)) == 0
        best = min(best, b.value)
    return best


def test_many_couplings_on_wide_levels_stay_in_registers():
    """Levels of 372 rows: eight couplings a row cost 1.2 times as much as six when a thread's two rows are
    in registers, twice as much when they spill."""
    pre = dict(solver=3, ipreflag=2, ILU_method=0, precon_thblock=24)
    assert _apply_ms(_stencil15(96, 96, 96), **pre) < 1.6 * _apply_ms(_stencil15(96, 96, 96, corners=3), **pre)


def test_lines_as_blocks_keep_their_shared_memory():
    """64-row lines have 64 levels, each a stretch of four positions: padding their one coupling to four
    took the D-ILU sweep (two arrays fewer than ILU(0)'s) to ILU(0)'s time, from 0.6 of it."""
    A = problems.poisson3d_reference(64, 64, 64)[0]
    pre = dict(solver=1, ipreflag=2, precon_thblock=4096)
    assert _apply_ms(A, ILU_method=1, **pre) < 0.8 * _apply_ms(A, ILU_method=0, **pre)


# ---- a sweep that gives up --------------------------------------------------------------------------
_FAIL = (C.c_int * 7)(0, 0, 1)   # the sweeps' error flag starts set, as if a bounded wait had run out


@pytest.mark.parametrize("blocks", [3, 1200])
@pytest.mark.parametrize("kw", [dict(solver=1), dict(solver=2), dict(solver=3), dict(solver=3, GMRES_GSflag=2),
                                dict(solver=4, CAGMRES_sstep=4, CAGMRES_tstep=4),
                                dict(solver=1, inner_precision=1), dict(solver=3, inner_precision=1)])
def test_solves_report_a_sweep_that_gave_up(kw, blocks):
    A = problems.poisson3d_reference(14, 14, 14)[0]
    b = problems.rhs_normal(A.n, 2)
    kw = dict(kw, ipreflag=2, ILU_method=1, precon_thblock=blocks, itrmax=500, rtolmax=1e-6)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        api.solve(A, b, reserved=_FAIL, **kw)
    assert api.solve(A, b, **kw)["iret"] == 0


@pytest.mark.parametrize("solver", [1, 2, 3])
def test_dd_solves_report_a_sweep_that_gave_up(solver):
    A = problems.poisson3d_reference(10, 10, 10)[0]
    kw = dict(solver=solver, ipreflag=2, ILU_method=1, precon_thblock=3, itrmax=60, rtolmax=1e-6)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        api.ddcg(A, problems.rhs_normal(A.n, 2), reserved=_FAIL, **kw)
    assert api.ddcg(A, problems.rhs_normal(A.n, 2), **kw)["iret"] == 0


def test_a_handle_reports_a_sweep_that_gave_up_in_every_start():
    """parcel_b_start clears the flag at its start: the next one reports its own outcome alone."""
    A = problems.poisson3d_reference(14, 14, 14)[0]
    L, n, i, h = _lib.load(), C.c_int(), C.c_int(), C.c_void_p()
    p = _lib.new_input(solver=3, ipreflag=2, ILU_method=0, precon_thblock=3, itrmax=60, rtolmax=1e-6, reserved=_FAIL)
    S = api.crs_struct(A)
    assert L.parcel_b_setup(C.byref(p), C.byref(S), C.byref(h)) == 0, _lib.last_error()
    b, hist = problems.rhs_normal(A.n, 2), np.zeros(60)
    for _ in range(2):
        x = np.zeros(A.n)
        assert L.parcel_b_start(h, b.ctypes.data, x.ctypes.data, hist.ctypes.data, C.byref(n), C.byref(i)) < 0
        assert "gave up waiting" in _lib.last_error()
    assert L.parcel_b_release(h) == 0


@pytest.mark.parametrize("ilu", [0, 1])
def test_plan_keeps_levels_that_the_sweep_can_take(ilu):
    """A chain of 2,500 rows, a row hanging on each, and the 84 rows at the end that are all those rows'
    only dependents: moved late they would form one level of 2,500 rows of 30 couplings, which no
    sweep takes, for a gap shorter by one."""
    m, per = 2500, 30
    chain = np.arange(m)
    side = m + chain
    end = 2 * m + 1 + chain // per
    last = np.unique(end)
    r = np.concatenate([chain[:-1], chain, side, [2 * m], last])
    c = np.concatenate([chain[1:], side, end, [2 * m + 1], np.full(last.size, m - 1)])
    A = _from_pairs(int(last[-1]) + 1, np.concatenate([r, c]), np.concatenate([c, r]), 4)
    assert _apply_both(A, ipreflag=2, ILU_method=ilu, precon_thblock=1) < 1e-11
