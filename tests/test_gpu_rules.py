"""Patterns other than 7-point grids at the sizes where the solve takes another
path: large colors beside the vector kernels or in launches of their own, a
solve in one launch or by the separate kernels; and 7-point grids where the
apply of two colors does.

Bounds: a solve's recursive residual is below tol * ||b||, the true one within
1e-3 of that (rounding is a few 1e-16 of |A||x| an iteration); operators to
1e-12 of the oracle's, as everywhere.
"""
import numpy as np
import pytest

from fpga_gb300 import GbIlu
from fpga_gb300.synth import BlockSystem, generate
from oracle_lib import Prepared

pytestmark = pytest.mark.gpu


def stencil(grid, keep, seed=0):
    """A grid coupled over the offsets (dz, dy, dx) in -1..1 that keep() takes,
    blocks and diagonals as in fpga_gb300.synth."""
    nx, ny, nz = grid
    nb = nx * ny * nz
    idx = np.arange(nb).reshape(nz, ny, nx)
    cut = lambda d, n: (slice(max(0, -d), n - max(0, d)), slice(max(0, d), n - max(0, -d)))
    ei, ej = [], []
    for d in np.ndindex(3, 3, 3):
        dz, dy, dx = (int(v) - 1 for v in d)
        if (dz, dy, dx) > (0, 0, 0) and keep(dz, dy, dx):
            z, y, x = cut(dz, nz), cut(dy, ny), cut(dx, nx)
            ei.append(idx[z[0], y[0], x[0]].ravel())
            ej.append(idx[z[1], y[1], x[1]].ravel())
    ei, ej = np.concatenate(ei), np.concatenate(ej)
    rng = np.random.default_rng(seed)
    t = np.exp(rng.standard_normal(ei.size))[:, None, None]
    bij, bji = (-t * (0.1 * rng.standard_normal((ei.size, 3, 3)) + np.eye(3)) for _ in range(2))
    diag = np.tile(0.5 * np.eye(3), (nb, 1, 1))
    for at, blk in ((ei, bij), (ej, bji)):
        for e in np.ndindex(3, 3):
            diag[:, e[0], e[1]] -= np.bincount(at, weights=blk[:, e[0], e[1]], minlength=nb)
    rows = np.concatenate([ei, ej, np.arange(nb)])
    cols = np.concatenate([ej, ei, np.arange(nb)])
    order = np.lexsort((cols, rows))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nb))]).astype(np.int32)
    return BlockSystem(nb=nb, rowptr=rowptr, colind=cols[order].astype(np.int32),
                       vals=np.ascontiguousarray(np.concatenate([bij, bji, diag])[order]),
                       b=rng.standard_normal(3 * nb), cell_of_row=np.arange(nb), grid=grid)


def layers(grid):   # nine points in a layer, two across: six colors, four of them large
    return stencil(grid, lambda z, y, x: z == 0 or (y == 0 and x == 0))


def check(s, g):
    """Forward and adjoint solve; the kernels an iteration of each launched."""
    A = s.to_scipy()
    n = np.linalg.norm(s.b)
    per_iter = []
    x, r = g.solve(s.b, tol=1e-6, maxit=500)
    per_iter.append(g.stats()["last_launches"] / (r.half_iters / 2 + 1))
    assert r.status == 0 and np.linalg.norm(s.b - A @ x) <= 1e-6 * n * (1 + 1e-3)
    lam, _, r = g.adjoint(s.b, s.b, tol=1e-6, maxit=500, want_dA=False)
    per_iter.append(g.stats()["last_launches"] / (r.half_iters / 2 + 1))
    assert r.status == 0 and np.linalg.norm(s.b - A.T @ lam) <= 1e-6 * n * (1 + 1e-3)
    return per_iter


# 12,300 and 13,300 rows a small step (the adjoint's limit between them), 23,400
# and 24,300 (the forward one's)
@pytest.mark.parametrize("nz,beside", [(27, (True, True)), (29, (True, False)),
                                       (51, (True, False)), (53, (False, False))])
def test_large_colors(built_lib, nz, beside):
    s = layers((60, 60, nz))
    with GbIlu(device=0, factor_on_device=True, one_launch=False) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        per_iter = check(s, g)
    # 7 kernels an iteration against 23, a few for the start and the end
    assert tuple(p < 15 for p in per_iter) == beside, per_iter


def points27(grid):   # eight large colors and two small ones
    return stencil(grid, lambda z, y, x: True)


# blocks below and above the limit of the colors and the precision
@pytest.mark.parametrize("precision,make,grid,one", [
    ("fp64", layers, (60, 60, 30), True), ("fp64", layers, (60, 60, 31), False),
    ("mixed", layers, (60, 60, 18), True), ("mixed", layers, (60, 60, 19), False),
    ("mixed", points27, (36, 36, 34), True), ("mixed", points27, (36, 36, 35), False),
    ("fp64", points27, (46, 46, 42), True), ("fp64", points27, (46, 46, 43), False)],
    ids=lambda v: v if isinstance(v, str) else getattr(v, "__name__", str(v)))
def test_one_launch_or_not(built_lib, precision, make, grid, one):
    s = make(grid)
    with GbIlu(device=0, factor_on_device=True, precision=precision) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        check(s, g)
        assert (g.stats()["launches_per_iter"] == 0) == one


# slices of a color for each of 152 x 16 warps: 0.597, 0.617, 0.98, 1.02, 1.23, 1.27
@pytest.mark.parametrize("nx,kernels", [(31, 2), (32, 1), (51, 1), (53, 2), (64, 2), (66, 1)])
def test_apply_of_two_colors(built_lib, nx, kernels):
    s = generate(nx, 60, 50, sigma=1.0, seed=4)
    P = Prepared(s)
    p = np.random.default_rng(5).standard_normal(s.n)
    out = []
    for sweep_mode in (1, 0):
        with GbIlu(device=0, factor_on_device=True, sweep_mode=sweep_mode) as g:
            g.analyze(s.rowptr, s.colind).factor(s.vals)
            for transpose in (False, True):
                z = g.ilu_apply(p, transpose)
                # beside the start's and the two permutations of the vectors
                assert g.stats()["last_launches"] - 3 == (2 if sweep_mode == 0 else kernels) + \
                    (1 if transpose and (sweep_mode == 0 or kernels == 2) else 0)
                z_ref = P.ilu_apply(p, transpose)
                assert np.linalg.norm(z - z_ref) <= 1e-12 * np.linalg.norm(z_ref)
                out.append(z)
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])


def test_kernel_timings_follow_the_small_steps(built_lib):
    """gbilu_bench_kernel counts the small colors' steps where they run: beside
    update_s and update_p, or (no cooperative launches) in the apply. The
    iteration's bytes are the same either way."""
    s = generate(30, 24, 12, sigma=1.5, inactive_frac=0.05, fault_frac=0.01, seed=7)
    got = []
    for options in (dict(), dict(one_launch=False, sweep_mode=0)):
        with GbIlu(device=0, factor_on_device=True, **options) as g:
            g.analyze(s.rowptr, s.colind).factor(s.vals)
            r = {k: g.bench_kernel(k + "64", reps=5) for k in ("apply", "update_s", "update_r", "update_p")}
            assert all(ms > 0 for ms, _, _ in r.values())
            got.append(({k: by for k, (_, by, _) in r.items()}, {k: la for k, (_, _, la) in r.items()},
                        g.stats()["alg_bytes_iter"][0]))
            # the handle solves as before
            x, res = g.solve(s.b, tol=1e-6, maxit=500)
            assert res.status == 0
    (beside, la, total), (inside, la0, total0) = got
    small = inside["apply"] - beside["apply"]
    assert small > 0 and total == total0 and beside["update_r"] == inside["update_r"]
    assert beside["update_s"] - inside["update_s"] == small == beside["update_p"] - inside["update_p"]
    assert set(la.values()) == {1} and la0["apply"] > 1
