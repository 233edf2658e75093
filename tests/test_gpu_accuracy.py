"""The true residual of a solve that reports status 0, on systems whose 3x3
blocks are ill conditioned, against the CPU oracle's full iteration.

The reduced iteration (color 0 eliminated) takes A p^ = p on color 0's rows,
which holds to rounding times the condition of their diagonal blocks under
the best scaling; above a limit the solver runs the full iteration. A step's
rounding is what the oracle's own run shows: its true residual less its
recursive one. The orders of summation differ, so the bound is ten times
that, beside the tolerance itself (1 + 1e-3: recursive against true).
"""
import numpy as np
import pytest

from fpga_gb300 import GbIlu
from fpga_gb300.synth import generate
from oracle_lib import Prepared

pytestmark = pytest.mark.gpu

GRIDS = {"two_colors": dict(nx=8, ny=10, nz=12),
         "faults": dict(nx=13, ny=11, nz=7, inactive_frac=0.05, fault_frac=0.02)}


def rows_of(s):
    return np.repeat(np.arange(s.nb), np.diff(s.rowptr))


def conditioned(grid, cond, side, seed=1):
    """Every block multiplied by a dense 3x3 one of the given condition, one
    per row from the left or one per column from the right."""
    s = generate(**GRIDS[grid], sigma=1.0, seed=3)
    rng = np.random.default_rng(seed)
    q = [np.linalg.qr(rng.standard_normal((s.nb, 3, 3)))[0] for _ in range(2)]
    c = (q[0] * np.array([1.0, cond ** -0.5, 1.0 / cond])) @ q[1]
    v = c[rows_of(s)] @ s.vals if side == "left" else s.vals @ c[s.colind]
    s.vals = np.ascontiguousarray(v)
    return s


def oracle_bound(P, b, tol, transpose):
    """tol and ten times the oracle's distance between true and recursive."""
    x, r = P.solve(b, tol=tol, maxit=500, transpose=transpose)
    assert r.status == 0
    true = np.linalg.norm(b - P.spmv(x, transpose)) / np.linalg.norm(b)
    return tol * (1 + 1e-3) + 10 * abs(true - r.relres)


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("side", ["left", "right"])
@pytest.mark.parametrize("cond", [1e4, 1e6])
@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_ill_conditioned_blocks(built_lib, grid, cond, side, on_device):
    s = conditioned(grid, cond, side)
    P = Prepared(s)
    A = s.to_scipy()
    with GbIlu(device=0, factor_on_device=on_device) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        x, r = g.solve(s.b, tol=1e-10, maxit=500)
        lam, _, ra = g.adjoint(s.b, s.b, tol=1e-10, maxit=500, want_dA=False)
    n = np.linalg.norm(s.b)
    assert r.status == 0 and ra.status == 0
    assert np.linalg.norm(s.b - A @ x) <= n * oracle_bound(P, s.b, 1e-10, False)
    assert np.linalg.norm(s.b - A.T @ lam) <= n * oracle_bound(P, s.b, 1e-10, True)


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_limit(built_lib, precision, on_device):
    """One diagonal block of color 0 with a relative gain of 1 / (1 - x^2),
    just below and just above the limit of 4, then a factorization each way
    again: the path follows the values, scaled rows and columns change
    nothing, and every solve meets its tolerance."""
    s = generate(13, 11, 7, sigma=1.0, inactive_frac=0.05, fault_frac=0.02, seed=3)
    P = Prepared(s)
    i = int(np.nonzero(P.color == 0)[0][5])
    k = s.rowptr[i] + int(np.searchsorted(s.colind[s.rowptr[i]:s.rowptr[i + 1]], i))
    rng = np.random.default_rng(2)
    # powers of two: the scaled gains are the same bits
    dr, dc = (2.0 ** rng.integers(-8, 9, (s.nb, 3)) for _ in range(2))
    scale = dr[rows_of(s)][:, :, None] * dc[s.colind][:, None, :]
    with GbIlu(device=0, precision=precision, factor_on_device=on_device) as g:
        g.analyze(s.rowptr, s.colind)
        for x2, full in ((0.74, False), (0.76, True), (0.74, False), (np.nan, False), (0.76, True)):
            v = s.vals.copy()
            if np.isfinite(x2):
                # 20: the row stays dominant
                v[k] = 20 * np.array([[1, np.sqrt(x2), 0], [np.sqrt(x2), 1, 0], [0, 0, 1]])
            for w in (v, v * scale):
                g.factor(w)
                A = type(s)(**{**s.__dict__, "vals": w}).to_scipy()
                x, r = g.solve(s.b, tol=1e-6, maxit=500)
                assert (g.stats()["launches_per_iter"] > 0) == full, x2
                assert r.status == 0
                assert np.linalg.norm(s.b - A @ x) <= 1e-6 * np.linalg.norm(s.b) * (1 + 1e-3)
                lam, _, ra = g.adjoint(s.b, s.b, tol=1e-6, maxit=500, want_dA=False)
                assert ra.status == 0
                assert np.linalg.norm(s.b - A.T @ lam) <= 1e-6 * np.linalg.norm(s.b) * (1 + 1e-3)
