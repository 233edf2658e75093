"""The reduced iteration (color 0 eliminated from every vector of BiCGSTAB):
right-hand sides that meet its special cases, against the CPU oracle's
operators.

On color 0's rows every vector is a multiple of the initial residual, so the
cases are the right-hand sides that are zero there, zero everywhere else (the
iteration then restarts after one step: (r, rt) is zero), one entry of either
kind, and general ones, from x0 = 0 and from a start vector. Bound: the
solver stops when its recursive residual is below tol * ||r0||; the true
residual b - A x differs from the recursive one by rounding, a few 1e-16 of
|A||x| an iteration, i.e. below 1e-12 * ||b|| on these systems, so with
tol = 1e-8 it is within 1e-8 * (1 + 1e-3).
"""
import numpy as np
import pytest

from fpga_gb300 import GbIlu
from fpga_gb300.synth import generate, make_config
from oracle_lib import Prepared

from test_gpu_edge import random_pattern, star

pytestmark = pytest.mark.gpu

CASES = {
    "two_colors": lambda: make_config("c1_20x20x10"),
    "faults": lambda: generate(30, 24, 12, sigma=1.5, inactive_frac=0.05, fault_frac=0.01, seed=7),
    # partly filled slices, an odd number of rows in every color
    "ragged": lambda: generate(13, 11, 7, sigma=1.0, inactive_frac=0.05, fault_frac=0.02, seed=3),
    "many_colors": lambda: random_pattern(300, 0.08, seed=6),
    "star": lambda: star(33, seed=3),
}


@pytest.fixture(scope="module", params=sorted(CASES))
def case(request, built_lib):
    s = CASES[request.param]()
    return s, s.to_scipy()


def right_hand_sides(s, color):
    rng = np.random.default_rng(4)
    head = np.repeat(color == 0, 3)
    b = rng.standard_normal(s.n)
    one_head, one_tail = np.zeros(s.n), np.zeros(s.n)
    one_head[np.nonzero(head)[0][-1]] = 1.0
    one_tail[np.nonzero(~head)[0][0]] = -2.0
    return {"general": b, "head only": np.where(head, b, 0.0), "tail only": np.where(head, 0.0, b),
            "one head entry": one_head, "one tail entry": one_tail,
            "small tail": np.where(head, b, 1e-9 * b)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("transpose", [False, True])
def test_right_hand_sides(case, precision, transpose):
    s, A = case
    M = A.T.tocsr() if transpose else A
    x0 = np.random.default_rng(5).standard_normal(s.n)
    with GbIlu(device=0, precision=precision) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        _, color, _, _ = g.ordering()
        for name, b in right_hand_sides(s, color).items():
            if transpose:
                x, _, r = g.adjoint(b, b, tol=1e-8, maxit=500, want_dA=False)
                r0 = np.linalg.norm(b)
            else:
                x, r = g.solve(b, tol=1e-8, maxit=500)
                r0 = np.linalg.norm(b)
            assert r.status == 0, (name, r.status)
            assert np.linalg.norm(b - M @ x) <= 1e-8 * r0 * (1 + 1e-3), name
            if not transpose:
                x, r = g.solve(b, x0=x0, tol=1e-8, maxit=500)
                r0 = np.linalg.norm(b - A @ x0)
                assert r.status == 0, (name, r.status)
                assert np.linalg.norm(b - A @ x) <= 1e-8 * r0 * (1 + 1e-3), name


@pytest.mark.parametrize("maxit", [0, 1, 5])
def test_stops_leave_the_iterate(case, maxit):
    """A stop after a first half (MAXIT): x is the oracle's iterate on every
    row, color 0's rebuilt from its equations included."""
    s, A = case
    P = Prepared(s)
    x0 = np.random.default_rng(6).standard_normal(s.n)
    with GbIlu(device=0) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        x, r = g.solve(s.b, x0=x0, tol=1e-13, maxit=maxit)
        x_ref, r_ref = P.solve(s.b, x0=x0, tol=1e-13, maxit=maxit)
    if r_ref.status == 1:
        assert r.status == 1 and r.half_iters == r_ref.half_iters
    assert np.linalg.norm(x - x_ref) <= 1e-10 * np.linalg.norm(x_ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_from_zero_is_the_solve_from_zeros(case, precision):
    """Without a start vector x is only written: the same bits as from an
    array of zeros, and zeros where no iteration ran, whatever x held."""
    s, A = case
    with GbIlu(device=0, precision=precision) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        x1, r1 = g.solve(s.b, tol=1e-6, maxit=500)
        x2, r2 = g.solve(s.b, x0=np.zeros(s.n), tol=1e-6, maxit=500)
        assert r1.half_iters == r2.half_iters and np.array_equal(x1, x2)
        x, r = g.solve(np.zeros(s.n), tol=1e-6, maxit=500)
        assert r.status == 2 and not x.any()
        b = s.b.copy()
        b[3] = np.inf
        x, r = g.solve(b, tol=1e-6, maxit=500)
        assert r.status == 4 and not x.any()
