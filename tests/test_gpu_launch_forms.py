"""The separate kernels of large systems on small ones (one_launch = 0): a
graph or host-driven launches, small colors beside the vector kernels, in the
apply's launch or in launches of their own, staged or not, with or without
the ring. Ragged slices, a hub, a dozen small colors, more colors than the
step list holds, and a grid whose large steps pass the staging limit.

Bounds as for the one-launch form: the true residual is below
tol * ||r0|| * (1 + 1e-3) (the recursive one stops the run, rounding adds a few
1e-16 of |A||x| an iteration); a stop after a few half-iterations leaves the
oracle's iterate to rounding times the system's condition, 1e-10. Forms that
add the same numbers in the same order agree bit for bit.
"""
import numpy as np
import pytest

from fpga_gb300 import GbIlu
from fpga_gb300.synth import generate
from oracle_lib import Prepared

from test_gpu_edge import dense
from test_gpu_reduced import CASES, right_hand_sides

pytestmark = pytest.mark.gpu

SYSTEMS = dict(CASES, above_the_step_list=lambda: dense(50, seed=4),
               large_steps=lambda: generate(60, 60, 20, sigma=1.5, inactive_frac=0.05,
                                            fault_frac=0.01, seed=5))


@pytest.fixture(scope="module", params=sorted(SYSTEMS))
def system(request, built_lib):
    s = SYSTEMS[request.param]()
    return request.param, s, s.to_scipy()


def handle(s, **options):
    g = GbIlu(device=0, **options)
    g.analyze(s.rowptr, s.colind).factor(s.vals)
    return g


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_option_chooses(system, precision):
    name, s, _ = system
    for one in (True, False):
        with handle(s, precision=precision, one_launch=one) as g:
            g.solve(s.b, tol=1e-4, maxit=500)
            separate = g.stats()["launches_per_iter"] > 0
            assert separate == (not one or name == "above_the_step_list")


@pytest.mark.parametrize("options", [dict(), dict(sweep_mode=0), dict(use_graph=False),
                                     dict(precision="mixed"),
                                     dict(precision="mixed", sweep_mode=0, use_graph=False)],
                         ids=lambda o: "-".join(f"{k}={v}" for k, v in o.items()) or "default")
def test_right_hand_sides(system, options):
    name, s, A = system
    x0 = np.random.default_rng(5).standard_normal(s.n)
    with handle(s, one_launch=False, **options) as g:
        for what, b in right_hand_sides(s, g.ordering()[1]).items():
            n = np.linalg.norm(b)
            x, r = g.solve(b, tol=1e-8, maxit=500)
            assert r.status == 0 and np.linalg.norm(b - A @ x) <= 1e-8 * n * (1 + 1e-3), what
            x, r = g.solve(b, x0=x0, tol=1e-8, maxit=500)
            assert r.status == 0, what
            assert np.linalg.norm(b - A @ x) <= 1e-8 * np.linalg.norm(b - A @ x0) * (1 + 1e-3), what
            lam, _, r = g.adjoint(b, b, tol=1e-8, maxit=500, want_dA=False)
            assert r.status == 0 and np.linalg.norm(b - A.T @ lam) <= 1e-8 * n * (1 + 1e-3), what


@pytest.mark.parametrize("sweep_mode", [0, 1])
def test_stops_leave_the_iterate(system, sweep_mode):
    name, s, _ = system
    P = Prepared(s)
    x0 = np.random.default_rng(6).standard_normal(s.n)
    with handle(s, one_launch=False, sweep_mode=sweep_mode) as g:
        for maxit in (0, 1, 4):
            x, r = g.solve(s.b, x0=x0, tol=1e-13, maxit=maxit)
            x_ref, r_ref = P.solve(s.b, x0=x0, tol=1e-13, maxit=maxit)
            if r_ref.status == 1:
                assert r.status == 1 and r.half_iters == r_ref.half_iters
            assert np.linalg.norm(x - x_ref) <= 1e-10 * np.linalg.norm(x_ref)


# forms of the same sums
SAME = {"fp64": [dict(), dict(use_graph=False), dict(stage_small_steps=False),
                 dict(stream_large_steps=True)],
        "fp64 by steps": [dict(sweep_mode=0), dict(sweep_mode=0, use_graph=False)],
        "mixed": [dict(), dict(use_graph=False), dict(sweep_mode=0), dict(stage_small_steps=False),
                  dict(stream_large_steps=True), dict(sweep_mode=0, use_graph=False)]}


@pytest.mark.parametrize("which", sorted(SAME))
def test_same_bits(system, which):
    name, s, _ = system
    precision = which.split()[0]
    gv = np.random.default_rng(9).standard_normal(s.n)
    ref = None
    for options in SAME[which]:
        with handle(s, precision=precision, one_launch=False, **options) as g:
            x, r = g.solve(s.b, tol=1e-6, maxit=500)
            lam, dA, ra = g.adjoint(gv, x, tol=1e-6, maxit=500)
        got = (x, lam, dA, r.half_iters, r.inner_half_iters, ra.half_iters)
        if ref is None:
            ref = got
        assert got[3:] == ref[3:], options
        assert all(np.array_equal(a, b) for a, b in zip(got[:3], ref[:3])), options
