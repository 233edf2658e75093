"""Sizes where the device code takes another path: the solve in one launch and
the separate kernels on either side of the row limit (with two colors, and with
more, whose small steps run beside the vector kernels), the factorization's
input in one and in several chunks, the allocation-free product's tiles.

Bounds. A solve stops when its recursive residual is below tol * ||b||; the
true residual differs from it by rounding, a few 1e-16 of |A||x| an iteration,
below 1e-12 * ||b|| on these systems: with tol = 1e-8 it is within 1e-8 * (1 +
1e-3). A stop after a few half-iterations leaves the oracle's iterate to
rounding, amplified by the system's condition: 1e-10. A row of a product sums
3k terms in any order with fused or separate rounding: off by at most 3k eps
sum|a||x| from the exact value, and so is the reference.
"""
import ctypes as C

import numpy as np
import pytest

from fpga_gb300 import GbIlu, load
from fpga_gb300.synth import generate
from oracle_lib import Prepared

from test_gpu_edge import random_pattern, star

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


# rows at and just above the limits of the one-launch solve: 170,000 in FP64,
# 140,000 for FP32 inner solves
@pytest.mark.parametrize("faults", [0.0, 0.002])
@pytest.mark.parametrize("precision,nx", [("fp64", 85), ("fp64", 86), ("mixed", 70), ("mixed", 71)])
def test_solves_around_the_limit(built_lib, precision, nx, faults):
    s = generate(nx, 80, 25, sigma=1.0, inactive_frac=0.0, fault_frac=faults, seed=5)
    A = s.to_scipy()
    assert s.nb == nx * 2000
    g_in = np.random.default_rng(3).standard_normal(s.n)
    with GbIlu(device=0, precision=precision) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        assert (len(np.unique(g.ordering()[1])) > 2) == (faults > 0)
        x, r = g.solve(s.b, tol=1e-8, maxit=500)
        lam, _, ra = g.adjoint(g_in, x, tol=1e-8, maxit=500, want_dA=False)
        stops = {m: g.solve(s.b, tol=1e-13, maxit=m) for m in (0, 1, 4)}
    assert r.status == 0 and ra.status == 0
    assert np.linalg.norm(s.b - A @ x) <= 1e-8 * np.linalg.norm(s.b) * (1 + 1e-3)
    assert np.linalg.norm(g_in - A.T @ lam) <= 1e-8 * np.linalg.norm(g_in) * (1 + 1e-3)
    if precision == "fp64":
        P = Prepared(s)
        for m, (x, r) in stops.items():
            x_ref, r_ref = P.solve(s.b, tol=1e-13, maxit=m)
            assert r.status == r_ref.status == 1 and r.half_iters == r_ref.half_iters, m
            assert np.linalg.norm(x - x_ref) <= 1e-10 * np.linalg.norm(x_ref), m


@pytest.mark.parametrize("numbering", ["grid", "shuffled"])
@pytest.mark.parametrize("grid", [(30, 24, 12), (60, 60, 11), (62, 60, 20)])
def test_factorization_in_chunks(built_lib, grid, numbering):
    """One, two and four chunks of input; shuffled, most rows wait for
    neighbours of a later chunk. The host's factors bit for bit."""
    s = generate(*grid, sigma=1.5, inactive_frac=0.0, fault_frac=0.01, seed=9)
    rowptr, colind, vals = s.rowptr, s.colind, s.vals.reshape(-1, 9)
    if numbering == "shuffled":
        new = np.random.default_rng(2).permutation(s.nb)   # row i becomes new[i]
        rows = np.repeat(np.arange(s.nb), np.diff(rowptr))
        order = np.lexsort((new[colind], new[rows]))
        count = np.bincount(new[rows], minlength=s.nb)
        rowptr = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
        colind = new[colind][order].astype(np.int32)
        vals = np.ascontiguousarray(vals[order])
    vals = vals.reshape(s.vals.shape)
    with GbIlu(device=0, factor_on_device=True) as d, GbIlu(device=0) as h:
        d.analyze(rowptr, colind)
        h.analyze(rowptr, colind)
        for v in (vals, vals * 1.25):
            d.factor(v)
            h.factor(v)
            for a, b in zip(d.factors(), h.factors()):
                assert np.array_equal(a, b)


@pytest.mark.parametrize("make", [lambda: random_pattern(1, 0.0, seed=1),
                                  lambda: random_pattern(31, 0.2, seed=2),
                                  lambda: random_pattern(32, 0.2, seed=3),
                                  lambda: random_pattern(33, 0.2, seed=4),
                                  lambda: random_pattern(290, 0.97, seed=5),   # tiles above 8,000 blocks
                                  lambda: star(700, seed=6)],                  # one row of 700 blocks
                         ids=["1", "31", "32", "33", "nearly_dense", "hub"])
def test_product_with_its_dot(built_lib, make):
    torch = pytest.importorskip("torch")
    s = make()
    A = s.to_scipy()
    rng = np.random.default_rng(8)
    x, w = rng.standard_normal(s.n), rng.standard_normal(s.n)
    f = load().gbilu_bsr_spmv_dot_noalloc
    f.argtypes = [C.c_int] + [C.c_void_p] * 8
    dev = torch.device("cuda:0")
    rp, ci, va, xd, wd = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in
                          (s.rowptr.astype(np.int32), s.colind.astype(np.int32),
                           s.vals.reshape(-1), x, w))
    outs = []
    for _ in range(2):
        y = torch.full((s.n,), float("nan"), dtype=torch.float64, device=dev)
        dot = torch.full((1,), float("nan"), dtype=torch.float64, device=dev)
        torch.cuda.synchronize(dev)
        assert f(s.nb, rp.data_ptr(), ci.data_ptr(), va.data_ptr(), xd.data_ptr(), y.data_ptr(),
                 wd.data_ptr(), dot.data_ptr(), torch.cuda.current_stream(dev).cuda_stream) == 0
        torch.cuda.synchronize(dev)
        outs.append((y.cpu().numpy(), float(dot.cpu())))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
    y, d = outs[0]
    size = abs(A) @ abs(x)                       # sum |a||x| of each row
    terms = np.repeat(3 * np.diff(s.rowptr), 3)
    assert np.all(np.abs(y - A @ x) <= 2 * EPS * terms * size)
    bound = 2 * EPS * (np.sum(np.abs(w) * terms * size) + s.n * np.sum(np.abs(w) * size))
    assert abs(d - np.dot(A @ x, w)) <= bound
