"""A one-launch solve whose grid barrier runs out (one CTA more is waited for
than there is; the poll limit is short, so it ends at once without a GPU
fault): the call returns TIMEOUT, what it leaves is defined, and the handle's
next calls are those of a fresh handle, bit for bit."""
import numpy as np
import pytest

from fpga_gb300 import GbIlu, GbIluError
from fpga_gb300.synth import generate

pytestmark = pytest.mark.gpu

TIMEOUT = 5


@pytest.fixture(scope="module")
def system(built_lib):
    return generate(20, 18, 9, sigma=1.5, inactive_frac=0.05, fault_frac=0.02, seed=3)


def test_solve_and_adjoint(system):
    torch = pytest.importorskip("torch")
    s = system
    x0 = np.random.default_rng(1).standard_normal(s.n)
    with GbIlu(device=0) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        x_ref, r_ref = g.solve(s.b, tol=1e-6, maxit=500)
        lam_ref, dA_ref, _ = g.adjoint(s.b, x_ref, tol=1e-6, maxit=500)
        dev = [torch.from_numpy(v).cuda() for v in (s.b, x_ref)]
        for again in range(2):
            g.wait_probe(2)
            x, r = g.solve(s.b, tol=1e-6, maxit=500)
            assert r.status == TIMEOUT and not x.any()
            g.wait_probe(2)
            x, r = g.solve(s.b, x0=x0, tol=1e-6, maxit=500)
            assert r.status == TIMEOUT and np.array_equal(x, x0)
            g.wait_probe(2)
            lam, dA, r = g.adjoint(s.b, x_ref, tol=1e-6, maxit=500)
            assert r.status == TIMEOUT and not lam.any() and not dA.any()
            g.wait_probe(2)
            out = [torch.full((k,), float("nan"), dtype=torch.float64, device="cuda")
                   for k in (s.n, 9 * s.nnzb)]
            torch.cuda.synchronize()
            r = g.adjoint_device(dev[0].data_ptr(), dev[1].data_ptr(), out[0].data_ptr(),
                                 out[1].data_ptr(), tol=1e-6, maxit=500)
            assert r.status == TIMEOUT and not any(bool(t.any()) for t in out)
            # the next ones are untouched by it
            x, r = g.solve(s.b, tol=1e-6, maxit=500)
            assert r.status == 0 and r.half_iters == r_ref.half_iters and np.array_equal(x, x_ref)
            lam, dA, r = g.adjoint(s.b, x_ref, tol=1e-6, maxit=500)
            assert r.status == 0 and np.array_equal(lam, lam_ref) and np.array_equal(dA, dA_ref)


def test_mixed(system):
    s = system
    A = s.to_scipy()
    with GbIlu(device=0, precision="mixed") as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        x_ref, _ = g.solve(s.b, tol=1e-8, maxit=500)
        g.wait_probe(2)
        x, r = g.solve(s.b, tol=1e-8, maxit=500)
        assert r.status == TIMEOUT and r.outer_iters == 1
        # the reported residual is that of the x that is returned
        true = np.linalg.norm(s.b - A @ x) / np.linalg.norm(s.b)
        assert abs(true - r.true_relres) <= 1e-10
        x, r = g.solve(s.b, tol=1e-8, maxit=500)
        assert r.status == 0 and np.array_equal(x, x_ref)


def test_waits_of_other_kernels_leave_no_mark(system):
    """The marks of waits that ran out elsewhere (modes 0 and 1) do not reach
    a one-launch solve, and a handle without one refuses mode 2."""
    s = system
    with GbIlu(device=0) as g:
        g.analyze(s.rowptr, s.colind).factor(s.vals)
        x_ref, _ = g.solve(s.b, tol=1e-6, maxit=500)
        g.wait_probe(1)
        x, r = g.solve(s.b, tol=1e-6, maxit=500)
        assert r.status == 0 and np.array_equal(x, x_ref)
    one_color = type(s)(nb=40, rowptr=np.arange(41, dtype=np.int32),
                        colind=np.arange(40, dtype=np.int32), vals=np.tile(2 * np.eye(3), (40, 1, 1)),
                        b=np.ones(120), cell_of_row=np.arange(40), grid=(40, 1, 1))
    with GbIlu(device=0) as g:
        g.analyze(one_color.rowptr, one_color.colind).factor(one_color.vals)
        with pytest.raises(GbIluError):
            g.wait_probe(2)
