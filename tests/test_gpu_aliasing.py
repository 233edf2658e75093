"""Device arrays that the caller passes twice: lambda written over x (the
forward solution that dL/dA is formed with) or over g, x written over b. The
same bits as with arrays of their own, on both sides of the size up to which
a solve is one launch, which reads and writes the caller's arrays itself.
"""
import numpy as np
import pytest

from fpga_gb300 import GbIlu
from fpga_gb300.synth import generate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [(13, 11, 7), (86, 80, 25)])
def test_arrays_passed_twice(built_lib, grid, precision):
    torch = pytest.importorskip("torch")
    s = generate(*grid, sigma=1.0, inactive_frac=0.0, fault_frac=0.002, seed=5)
    rng = np.random.default_rng(6)
    g0, x0 = (torch.from_numpy(rng.standard_normal(s.n)).cuda() for _ in range(2))

    def new(v=None):
        t = torch.full_like(x0, float("nan")) if v is None else v.clone()
        torch.cuda.synchronize()
        return t

    with GbIlu(device=0, precision=precision) as h:
        h.analyze(s.rowptr, s.colind).factor(s.vals)

        def adjoint(g, x, lam):
            dA = torch.full((9 * s.nnzb,), float("nan"), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            r = h.adjoint_device(g.data_ptr(), x.data_ptr(), lam.data_ptr(), dA.data_ptr(),
                                 tol=1e-6, maxit=500)
            assert r.status == 0
            return lam.cpu().numpy(), dA.cpu().numpy()

        lam, dA = adjoint(new(g0), new(x0), new())
        t = new(x0)
        over_x = adjoint(new(g0), t, t)
        t = new(g0)
        over_g = adjoint(t, new(x0), t)
        # lambda three entries behind x in one allocation
        t = torch.cat([new(x0), torch.zeros(3, dtype=torch.float64, device="cuda")])
        shifted = adjoint(new(g0), t[:-3], t[3:])
        for a, b in (over_x, over_g, shifted):
            assert np.array_equal(a, lam) and np.array_equal(b, dA)

        def solve(b, x):
            r = h.solve_device(b.data_ptr(), x.data_ptr(), 1e-6, 500)
            assert r.status == 0
            return x.cpu().numpy()

        x = solve(new(g0), new(g0))     # from x0 = b
        t = new(g0)
        assert np.array_equal(solve(t, t), x)
