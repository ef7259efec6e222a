"""The adjoint's products on both sides of the size from which their target is
cleared by a launch of its own instead of by the kernel that reads it: the
residual that the solve reports is that of a product made afresh."""
import numpy as np
import pytest

from _helpers import gpu_for
from coldplate_b200 import cases

pytestmark = pytest.mark.gpu


# three fields of 0.03, 3.2, 4.2 and 7.1 MB (the line is at 4)
@pytest.mark.parametrize("Ny,Nx", [(24, 40), (256, 512), (300, 570), (384, 768)])
@pytest.mark.parametrize("solver", [1, 4])
def test_reported_residual(Ny, Nx, solver):
    case = cases.density_field(Ny, Nx, seed=2)
    with gpu_for(case, pressureSolverType=solver, pTol=1e-6, precision="fp64") as g:
        g.step(30)
        dj, _ = g.adjoint_probe(1)
        lam, meta = g.adjoint_probe(2, max_iter=45, tol=1e-14)
        y, _ = g.adjoint_probe(0, lam)
        gn = np.sqrt(sum((a * a).sum() for a in dj.values()))
        r = np.sqrt(sum(((dj[f] - y[f]) ** 2).sum() for f in dj)) / gn
        # one rounding a term (at most 30 of a row) of J^T lambda, and of the sum of squares
        scale = np.sqrt(sum((a * a).sum() for a in y.values())) / gn
        assert abs(r - meta["residual"]) <= 64 * 2.0 ** -53 * max(scale, 1.0) * 10 + 1e-12 * r, (r, meta)
        assert meta["iterations"] == 45 or meta["converged"]
