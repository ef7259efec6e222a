"""Adjoint of small plates in mixed precision: the float V-cycle, whose coarsest
levels are a matrix product here, leaves BiCGStab about the iterations that the
FP64 one does."""
import numpy as np
import pytest

from coldplate_b200 import Thermal

pytestmark = pytest.mark.gpu

PLATES = [(7, 6, 8, 2), (16, 8, 6, 9), (13, 4, 5, 7), (51, 8, 8, 3), (25, 5, 7, 7), (14, 7, 6, 2), (72, 42, 6, 2), (115, 67, 6, 2)]


@pytest.mark.parametrize("Nx,Ny,solid,fluid", PLATES)
def test_mixed_adjoint_takes_about_the_iterations_of_fp64(Nx, Ny, solid, fluid):
    total = [0, 0]
    for seed in range(6):
        rng = np.random.default_rng(seed)
        gamma = (rng.random((Ny, Nx)) > 0.4).astype(float) if seed % 2 else np.ones((Ny, Nx))
        u = 0.3 * rng.random((Ny, Nx)) * gamma
        for prec in (0, 1):
            with Thermal(Nx=Nx, Ny=Ny, nz_solid=solid, nz_fluid=fluid, dx=1e-5, dy=2e-5, H_t=2e-4, rtol=1e-10,
                         precision=prec) as th:
                th.set_inputs(gamma, u, np.zeros_like(u), np.full((Ny, Nx), 5e5))
                assert th.solve()["converged"]
                rep = th.pnorm_gradient(8.0)[2]
            assert rep["converged"], (seed, prec, rep)
            total[prec] += rep["iterations"]
    # a float solve is restarted from its iterate up to three times until the true
    # residual meets rtol; over six systems that is well below one more solve each
    assert total[1] <= 2.0 * total[0], total
