"""The thermal solve where its passes change form: tiles of whole columns at
and around their width (256 / Nz columns), odd edges of the aggregation, levels
of one row or column, the smallest and the most layers, and hierarchies whose
first coarse level is already solved by its matrix."""
import numpy as np
import pytest

from test_gpu_thermal import inputs, oracle_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ny,Nx,nzs,nzf", [(2, 2, 1, 1), (2, 64, 1, 1), (2, 65, 2, 7), (37, 2, 1, 3), (5, 17, 8, 8),
                                           (4, 7, 2, 7), (8, 16, 1, 7), (9, 15, 8, 4), (33, 31, 2, 7), (40, 63, 3, 4)])
@pytest.mark.parametrize("prec", [0, 1])
def test_temperature_and_gradient_at_every_tile_form(Ny, Nx, nzs, nzf, prec):
    from coldplate_b200 import Thermal
    from thermal_oracle import pnorm_gradient, solve
    gam, u, v, q0 = inputs(Ny, Nx, 5, "graded")
    prm = dict(Nx=Nx, Ny=Ny, nz_solid=nzs, nz_fluid=nzf, dx=2e-5, dy=2e-5, H_t=2e-4, rtol=1e-12, maxiter=5000)
    To = solve(oracle_params(**prm), gam, u, v, q0)
    Jo, go, _, _ = pnorm_gradient(oracle_params(**prm), gam, u, v, q0, 8.0)
    with Thermal(precision=prec, **prm) as th:
        th.set_inputs(gam, u, v, q0)
        assert th.solve()["converged"]
        T = th.T
        J, g, rep = th.pnorm_gradient(8)
    assert rep["converged"]
    # the bounds of the oracle comparisons at one size
    assert np.linalg.norm(T - To) <= 1e-9 * np.linalg.norm(To)
    assert abs(J - Jo) <= 1e-9 * Jo
    assert np.abs(g - go).max() <= 1e-8 * np.abs(go).max()
