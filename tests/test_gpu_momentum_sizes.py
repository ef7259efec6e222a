"""The momentum sweeps at the sizes where they change form: strips of 30
columns, one element, two elements or 16 bytes a lane, several rows a warp.
With momentumTol 0 both the GPU and the oracle run exactly maxMomentumIter
sweeps, so the results differ by rounding alone."""
import numpy as np
import pytest

from _helpers import gpu_for, oracle_for
from coldplate_b200 import cases

pytestmark = pytest.mark.gpu
SWEEPS = 5


@pytest.mark.parametrize("Ny,Nx", [(4, 8), (9, 30), (30, 31), (31, 32), (64, 61), (127, 253), (241, 517), (300, 900)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_sweeps_match_the_oracle(Ny, Nx, prec):
    case = cases.density_field(Ny, Nx, seed=3)
    over = dict(momentumTol=0.0, maxMomentumIter=SWEEPS)
    o = oracle_for(case, **over)
    o.run(3)
    u, v, p = o.get("u"), o.get("v"), o.get("p")
    o.momentum(True)
    o.momentum(False)
    with gpu_for(case, precision=prec, **over) as g:
        for f, a in (("u", u), ("v", v), ("p", p)):
            g.set(f, a)
        assert g.solveUMomentumImplicit()[0] == SWEEPS
        assert g.solveVMomentumImplicit()[0] == SWEEPS
        for f, x in (("uStar", u), ("vStar", v)):
            # a sweep rounds at most 16 terms no larger than twice the change it makes
            eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
            # (the calls write the unknowns; the boundary values are the outer iteration's)
            on = (slice(1, -1), slice(1, -1))
            a, b, x0 = g.get(f)[on], o.get(f)[on], x[on]
            scale = np.abs(b - x0).max() + (np.abs(x0).max() if prec == "fp64" else 0.0)
            assert np.abs(a - b).max() <= 32 * SWEEPS * eps * scale, f
