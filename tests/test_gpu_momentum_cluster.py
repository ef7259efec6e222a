"""The momentum sweeps on clusters at their edges: exactly 512 and 2048 unknowns
a CTA and one more, CTAs without rows, a short last block, a grid just too large;
and each component's own stop.  With momentumTol 0 both the GPU and the oracle
run exactly maxMomentumIter sweeps, so the results differ by rounding alone."""
import numpy as np
import pytest

from _helpers import gpu_for, oracle_for
from coldplate_b200 import cases

pytestmark = pytest.mark.gpu
SWEEPS = 5


def start(Ny, Nx, over):
    case = cases.density_field(Ny, Nx, seed=5)
    o = oracle_for(case, **over)
    o.run(2)
    return case, o, {f: o.get(f) for f in ("u", "v", "p")}


@pytest.mark.parametrize("Ny,Nx", [(3, 8), (16, 512), (16, 513), (17, 40), (300, 9), (32, 1024), (33, 1024), (33, 1026)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_cluster_sweeps_match_the_oracle(Ny, Nx, prec):
    over = dict(momentumTol=0.0, maxMomentumIter=SWEEPS)
    case, o, fields = start(Ny, Nx, over)
    o.momentum(True)
    o.momentum(False)
    with gpu_for(case, precision=prec, **over) as g:
        for f, a in fields.items():
            g.set(f, a)
        assert g.solveUMomentumImplicit()[0] == SWEEPS
        assert g.solveVMomentumImplicit()[0] == SWEEPS
        for f, x in (("uStar", fields["u"]), ("vStar", fields["v"])):
            # a sweep rounds at most 16 terms no larger than twice the change it makes
            eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
            on = (slice(1, -1), slice(1, -1))
            a, b, x0 = g.get(f)[on], o.get(f)[on], x[on]
            scale = np.abs(b - x0).max() + (np.abs(x0).max() if prec == "fp64" else 0.0)
            assert np.abs(a - b).max() <= 32 * SWEEPS * eps * scale, f


@pytest.mark.parametrize("Ny,Nx", [(40, 80), (127, 253)])
def test_cluster_components_stop_on_their_own(Ny, Nx):
    case, o, fields = start(Ny, Nx, dict(momentumTol=1e-7))
    nU, nV = o.momentum(True)[0], o.momentum(False)[0]
    assert 1 < min(nU, nV) and nU != nV
    with gpu_for(case, precision="fp64", momentumTol=1e-7) as g:
        for f, a in fields.items():
            g.set(f, a)
        assert (g.solveUMomentumImplicit()[0], g.solveVMomentumImplicit()[0]) == (nU, nV)
