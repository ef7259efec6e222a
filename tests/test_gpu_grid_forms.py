"""The passes on every SM at sizes that no cluster takes (rows a CTA of 16, rounded
up, times the unknowns of a row above 3072): strips of 30 columns of one element,
two floats or 16 bytes a lane, both components of the momentum at once, and one
after the other."""
import numpy as np
import pytest

from _helpers import gpu_for, oracle_for
from coldplate_b200 import cases
from test_gpu_pressure_cluster import cg
from test_gpu_pressure_sa_sizes import gpu_solve, system

pytestmark = pytest.mark.gpu
SWEEPS = 5

# one element a lane, with 1559 .. 1562 unknowns a row around a whole number of
# strips; two floats (one strip of doubles); 16 bytes; one component after the
# other in double (two components of 76 MB each do not fit the L2)
SIZES = [(17, 1559), (17, 1560), (17, 1561), (18, 1562), (48, 1100), (300, 901), (900, 1300)]


@pytest.mark.parametrize("Ny,Nx", SIZES)
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_sweeps_match_the_oracle(Ny, Nx, prec):
    """With momentumTol 0 both the GPU and the oracle run exactly maxMomentumIter
    sweeps: one component by its own call, both within an iteration."""
    over = dict(momentumTol=0.0, maxMomentumIter=SWEEPS, pressureSolverType=1, maxPressureIter=3)
    case = cases.density_field(Ny, Nx, seed=3)
    o = oracle_for(case, **over)
    o.run(2)
    x = {f: o.get(f) for f in ("u", "v", "p")}
    o.momentum(True)
    o.momentum(False)
    # a sweep rounds at most 16 terms no larger than twice the change it makes
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    on = (slice(1, -1), slice(1, -1))
    with gpu_for(case, precision=prec, **over) as g:
        for whole in (False, True):
            g.reset()
            for f, a in x.items():
                g.set(f, a)
            if whole:
                r = g.step(1)
                assert (r["momentumItersU"], r["momentumItersV"]) == (SWEEPS, SWEEPS)
            else:
                assert g.solveUMomentumImplicit()[0] == SWEEPS
                assert g.solveVMomentumImplicit()[0] == SWEEPS
            for f, x0 in (("uStar", x["u"][on]), ("vStar", x["v"][on])):
                a, b = g.get(f)[on], o.get(f)[on]
                scale = np.abs(b - x0).max() + (np.abs(x0).max() if prec == "fp64" else 0.0)
                assert np.abs(a - b).max() <= 32 * SWEEPS * eps * scale, (whole, f)


@pytest.mark.parametrize("Ny,Nx", SIZES[:-1] + [(90, 1100)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_jacobi_pcg_iterates(Ny, Nx, prec):
    """A set number of iterations against the same recurrences in numpy: an
    iterate moves by roundings, amplified by the few thousand that the
    iteration's coefficients span."""
    its = 8
    fields, _, A, b = system(Ny, Nx)
    it, x = gpu_solve(Ny, Nx, fields, pressureSolverType=1, maxPressureIter=its, pTol=0.0, precision=prec)
    y, _ = cg(A, b, its)
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    assert it == its
    assert np.linalg.norm(x - y) <= 1e4 * its * eps * np.linalg.norm(y)
