"""The Jacobi-PCG on one cluster at its edges: exactly 512, 1024, 2048 and 3072
unknowns a CTA and one more, CTAs without rows, blocks of one row, the last
block short; and the exits."""
import numpy as np
import pytest

from test_gpu_pressure_sa_sizes import gpu_solve, system

pytestmark = pytest.mark.gpu


def cg(A, b, its):
    d = A.diagonal()
    y, r = np.zeros_like(b), b.copy()
    z = r / d
    p, rz, rr = z.copy(), r @ z, []
    for _ in range(its):
        Ap = A @ p
        a = rz / (p @ Ap)
        y += a * p
        r -= a * Ap
        z = r / d
        rr.append(np.sqrt(r @ r))
        p, rz = z + (r @ z) / rz * p, r @ z
    return y, rr


@pytest.mark.parametrize("Ny,Nx", [(5, 9), (16, 513), (16, 514), (15, 1025), (17, 40), (300, 3), (32, 1025), (33, 1025),
                                   (33, 1026), (100, 400)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_cluster_pcg_iterates(Ny, Nx, prec):
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


def test_cluster_pcg_exits():
    fields, _, A, b = system(40, 61)
    y, rr = cg(A, b, 12)
    # stops behind the first residual under the tolerance, with that step taken
    low = [k for k in range(1, 12) if rr[k] < min(rr[:k])][-1]
    it, x = gpu_solve(40, 61, fields, pressureSolverType=1, maxPressureIter=30, pTol=rr[low] * 1.0001, precision="fp64")
    assert it == low
    y, _ = cg(A, b, low + 1)
    assert np.linalg.norm(x - y) <= 1e4 * 12 * 2.0 ** -53 * np.linalg.norm(y)
    # nothing to solve: no step, zero correction
    for f in ("uStar", "vStar"):
        fields[f] = np.zeros_like(fields[f])
    it, x = gpu_solve(40, 61, fields, pressureSolverType=1, maxPressureIter=30, pTol=1e-6, precision="fp64")
    assert it == 0 and not x.any()
    it, x = gpu_solve(40, 61, fields, pressureSolverType=1, maxPressureIter=0, pTol=1e-6, precision="fp64")
    assert it == 0 and not x.any()
