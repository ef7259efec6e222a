"""The pressure solvers at the sizes where their passes change form: strips of
27 and 30 lanes, one row of aggregates, the smallest grid, a coarse level of
exactly the size that is solved by its matrix, and levels large enough for two
elements a lane and for the marching passes."""
import numpy as np
import pytest
import scipy.sparse as sp

from coldplate_b200.solver import Simple
from pressure_sa import Level, galerkin, pcg, pressure_stencil, vcycle

pytestmark = pytest.mark.gpu

RHO, H = 1000.0, 1e-5


def stencil_matrix(A):
    """The stencil dict of oracle/pressure_sa.py as a sparse matrix."""
    ni, nj = A[(0, 0)].shape
    n = ni * nj
    at = np.arange(n).reshape(ni, nj)
    rows, cols, vals = [], [], []
    for (di, dj), c in A.items():
        i, j = np.meshgrid(np.arange(ni), np.arange(nj), indexing="ij")
        on = (i + di >= 0) & (i + di < ni) & (j + dj >= 0) & (j + dj < nj)
        rows.append(at[on])
        cols.append(at[i[on] + di, j[on] + dj])
        vals.append(c[on])
    return sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(n, n))


def system(Ny, Nx):
    """Random face coefficients and intermediate velocities, the matrix and rhs."""
    rng = np.random.default_rng(Ny * 1000 + Nx)
    M, N = Ny + 1, Nx + 1
    dE, dN, uS, vS = np.zeros((M + 1, N)), np.zeros((M, N + 1)), np.zeros((M + 1, N)), np.zeros((M, N + 1))
    dE[1:M, 1:N - 1] = 10.0 ** rng.uniform(-1, 0, (M - 1, N - 2))
    dN[1:M - 1, 1:N] = 10.0 ** rng.uniform(-1, 0, (M - 2, N - 1))
    uS[1:M], vS[1:M - 1, 1:N] = rng.standard_normal((M - 1, N)), rng.standard_normal((M - 2, N - 1))
    St = pressure_stencil(dE, dN, RHO, H, H)
    b = RHO * H * (uS[1:M, :-2] - uS[1:M, 1:-1] + vS[:-1, 1:-2] - vS[1:, 1:-2]).reshape(-1)
    return dict(dE=dE, dN=dN, uStar=uS, vStar=vS), St, stencil_matrix(St), b


def gpu_solve(Ny, Nx, fields, **knobs):
    with Simple(Ny=Ny, Nx=Nx, hx=H, hy=H, rho=RHO, targetVel=0.5, **knobs) as g:
        for f, a in fields.items():
            g.set(f, a)
        it, _ = g.solvePressureSystem()
        return it, g.get("pStar")[1:-1, 1:-2].reshape(-1)


@pytest.mark.parametrize("Ny,Nx", [(2, 3), (3, 82), (40, 4), (27, 28), (26, 31), (31, 30), (55, 61), (90, 109), (96, 97),
                                   (130, 247), (250, 331), (333, 700)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_sa_pcg_solves_the_system_at_every_pass_form(Ny, Nx, prec):
    fields, St, A, b = system(Ny, Nx)
    tol = 1e-6 if prec == "fp64" else 1e-4
    it, x = gpu_solve(Ny, Nx, fields, pressureSolverType=4, maxPressureIter=200, pTol=tol, precision=prec)
    rel = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
    # the recursive residual of a float CG drifts by a rounding of A x an iteration
    drift = 0.0 if prec == "fp64" else it * 2.0 ** -24 * np.linalg.norm(abs(A) @ abs(x)) / np.linalg.norm(b)
    assert it < 200 and rel <= 1.001 * tol + drift, (it, rel, drift)
    if prec == "fp64" and b.size > 64:
        levels, Al = [], St
        while Al[(0, 0)].size > 64:
            levels.append(Level(Al, 2.0 / 3.0 if not levels else 0.8))
            Al = galerkin(levels[-1])
        levels.append(Level(Al, None))
        shape = St[(0, 0)].shape
        _, it_o = pcg(St, b.reshape(shape), lambda r: vcycle(levels, r, 0.9), tol=tol, maxit=200)
        assert abs(it - it_o) <= 1, (it, it_o)


@pytest.mark.parametrize("Ny,Nx", [(2, 3), (31, 30), (30, 32), (90, 109), (130, 247), (250, 331), (333, 700)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_jacobi_pcg_iterates_at_every_pass_form(Ny, Nx, prec):
    """Type 1 after a set number of iterations against the same recurrences in
    numpy: a CG iterate moves by roundings, amplified by the few thousand that
    the iteration's coefficients span."""
    its = 10 if Ny > 2 else 2
    fields, _, A, b = system(Ny, Nx)
    it, x = gpu_solve(Ny, Nx, fields, pressureSolverType=1, maxPressureIter=its, pTol=0.0, precision=prec)
    d = A.diagonal()
    y, r = np.zeros_like(b), b.copy()
    z = r / d
    p, rz = z.copy(), r @ z
    for _ in range(its):
        Ap = A @ p
        a = rz / (p @ Ap)
        y += a * p
        r -= a * Ap
        z = r / d
        p, rz = z + (r @ z) / rz * p, r @ z
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    assert it == its
    assert np.linalg.norm(x - y) <= 1e4 * its * eps * np.linalg.norm(y)
