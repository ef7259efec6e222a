"""Smoothed-aggregation PCG on grids a few columns or rows wide, whose coarse
levels are far shorter than their row pitch: the solve, and the memory that the
stored V-cycle matrices take."""
import numpy as np
import pytest
import torch

from coldplate_b200 import Simple, _native
from test_gpu_pressure_sa_sizes import H, RHO, gpu_solve, system

pytestmark = pytest.mark.gpu

SIZES = [(3070, 4), (1000, 10), (700, 3), (5, 3000)]


@pytest.mark.parametrize("Ny,Nx", SIZES)
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_narrow_grids_are_solved(Ny, Nx, prec):
    fields, _, A, b = system(Ny, Nx)
    tol = 1e-6 if prec == "fp64" else 1e-4
    it, x = gpu_solve(Ny, Nx, fields, pressureSolverType=4, maxPressureIter=400, pTol=tol, precision=prec)
    rel = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
    # the recursive residual of a float CG drifts by a rounding of A x an iteration
    drift = 0.0 if prec == "fp64" else it * 2.0 ** -24 * np.linalg.norm(abs(A) @ abs(x)) / np.linalg.norm(b)
    assert it < 400 and rel <= 1.001 * tol + drift, (it, rel, drift)


@pytest.mark.parametrize("Ny,Nx", SIZES)
def test_narrow_grids_take_little_memory(Ny, Nx):
    """A matrix of at most 1024 x 1024 doubles and one of a ninth of it, 40 arrays
    of the grid with its rows padded to 32 elements, and blocks of up to 32 MB that
    are not full."""
    assert _native.lib().cp_release_cached_memory() == 0
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with Simple(Ny=Ny, Nx=Nx, hx=H, hy=H, rho=RHO, targetVel=0.5, pressureSolverType=4, precision="fp64"):
        used = free - torch.cuda.mem_get_info()[0]
    grid = (Ny + 3) * ((Nx + 2 + 31) // 32 * 32) * 8
    assert used <= 1.2 * 1024 * 1024 * 8 + 60 * grid + (48 << 20), used
