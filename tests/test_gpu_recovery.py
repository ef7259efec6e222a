"""A context after a solve that overflowed (finite inputs, no GPU fault): once
it holds good fields again it gives the bits of a fresh context, from the
dispatch calls and from whole iterations, on grids whose pressure solve runs on
every SM and on one cluster."""
import numpy as np
import pytest

from _helpers import gpu_for
from coldplate_b200 import CpError, cases

pytestmark = pytest.mark.gpu

SIZES = [(241, 517), (17, 1600), (60, 120)]


def good(g, shapes):
    """A dispatch pressure solve on given fields, then whole iterations."""
    rng = np.random.default_rng(4)
    g.reset()
    for f in ("uStar", "vStar"):
        g.set(f, rng.standard_normal(shapes[f]))
    for f in ("dE", "dN"):
        g.set(f, 10.0 ** rng.uniform(-8, -7, shapes[f]))
    its = [g.solvePressureSystem()[0]]
    out = [g.get("pStar")]
    g.reset()
    its.append(g.step(3)["pressureIterations"])
    return its, out + [g.get(f) for f in ("u", "v", "p", "pStar")]


def overflow_dispatch(g, shapes):
    for f in ("uStar", "vStar"):
        g.set(f, np.full(shapes[f], 0.5))
    for f in ("dE", "dN"):
        g.set(f, np.full(shapes[f], 1e-7))
    a = np.full(shapes["uStar"], 0.5)
    a[5:9, 7:11] = 1e300
    g.set("uStar", a)
    g.solvePressureSystem()
    assert not np.isfinite(g.get("pStar")).all()


def overflow_step(g, shapes):
    g.step(2)
    u = g.get("u")
    u[5, 7] = 1e300
    g.set("u", u)
    with pytest.raises(CpError) as e:
        g.step(3)
    assert e.value.status == 3   # CP_ERR_NONFINITE


@pytest.mark.parametrize("Ny,Nx", SIZES)
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("solver", [1, 2, 4])
@pytest.mark.parametrize("overflow", [overflow_dispatch, overflow_step])
def test_an_overflowed_solve_leaves_nothing_behind(overflow, solver, prec, Ny, Nx):
    case = cases.density_field(Ny, Nx, seed=6)
    over = dict(pressureSolverType=solver, pTol=1e-6, precision=prec)
    with gpu_for(case, **over) as g:
        shapes = {f: g.shape(f) for f in ("uStar", "vStar", "dE", "dN")}
        its, want = good(g, shapes)
        assert all(np.isfinite(a).all() for a in want)
    with gpu_for(case, **over) as g:
        overflow(g, shapes)
        its2, got = good(g, shapes)
    assert its2 == its
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
