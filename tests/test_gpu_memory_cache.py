"""Contexts made from the cached memory of destroyed ones: the same results as
from fresh memory, in any order of sizes, from several threads, and after the
cache was given back."""
import threading

import numpy as np
import pytest

from _helpers import gpu_for
from coldplate_b200 import Thermal, _native, cases

pytestmark = pytest.mark.gpu


def flow(Ny, Nx, prec):
    case = cases.density_field(Ny, Nx, seed=2)
    with gpu_for(case, pressureSolverType=4, pTol=1e-6, precision=prec) as g:
        g.step(4)
        # run for the memory it takes; its scattered sums (atomics) make the
        # gradient itself differ in the last bits from run to run
        g.adjoint_dp_dgamma(tol=1e-4, max_iter=40)
        g.step(2)
        return [g.get(f) for f in ("u", "v", "p")]


def thermal(Ny, Nx):
    rng = np.random.default_rng(7)
    with Thermal(Nx=Nx, Ny=Ny, dx=2e-5, dy=2e-5, H_t=2e-4) as th:
        th.set_inputs(rng.random((Ny, Nx)), rng.random((Ny, Nx)), np.zeros((Ny, Nx)), np.full((Ny, Nx), 5e5))
        th.solve()
        return [th.T, th.pnorm_gradient(8.0)[1]]


JOBS = [lambda: flow(40, 90, "fp64"), lambda: flow(130, 300, "mixed"), lambda: thermal(33, 50), lambda: flow(300, 500, "fp64")]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_cached_memory_gives_the_results_of_fresh_memory():
    lib = _native.lib()
    fresh = []
    for job in JOBS:
        assert lib.cp_release_cached_memory() == 0
        fresh.append(job())
    for order in ((3, 1, 0, 2), (0, 1, 2, 3), (2, 2, 3, 0)):
        for q in order:
            assert same(JOBS[q](), fresh[q]), q
    wrong = []

    def work(first):
        for n in range(6):
            q = (first + n) % len(JOBS)
            if not same(JOBS[q](), fresh[q]):
                wrong.append(q)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    assert lib.cp_release_cached_memory() == 0
    assert same(JOBS[0](), fresh[0])
