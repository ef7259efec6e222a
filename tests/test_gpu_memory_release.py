"""What the library holds of the device when no context is alive: nothing after
the Python package's release call or with a limit of 0, and a batch takes its
arrays from what is kept."""
import numpy as np
import pytest
import torch

from _helpers import gpu_for
from coldplate_b200 import Batch, cases, release_cached_memory, set_cached_memory_limit

pytestmark = pytest.mark.gpu


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def solve(Ny=300, Nx=400):
    case = cases.density_field(Ny, Nx, seed=1)
    with gpu_for(case, pressureSolverType=4) as g:
        g.step(2)


def test_release_and_limit():
    solve()                      # what stays with the process (kernels, events) is there
    release_cached_memory()
    before = free()
    solve()
    assert free() < before       # kept
    release_cached_memory()
    assert free() >= before
    try:
        set_cached_memory_limit(0, 0)
        solve()
        assert free() >= before
    finally:
        set_cached_memory_limit(4 << 30, 256 << 20)
    solve()
    assert free() < before


def test_a_batch_takes_its_arrays_from_the_cache():
    fields = [gpu_for(cases.density_field(40, 80, seed=k), pressureSolverType=4) for k in range(3)]
    try:
        with Batch(fields) as b:
            b.run(2)
        solve()                  # leaves blocks behind, enough for a batch's few hundred KB
        release = free()
        with Batch(fields) as b:
            b.run(2)
            assert free() >= release
        assert all(np.isfinite(f.get("p")).all() for f in fields)
    finally:
        for f in fields:
            f.close()
