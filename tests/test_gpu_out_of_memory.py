"""The adjoint's working arrays do not fit: the call returns an error, and once
there is room the next one works (no GPU fault: the allocation is refused)."""
import numpy as np
import pytest
import torch

from _helpers import gpu_for
from coldplate_b200 import CpError, cases, release_cached_memory

pytestmark = pytest.mark.gpu

CP_ERR_CUDA = 6


def test_adjoint_after_its_allocations_failed():
    case = cases.density_field(512, 768, seed=2)
    with gpu_for(case, pressureSolverType=4, precision="fp64") as g:
        g.step(10)
        release_cached_memory()
        torch.cuda.empty_cache()
        # some 800 MB are needed; leave the first arrays room and the basis none
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (400 << 20), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            with pytest.raises(CpError) as e:
                g.adjoint_dp_dgamma(max_iter=3, tol=1e-2)
            assert e.value.status == CP_ERR_CUDA
        del fill
        torch.cuda.empty_cache()
        grad, rep = g.adjoint_dp_dgamma(max_iter=3, tol=1e-2)
        assert rep["iterations"] <= 3 and np.isfinite(grad).all()
