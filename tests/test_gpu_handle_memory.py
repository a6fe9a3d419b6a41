"""A small handle does not hold the solve's lists at their maxima: what one CTA
can own, publish, fetch and index on the grid bounds them."""
import pytest
import torch

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu


# grid; megabytes: fields and sort buffers (about 150 bytes a cell) plus the solve's lists
@pytest.mark.parametrize("n,most", [(12, 12), (24, 20), (64, 100)])
def test_memory_of_a_small_handle(n, most):
    warm = FluidSolver(nx=8, ny=8, nz=8, dx=1.0, coreR=1.0, targetParticles=10.0, capacity=100)   # the module itself
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    fs = FluidSolver(nx=n, ny=n, nz=n, dx=1.0, coreR=1.0, targetParticles=1000.0, capacity=1000)
    torch.cuda.synchronize()
    used = (free - torch.cuda.mem_get_info()[0]) / 1e6
    fs.close()
    warm.close()
    assert used <= most
