"""Periodic channels whose levels launch thousands of blocks (B200): the pending
means are finished by the producer there (kPendingMost) and left as partials on the
levels below; cycles against the oracle, whose tolerance is the solver tests' (2e-11
of the iterate for a cycle).
"""
import numpy as np
import pytest
import torch
from oracle import mg as omg
from afsi_gpu_b200.grid import ChannelGrid
from afsi_gpu_b200.multigrid import ChannelMultigrid, MGOptions

pytestmark = pytest.mark.gpu


# blocks of 32 x 8 cells per level: 4096, 1024, ...; 2048, 512, ...; 1216, just above; 1152, below
@pytest.mark.parametrize('shape', [(1024, 1024), (2048, 256), (1216, 256), (1152, 256)])
@pytest.mark.parametrize('smoother', ['jacobi', 'red-black'])
def test_cycles_match_the_oracle(shape, smoother):
    grid = ChannelGrid(shape, (1., .25), periodic=True)
    r = np.random.default_rng(11).standard_normal(shape)
    r -= r.mean()
    mg = ChannelMultigrid(grid, backend='b200', smoother=smoother, options=MGOptions(smooth=2))
    mg.initialize(torch.zeros(shape, device='cuda', dtype=torch.float64), torch.as_tensor(r, device='cuda'))
    h = omg.Hierarchy(grid.shape, grid.spacing, 'periodic')
    p = np.zeros(shape)
    for _ in range(2):
        p = omg.cycle(h, 0, p, r, 2, smoother)
        got = mg.cycle().cpu().numpy()
        assert np.abs(got - p).max() <= 2e-11 * np.abs(p).max()
    first = mg.workspace.p[0].clone()
    mg.initialize(torch.zeros(shape, device='cuda', dtype=torch.float64), torch.as_tensor(r, device='cuda'))
    mg.advance(2)
    assert torch.equal(first, mg.workspace.p[0])  # a fixed order whichever block ends last
