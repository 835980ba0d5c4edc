"""Launched 3D V-cycles (marching sweeps, octet prolongation, pending means)
against the oracle on box shapes whose columns, chunks and ends differ (B200).

One cycle and a solve, on levels with few or many planes per chunk, odd
coarse extents and one, two or three launched levels; tolerances are the
solver tests' (2e-11 of the iterate for one cycle, 2e-8 for a solve, the oracle's
cycle count).  FP32 cycles are within 2e-4 of the FP64 oracle's.
"""
import numpy as np
import pytest
import torch
from oracle import mg as omg
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.multigrid import DirichletMultigrid, GeometricMultigrid, MGOptions

pytestmark = pytest.mark.gpu
DEV = 'cuda'
SOLVERS = {'neumann': GeometricMultigrid, 'dirichlet': DirichletMultigrid}


@pytest.mark.parametrize('bc', list(SOLVERS))
@pytest.mark.parametrize('shape,lengths', [((48, 32, 40), (1., 1., 1.)), ((20, 24, 28), (1., .7, 1.3)),
                                          ((64, 32, 96), (1., .5, 2.)), ((144, 80, 64), (2., 1., 1.))])
@pytest.mark.parametrize('smooth', [1, 4])
def test_cycle_and_solve_match_oracle(bc, shape, lengths, smooth):
    grid = MACGrid(shape, lengths)
    r = np.random.default_rng(7).standard_normal(shape)
    r -= r.mean()
    h = omg.Hierarchy(grid.shape, grid.spacing, bc)
    opts = MGOptions(smooth=smooth, rtol=1e-6)
    for backend in ('b200', 'b200-graph'):
        mg = SOLVERS[bc](grid, options=opts, backend=backend)
        p, info = mg.solve(torch.as_tensor(r, device=DEV))
        ref, rinfo = omg.solve(h, r, sweeps=smooth, rtol=1e-6)
        assert info['cycles'] == rinfo['cycles']
        assert np.abs(p.cpu().numpy() - ref).max() <= 2e-8 * np.abs(ref).max()
    host = SOLVERS[bc](grid, options=opts, backend='b200')
    q, _ = host.solve(torch.as_tensor(r, device=DEV))
    assert torch.equal(p, q)  # the device loop's fused check and the host loop's finalize: the same bits


def test_fp32_cycles_follow_the_fp64_solution():
    grid = MACGrid((40, 48, 32), (1., 1., 1.))
    r = np.random.default_rng(3).standard_normal(grid.shape)
    r -= r.mean()
    out = []
    for dtype in (torch.float64, torch.float32):
        mg = GeometricMultigrid(grid, dtype=dtype, coarse_dtype=torch.float64, backend='b200')
        mg.initialize(torch.zeros(grid.shape, device=DEV, dtype=dtype), torch.as_tensor(r, device=DEV, dtype=dtype))
        mg.advance(3)
        out.append(mg.workspace.p[0].double())
    assert float((out[0] - out[1]).abs().max()) <= 2e-4 * float(out[0].abs().max())
