"""Batched tile operations on shapes whose tiles, rows and ends differ (B200):
the iterates stay bitwise those of each instance's own V-cycles."""
import numpy as np
import pytest
import torch
from afsi_gpu_b200.batch import BatchedChannels, BatchedVCycles, Schedule, leaflet_points
from afsi_gpu_b200.grid import ChannelGrid
from afsi_gpu_b200.multigrid import ChannelMultigrid, MGOptions

pytestmark = pytest.mark.gpu
DEV = 'cuda'
SHAPES = [(160, 48), (144, 80), (176, 112), (72, 120), (512, 64), (192, 96)]


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('smooth', [1, 3])
def test_batched_cycles_equal_single_instances(smooth, dtype):
    rng = np.random.default_rng(5)
    opts = MGOptions(smooth=smooth)
    make = lambda: [ChannelMultigrid(ChannelGrid(s, (4., 1.)), dtype=dtype, coarse_dtype=torch.float64, backend='b200',
                                     options=opts) for s in SHAPES]
    alone, batch = make(), make()
    rhs = [torch.as_tensor(rng.standard_normal(s), device=DEV, dtype=dtype) for s in SHAPES]
    BatchedVCycles(batch, rhs).run(3)
    for mg, b, r in zip(alone, batch, rhs):
        mg.initialize(torch.zeros_like(r), r)
        mg.advance(3)
        assert torch.equal(mg.workspace.p[0], b.workspace.p[0])


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_batched_spread_of_few_and_odd_point_counts(dtype):
    rng = np.random.default_rng(6)
    shapes, counts = [(128, 32), (160, 48), (96, 40)], [1, 7, 2050]
    grids = [ChannelGrid(s, (4., 1.)) for s in shapes]
    pts = [leaflet_points(g, n, seed=i) for i, (g, n) in enumerate(zip(grids, counts))]
    forces = [rng.standard_normal((n, 2)) for n in counts]
    vel = [tuple(rng.standard_normal(g.face_shape(c)) for c in range(2)) for g in grids]
    rhs = [rng.standard_normal(s) for s in shapes]
    b = BatchedChannels(grids, pts, forces, vel, rhs, transfer_dtype=dtype,
                        schedule=Schedule(streams=1, cycles=1, vcycles='batched'))
    b.run()
    b.check()
    tol = 1e-13 if dtype == torch.float64 else 4e-6  # hundreds of links per face at the unit roundoff
    for i, g in enumerate(grids):
        from afsi_gpu_b200 import cuda_ib
        x, f = torch.as_tensor(pts[i], device=DEV), torch.as_tensor(forces[i], device=DEV)
        for got, ref in zip(b.fields(i), cuda_ib.spread2d(g, f, cuda_ib.prepare2d(g, x))):
            assert float((got.double() - ref).abs().max()) <= tol * float(ref.abs().max())
