"""Which dense clouds take the binned spread (cuda_ib._binned_per_cell).

The binned form keeps two words per cell of the grid, so a small dense body in a
large box takes the plain one; the other lines are those of the measured table beside
the rule.
"""
import pytest
import torch
from afsi_gpu_b200 import cuda_ib, _lib
from afsi_gpu_b200.grid import MACGrid


def _bytes(n, points, dtype):
    grid = MACGrid((n, n, n), (1., 1., 1.))
    phi = torch.zeros((1, 3, 4), dtype=dtype)
    stencil = cuda_ib.CompactStencil(torch.zeros((3, 1, 3), dtype=torch.int64), phi, dense=True)
    return cuda_ib._binned_bytes(grid, stencil, points, phi)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('n,points', [(256, 70000), (512, 70000), (512, 1000000), (192, 60000), (1024, 4000000)])
def test_a_small_dense_body_in_a_large_box_takes_the_plain_form(n, points, dtype):
    assert _lib.load().afsi_b200_compact_binned_bytes(points, n, n, n) > 0
    assert _bytes(n, points, dtype) == 0
    assert cuda_ib._binned_per_cell(points, (n, n, n), dtype) is None


@pytest.mark.parametrize('n,points', [(64, 60000), (64, 400000), (128, 200000), (256, 400000)])
def test_scratch_stays_below_that_of_the_cells_per_point(n, points):
    need = _bytes(n, points, torch.float64)
    # 12 bytes per point, two words for each of 64 cells of a tile, the tiles padded, and the scan's own
    assert 0 < need <= 12 * points + 8 * (n + 4) ** 3 * 1.05 + (1 << 20)
    assert need <= 12 * points + 96 * 9 * points + (1 << 20)


def test_points_per_cell_follow_the_measured_lines():
    at = lambda n, points, dtype=torch.float64: cuda_ib._binned_per_cell(points, (n, n, n), dtype)
    assert at(64, 59999) is None and 17 < at(64, 60000) < 22 and 25 < at(128, 60000) < 31
    assert at(64, 200000) == at(64, 400000) == at(256, 1000000) == 9
    assert 14 < at(256, 400000) < 18


def test_fp32_clouds_have_a_line_of_their_own():
    at = lambda n, points: cuda_ib._binned_per_cell(points, (n, n, n), torch.float32)
    assert at(64, 60000) > 50 and 30 < at(64, 100000) < 40 and at(64, 200000) == at(128, 400000) == 22
    assert 22 < at(128, 200000) < 25
    assert at(32, 60000) < 30 < 70 < at(128, 60000)  # the latter measured faster at no density
    assert at(256, 1000000) is at(256, 4000000) is None


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_a_dense_corner_of_a_large_grid(dtype):
    grid, points = MACGrid((256, 256, 256), (1., 1., 1.)), 70000
    g = torch.Generator(device='cuda').manual_seed(4)
    x = (.02 + .02 * torch.rand((points, 3), device='cuda', dtype=torch.float64, generator=g)).to(dtype)
    st = cuda_ib.compact_prepare(grid, x)
    assert not st.dense
    force = torch.ones((points, 3), device='cuda', dtype=dtype)
    cuda_ib.compact_spread(grid, force, st)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    fields = cuda_ib.compact_spread(grid, force, st)
    faces = sum(u.numel() * u.element_size() for u in fields)
    assert torch.cuda.max_memory_allocated() - before <= faces + (1 << 20)
    for u in fields:  # 70,000 unit forces, weights that sum to one
        assert float(u.double().sum()) * grid.volume == pytest.approx(points, rel=1e-9 if dtype == torch.float64 else 1e-4)
