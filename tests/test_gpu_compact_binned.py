"""The binned compact spread against the plain one (B200).

Both add the same products in another order (and FP64 in another grouping: an
x weight times the other factors): a face that m points reach, each with a
handful of roundings, differs by at most (m + 8) eps times the sum S of its
terms' magnitudes, in either form.
"""
import numpy as np
import pytest
import torch
from afsi_gpu_b200 import cuda_ib
from afsi_gpu_b200._lib import call, dtype_code, ptr, status_word, stream
from afsi_gpu_b200 import _lib
from afsi_gpu_b200.grid import MACGrid

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _spread(grid, force, base, phi, binned):
    out = [torch.full(grid.face_shape(c), 7., device=DEV, dtype=force.dtype) for c in range(3)]
    head = (ptr(force), ptr(base), ptr(phi), base.shape[1], *grid.shape, float(grid.volume), *(ptr(u) for u in out))
    tail = (ptr(status_word(force.device)), dtype_code(force.dtype), stream(force.device))
    if binned:
        need = _lib.load().afsi_b200_compact_binned_bytes(base.shape[1], *grid.shape)
        work = torch.full((need,), 255, device=DEV, dtype=torch.uint8)
        call('afsi_b200_compact_spread3_binned', *head, ptr(work), need, *tail)
    else:
        call('afsi_b200_compact_spread3', *head, *tail)
    return out


def _compare(grid, force, base, phi):
    got, want = _spread(grid, force, base, phi, True), _spread(grid, force, base, phi, False)
    S = _spread(grid, force.abs(), base, phi.abs(), False)
    m = _spread(grid, torch.ones_like(force), base, torch.ones_like(phi), False)
    eps = torch.finfo(force.dtype).eps
    for a, b, s, k in zip(got, want, S, m):
        assert bool(((a - b).abs() <= 2 * (k * grid.volume + 8) * eps * s).all())
    return got


CLOUDS = [('uniform', (9, 8, 8), 1), ('uniform', (17, 24, 31), 63), ('uniform', (32, 33, 20), 65),
          ('uniform', (33, 30, 41), 20011), ('uniform', (64, 16, 40), 300), ('line', (40, 12, 9), 5003),
          ('cell', (16, 16, 16), 4097), ('sheet', (24, 40, 36), 60000)]


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('kind,shape,points', CLOUDS)
def test_binned_spread_equals_plain(kind, shape, points, dtype):
    grid = MACGrid(shape, (1., .9, 1.1), (.5, -.25, 0.))
    h, r = np.asarray(grid.spacing), np.random.default_rng(points)
    t = r.uniform(0, 1, (points, 3))
    if kind == 'line':
        t[:, 1:] = .5
    elif kind == 'cell':
        t = .5 + t * .5 / 16
    elif kind == 'sheet':
        t[:, 0] = .5 + .1 * np.sin(7 * t[:, 1])
    lo, hi = np.asarray(grid.origin) + 2.01 * h, np.asarray(grid.origin) + np.asarray(grid.lengths) - 2.01 * h
    x = torch.as_tensor(lo + t * (hi - lo), device=DEV, dtype=dtype)
    st = cuda_ib.compact_prepare(grid, x)
    force = torch.as_tensor(r.normal(size=(points, 3)), device=DEV, dtype=dtype)
    _compare(grid, force, st.base, st.phi)
    assert cuda_ib.check() == 0


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_binned_spread_takes_any_table(dtype):
    """Component tables unrelated to one another, signed weights, rows outside
    the grid (skipped and flagged by themselves) and nonfinite forces."""
    grid = MACGrid((20, 17, 23), (1., 1., 1.))
    g = torch.Generator(device=DEV).manual_seed(3)
    points = 3000
    base = torch.stack([torch.stack([torch.randint(0, n + (a == c) - 3, (points,), device=DEV, generator=g)
                                     for a, n in enumerate(grid.shape)], -1) for c in range(3)])
    phi = torch.randn((3, points, 3, 4), device=DEV, dtype=dtype, generator=g)
    force = torch.randn((points, 3), device=DEV, dtype=dtype, generator=g)
    _compare(grid, force, base, phi)
    assert cuda_ib.check() == 0
    base[0, 5, 0], base[1, 6, 2], base[2, 7, 1] = -1, 21, 1 << 40
    base[0, 8:200] = -7
    _compare(grid, force, base, phi)
    with pytest.raises(RuntimeError):
        cuda_ib.check()
    force[11, 1] = float('inf')
    force[900, 2] = float('nan')
    got, want = _spread(grid, force, base, phi, True), _spread(grid, force, base, phi, False)
    for a, b in zip(got, want):
        assert torch.equal(a.isfinite(), b.isfinite())
    with pytest.raises(RuntimeError):
        cuda_ib.check()


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_wrapper_bins_large_clouds(dtype):
    """The wrapper's rule: a dense cloud is binned, with the results of the
    per-component operators, off a 16-byte boundary and captured; a cloud of few
    points per cell, or of few points, is not."""
    grid, points = MACGrid((40, 36, 32), (1., 1., 1.)), 70001
    r = np.random.default_rng(5)
    u = r.uniform(0, 1, (points, 3))
    force = torch.as_tensor(r.normal(size=(points, 3)), device=DEV, dtype=dtype)

    def cloud(lo, hi, n=points):
        return cuda_ib.compact_prepare(grid, torch.as_tensor(lo + (hi - lo) * u[:n], device=DEV, dtype=dtype))

    st = cloud(.3, .6)  # some 1,300 cells, 54 points each
    assert cuda_ib._binned_bytes(grid, st, points, st.phi) > 0
    assert not cloud(.1, .9).dense and not cloud(.3, .6, 50000).dense  # 3 points per cell; too few points
    assert cuda_ib.check() == 0
    raw = torch.empty(st.phi.numel() + 1, device=DEV, dtype=dtype)
    raw[1:] = st.phi.reshape(-1)
    off = cuda_ib.CompactStencil(st.base, raw[1:].view(st.phi.shape), dense=True)
    assert cuda_ib._binned_bytes(grid, off, points, off.phi) == 0
    graph = torch.cuda.CUDAGraph()
    first = cuda_ib.compact_spread(grid, force, st)
    with torch.cuda.graph(graph):
        captured = cuda_ib.compact_spread(grid, force, st)
    graph.replay()
    # a face is reached by the points of 4 x 4 x 4 cells: 64 x 54 on average, 4500 at most
    tol = 2 * (4500 + 8) * torch.finfo(dtype).eps
    scale = cuda_ib.compact_spread(grid, force.abs(), st)
    for form in (first, captured):
        for a, b, s in zip(form, cuda_ib.compact_spread(grid, force, off), scale):
            assert bool(((a - b).abs() <= tol * s).all())
    with pytest.raises(ValueError):  # the support screen is read with the density
        cloud(-.3, .6)
    assert cuda_ib.check() == 0
