"""One-launch compact and 2D transfers against the per-component operators (B200).

Both forms add the same products; the spread's atomic order and the gather's
grouping differ, so they agree to rounding: 64 links per point, up to some
thousand points per face, eps * sqrt(terms) of the field scale (FP64 1e-14, FP32 5e-6).
"""
from types import SimpleNamespace
import numpy as np
import pytest
import torch
from afsi_gpu_b200 import cuda_ib
from afsi_gpu_b200.grid import ChannelGrid, MACGrid

pytestmark = pytest.mark.gpu
DEV = 'cuda'
TOL = {torch.float64: 1e-14, torch.float32: 5e-6}


def _close(a, b, dtype):
    assert a.shape == b.shape and a.dtype == b.dtype
    assert float((a - b).abs().max()) <= TOL[dtype] * max(float(b.abs().max()), 1e-300)


def _cloud(n, dim, lo, hi, dtype, seed=0):
    r = np.random.default_rng(seed).uniform(lo, hi, (n, dim))
    return torch.as_tensor(r, device=DEV, dtype=dtype)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('shape,points', [((9, 8, 8), 1), ((17, 24, 31), 31), ((32, 33, 20), 33), ((64, 16, 40), 5003)])
def test_compact_three_components_in_one_launch(shape, points, dtype):
    grid = MACGrid(shape, (1., 1., 1.), (.5, -.25, 0.))
    h = np.asarray(grid.spacing)
    x = _cloud(points, 3, np.asarray(grid.origin) + 2.01 * h, np.asarray(grid.origin) + 1 - 2.01 * h, dtype)
    force = _cloud(points, 3, -1, 1, dtype, 1)
    vel = tuple(torch.randn(grid.face_shape(c), device=DEV, dtype=dtype) for c in range(3))
    st = cuda_ib.compact_prepare(grid, x)
    # lists of per-component tables take the per-component operators
    lists = SimpleNamespace(base=[b.clone() for b in st.base], phi=[p.clone() for p in st.phi])
    for a, b in zip(cuda_ib.compact_spread(grid, force, st), cuda_ib.compact_spread(grid, force, lists)):
        _close(a, b, dtype)
    _close(cuda_ib.compact_gather(grid, vel, st), cuda_ib.compact_gather(grid, vel, lists), dtype)
    # non-contiguous inputs, and a table whose weights start off a 16-byte boundary
    wide = torch.stack((force, force), -1)[..., 0]
    strided = tuple(torch.stack((v, v), -1)[..., 1] for v in vel)
    _close(cuda_ib.compact_spread(grid, wide, st)[1], cuda_ib.compact_spread(grid, force, st)[1], dtype)
    _close(cuda_ib.compact_gather(grid, strided, st), cuda_ib.compact_gather(grid, vel, st), dtype)
    raw = torch.empty(st.phi.numel() + 1, device=DEV, dtype=dtype)
    raw[1:] = st.phi.reshape(-1)
    off = SimpleNamespace(base=st.base, phi=raw[1:].view(st.phi.shape))
    _close(cuda_ib.compact_gather(grid, vel, off), cuda_ib.compact_gather(grid, vel, st), dtype)
    _close(cuda_ib.compact_spread(grid, force, off)[2], cuda_ib.compact_spread(grid, force, st)[2], dtype)
    assert cuda_ib.check() == 0


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('shape,points', [((16, 8), 1), ((37, 19), 33), ((64, 16), 4097)])
def test_channel_components_in_one_launch(shape, points, dtype):
    grid = ChannelGrid(shape, (1., .25))
    hx, hy = grid.spacing
    x = _cloud(points, 2, (2.01 * hx, -.9 * hy), (1 - 2.01 * hx, .25 + .9 * hy), dtype)
    force = _cloud(points, 3, -1, 1, dtype, 1)  # a third column is ignored
    vel = tuple(torch.randn(grid.face_shape(c), device=DEV, dtype=dtype) for c in range(2))
    st = cuda_ib.prepare2d(grid, x)
    one = [cuda_ib.indexed_spread(force[:, c:c + 1], st.indices[c], st.weights[c], int(np.prod(grid.face_shape(c))),
                                  grid.volume).view(grid.face_shape(c)) for c in range(2)]
    for a, b in zip(cuda_ib.spread2d(grid, force, st), one):
        _close(a, b, dtype)
    ref = torch.cat([cuda_ib.indexed_gather(u.reshape(-1, 1), i, w) for u, i, w in zip(vel, st.indices, st.weights)], -1)
    assert torch.equal(cuda_ib.gather2d(vel, st), ref)
    assert cuda_ib.check() == 0


def test_out_of_range_rows_are_flagged_and_skipped_and_refusals_stay():
    grid = MACGrid((16, 16, 16), (1., 1., 1.))
    x = _cloud(40, 3, .3, .7, torch.float64)
    force, vel = _cloud(40, 3, -1, 1, torch.float64, 1), grid.zeros(device=DEV)
    st = cuda_ib.compact_prepare(grid, x)
    base = st.base.clone()
    base[1, 7, 2] = 14
    broken = cuda_ib.CompactStencil(base, st.phi)
    cuda_ib.compact_spread(grid, force, broken)
    with pytest.raises(RuntimeError, match='outside the MAC grid'):
        cuda_ib.check()
    with pytest.raises(RuntimeError):
        cuda_ib.compact_spread(grid, force.float(), st)
    with pytest.raises(RuntimeError):
        cuda_ib.compact_spread(grid, force[:39], st)
    with pytest.raises(RuntimeError):
        cuda_ib.compact_gather(grid, (vel[1], vel[0][:-1], vel[2]), st)
    with pytest.raises(RuntimeError, match='autograd'):
        cuda_ib.compact_spread(grid, force.clone().requires_grad_(), st)
    channel = ChannelGrid((16, 8), (1., .25))
    s2 = cuda_ib.prepare2d(channel, _cloud(9, 2, (.3, .05), (.7, .2), torch.float64))
    ids = s2.indices[0].clone()
    ids[3, 5] = 17 * 8
    cuda_ib.spread2d(channel, force[:9], cuda_ib.Stencil2D((ids, s2.indices[1]), s2.weights))
    with pytest.raises(RuntimeError, match='outside the MAC grid'):
        cuda_ib.check()
    with pytest.raises(RuntimeError):
        cuda_ib.spread2d(channel, force[:8], s2)
