"""The deterministic table spread in a time loop (B200): positions move, tables are
prepared into the same buffers or into recycled memory, and every spread equals the
atomic one of the same tables (1e-12 of the field, the bar of the transfer tests)."""
import pytest
import torch
from afsi_gpu_b200 import synthetic, p2_cuda_transfer as p2t
from afsi_gpu_b200.grid import MACGrid

pytestmark = pytest.mark.gpu
DEV = 'cuda'


@pytest.mark.parametrize('reuse', [True, False])
def test_steps_follow_their_own_tables(reuse):
    X, cells = synthetic.p2_shell(1, 8, 12, inner=(.1, .07, .07), outer=(.13, .1, .1))
    x, cells = torch.as_tensor(X, device=DEV), torch.as_tensor(cells, device=DEV)
    grid = MACGrid((48, 48, 48), (1., 1., 1.))
    det = p2t.P2Transfer(grid, x, cells, deterministic=True, max_order=22)
    atomic = p2t.P2Transfer(grid, x, cells, max_order=22)
    coef = torch.randn(x.shape, device=DEV, dtype=torch.float64, generator=torch.Generator(device=DEV).manual_seed(3))
    buffers, last = None, None
    for step in range(4):
        shift = torch.tensor([.11, -.07, .05], device=DEV, dtype=torch.float64) * step
        st = det.prepare(x + shift, buffers=buffers)
        if reuse:
            buffers = st.base, st.phi
        got, want = det.spread(coef, st), p2t.spread(atomic, coef, st)
        for a, b in zip(got, want):
            assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())
        if reuse and last is not None:  # its tables were written anew: rows outside its tiles are left out
            assert all(bool(u.isfinite().all()) for u in det.spread(coef, last))
        last = st if reuse else None
        del st
