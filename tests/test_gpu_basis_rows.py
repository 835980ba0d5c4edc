"""Basis tables on and off a pair's boundary (B200): the element transfers read
their rows by pairs of values where the table's address allows it and value by
value otherwise.  The values are the same, so element sums without atomics are
bitwise equal and the spreads agree to the order of their reductions, 1e-14 of the
field scale (some hundred links per face).
"""
import pytest
import torch
from afsi_gpu_b200 import synthetic, p2_cuda_transfer as p2t
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.quadrature import InteractionRule, QuadratureGroup

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _shifted(rule):
    groups = []
    for g in rule.groups:
        raw = torch.empty(g.values.numel() + 1, device=DEV, dtype=g.values.dtype)
        raw[1:] = g.values.reshape(-1)
        values = raw[1:].view(g.values.shape)
        assert values.data_ptr() % 16 == 8
        groups.append(QuadratureGroup(g.cells, values, g.weights, g.order))
    return InteractionRule(tuple(groups), rule.orders, rule.point_count)


@pytest.mark.parametrize('kind,n,shape', [('p1', (1, 30, 48), 48), ('p2', (1, 6, 8), 24), ('p2', (1, 6, 8), 48)])
def test_shifted_tables_give_the_same_transfers(kind, n, shape):
    X, cells = synthetic.prolate_shell(*n, inner=(.2, .12, .12), outer=(.215, .135, .135))
    if kind == 'p2':
        X, cells = synthetic.promote_p1(X, cells)
    x = torch.as_tensor(X, device=DEV)
    cls = p2t.P1Transfer if kind == 'p1' else p2t.P2Transfer
    args = (MACGrid((shape, shape, shape), (1., 1., 1.)), x, torch.as_tensor(cells, device=DEV))
    tr, det = cls(*args, max_order=22), cls(*args, max_order=22, deterministic=True)
    rule = tr.rule(x)
    g = torch.Generator(device=DEV).manual_seed(0)
    coef = torch.randn(x.shape, device=DEV, dtype=torch.float64, generator=g)
    vel = tuple(torch.randn(tr.grid.face_shape(c), device=DEV, dtype=torch.float64, generator=g) for c in range(3))
    out = []
    for r in (rule, _shifted(rule)):
        st = p2t.TableFreeStencil(x, r, torch.zeros((), dtype=torch.int32, device=DEV))
        out.append((p2t.spread(tr, coef, st), p2t.assemble_velocity_deterministic(det, vel, st)))
        tr.check(st)
    assert torch.equal(out[0][1], out[1][1])
    for a, b in zip(out[0][0], out[1][0]):
        assert float(b.abs().max()) > 0
        assert float((a - b).abs().max()) <= 1e-14 * float(b.abs().max())
