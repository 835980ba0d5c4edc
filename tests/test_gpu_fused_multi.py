"""Several elements per warp in the table-free transfers (csrc/fe_fused.cu)
against the warp-per-element kernels (B200).

Groups of fewer than 2 x 1184 elements take the warp-per-element kernels, so
the same rule cut into small groups is the reference: the same rows and force
factors, summed in another order.  A face sums some hundred links and a node some
hundred points, so the two agree to about 1e-14 (FP64) and 5e-6 (FP32) of the
field scale.
"""
import numpy as np
import pytest
import torch
from afsi_gpu_b200 import synthetic, p2_cuda_transfer as p2t
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.quadrature import InteractionRule, QuadratureGroup

pytestmark = pytest.mark.gpu
DEV = 'cuda'
WALLS = dict(inner=(.2, .12, .12), outer=(.215, .135, .135))


def _cut(rule, most=1200):
    """The rule with every group cut into pieces of at most `most` elements."""
    groups = []
    for g in rule.groups:
        for lo in range(0, g.cells.shape[0], most):
            groups.append(QuadratureGroup(g.cells[lo:lo + most].contiguous(), g.values,
                                          g.weights[lo:lo + most].contiguous(), g.order))
    return InteractionRule(tuple(groups), rule.orders, rule.point_count)


def _free(x, rule):
    return p2t.TableFreeStencil(x, rule, torch.zeros((), dtype=torch.int32, device=DEV))


def _both(tr, x, rule, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    coef = torch.randn(x.shape, device=DEV, dtype=torch.float64, generator=g).to(tr.transfer_dtype)
    vel = tuple(torch.randn(tr.grid.face_shape(c), device=DEV, dtype=torch.float64, generator=g).to(tr.transfer_dtype)
                for c in range(3))
    out = []
    for r in (rule, _cut(rule)):
        st = _free(x, r)
        out.append((*p2t.spread(tr, coef, st), p2t.assemble_velocity(tr, vel, st), st))
    return out


def _close(a, b, dtype):
    tol = 1e-14 if dtype == torch.float64 else 5e-6
    for x, y in zip(a[:4], b[:4]):
        assert float(y.abs().max()) > 0
        assert float((x - y).abs().max()) <= tol * float(y.abs().max())


@pytest.mark.parametrize('order', ['mesh', 'shuffled'])
@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('kind,n,shape', [('p1', (1, 30, 48), 48), ('p1', (2, 20, 31), 40), ('p1', (2, 24, 40), 24),
                                          ('p2', (2, 21, 34), 24)])
def test_groups_of_elements_equal_single_elements(kind, n, shape, dtype, order):
    n = (n[0], n[1], n[2] + n[2] % 2)
    X, cells = synthetic.prolate_shell(*n, **WALLS)
    if kind == 'p2':
        X, cells = synthetic.promote_p1(X, cells)
    if order == 'shuffled':  # no neighbours: the union box does not fit
        cells = np.random.default_rng(1).permutation(cells)
    cells = cells[:len(cells) - 3]  # a ragged last group
    x = torch.as_tensor(X, device=DEV)
    cls = p2t.P1Transfer if kind == 'p1' else p2t.P2Transfer
    tr = cls(MACGrid((shape, shape + 5, shape), (1., 1., 1.)), x, torch.as_tensor(cells, device=DEV), max_order=22,
             transfer_dtype=dtype)
    rule = tr.rule(x)
    assert max(g.cells.shape[0] for g in rule.groups) >= 2 * 1184 and min(g.values.shape[0] for g in rule.groups) <= 16
    a, b = _both(tr, x, rule)
    _close(a, b, dtype)
    tr.check(a[4]), tr.check(b[4])
    # the deterministic gather-assemble: element sums without atomics
    det = cls(tr.grid, x, tr.cells, max_order=22, transfer_dtype=dtype, deterministic=True)
    vel = tuple(torch.randn(tr.grid.face_shape(c), device=DEV, dtype=dtype) for c in range(3))
    first = p2t.assemble_velocity_deterministic(det, vel, _free(x, rule))
    assert torch.equal(first, p2t.assemble_velocity_deterministic(det, vel, _free(x, rule)))
    ref = p2t.assemble_velocity(det, vel, _free(x, _cut(rule)))
    assert float((first - ref).abs().max()) <= (1e-14 if dtype == torch.float64 else 5e-6) * float(ref.abs().max())


def test_bad_nodes_and_supports_are_flagged_and_the_others_transferred():
    X, cells = synthetic.prolate_shell(1, 30, 48, **WALLS)
    x = torch.as_tensor(X, device=DEV)
    tr = p2t.P1Transfer(MACGrid((48, 48, 48), (1., 1., 1.)), x, torch.as_tensor(cells, device=DEV))
    rule = tr.rule(x)
    k = max(range(len(rule.groups)), key=lambda i: rule.groups[i].cells.shape[0])
    g = rule.groups[k]
    bad = g.cells.clone()
    bad[101, 1], bad[2000, 3] = -1, x.shape[0]
    groups = list(rule.groups)
    groups[k] = QuadratureGroup(bad, g.values, g.weights, g.order)
    broken = InteractionRule(tuple(groups), rule.orders, rule.point_count)
    a, b = _both(tr, x, broken)
    _close(a, b, torch.float64)
    with pytest.raises(RuntimeError, match='connectivity'):
        tr.check(a[4])
    moved = x.clone()
    moved[cells[77, 2]] = torch.tensor([.5, .5, -1.], device=DEV, dtype=torch.float64)
    a, b = _both(tr, moved, rule)
    _close(a, b, torch.float64)
    with pytest.raises(ValueError, match='support'):
        tr.check(a[4])
