"""Row-by-row P1 operators (csrc/csr_rows.cu) against the hash assembly (B200).

The two forms add the same products (phi_x phi_y phi_z) W N in another order:
the patterns must be equal, the values differ by rounding only.  An entry sums at
most n = (cells of a node) x (points of a cell) nonnegative terms, so either form
is within n u of it (u the unit roundoff) and the two within 2 n u; the weights at
the edge of a support may be rounding errors of either sign, u of the largest.
"""
import numpy as np
import pytest
import torch
from afsi_gpu_b200 import synthetic
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.p1_csr import P1CSRTransfer
from afsi_gpu_b200.p2_cuda_transfer import SharedAdaptiveStencil
from afsi_gpu_b200.quadrature import InteractionRule, QuadratureGroup

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _fan(cells, turn=5.):
    """`cells` tetrahedra around one node (more than the 32 cells of one pass)."""
    t = np.linspace(0, turn, cells + 1)
    ring = np.stack((.5 + .06 * np.cos(t), .5 + .06 * np.sin(t), np.full(cells + 1, .47)), -1)
    X = np.concatenate(([[.5, .5, .5], [.5, .5, .41]], ring))
    i = np.arange(cells)
    return X, np.stack((np.zeros_like(i), np.ones_like(i), 2 + i, 3 + i), -1)


def _shell(*n):
    return synthetic.prolate_shell(*n, inner=(.125, .075, .075), outer=(.16, .11, .11))


MESHES = {'single': lambda: _fan(1), 'flat': lambda: _fan(2, 0.),  # no volume: empty operators
          'fan33': lambda: _fan(33), 'fan150': lambda: _fan(150),
          'shell': lambda: _shell(2, 10, 16), 'coarse': lambda: _shell(1, 4, 6)}


def _transfer(mesh, dtype, shape=(40, 32, 36)):
    X, cells = MESHES[mesh]()
    x = torch.as_tensor(X, device=DEV, dtype=dtype)
    tr = P1CSRTransfer(MACGrid(shape, (1., 1., 1.)), x, torch.as_tensor(cells, device=DEV), max_order=22)
    return tr, tr.prepare_tables(x)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('mesh', list(MESHES))
def test_rows_equal_the_hash_assembly(mesh, dtype):
    tr, st = _transfer(mesh, dtype)
    a, b = tr._assemble_rows(st), tr._assemble_hash(st)
    u = torch.finfo(dtype).eps / 2
    terms = int(torch.bincount(tr.cells.reshape(-1)).max()) * max(g.values.shape[0] for g in st.rule.groups)
    for x, y in zip(a.gather + a.spread, b.gather + b.spread):
        assert x.shape == y.shape and torch.equal(x.crow, y.crow) and torch.equal(x.col, y.col)
        torch.testing.assert_close(x.val, y.val, rtol=2 * terms * u, atol=u * float(y.val.abs().amax()) if y.nnz else 0.)
    again = tr._assemble_rows(st)  # a fixed order: the same bits
    assert all(torch.equal(x.val, y.val) for x, y in zip(a.gather + a.spread, again.gather + again.spread))
    assert a.assembly['total_nnz'] == b.assembly['total_nnz']


def test_large_boxes_and_bad_connectivity_take_the_hash_form():
    # supports of one cell over about 24 faces per axis: no row box fits shared memory
    X = torch.tensor([[.35, .35, .35], [.65, .36, .35], [.35, .65, .36], [.36, .35, .65]], device=DEV,
                     dtype=torch.float64)
    cells = torch.tensor([[0, 1, 2, 3]], device=DEV)
    tr = P1CSRTransfer(MACGrid((64, 64, 64), (1., 1., 1.)), X, cells, max_order=62)
    st = tr.prepare_tables(X)
    assert tr._assemble_rows(st) is None
    A = tr.assemble_stencil(st)
    assert A.assembly['assembly_backend'] == 'hash' and A.gather[0].nnz > 0
    tr, st = _transfer('shell', torch.float64)
    g = st.rule.groups[0]
    bad = g.cells.clone()
    bad[0, 2] = tr.node_count
    rule = InteractionRule((QuadratureGroup(bad, g.values, g.weights, g.order), *st.rule.groups[1:]), st.rule.orders,
                           st.rule.point_count)
    broken = SharedAdaptiveStencil(st.base, st.phi, rule)
    assert tr._assemble_rows(broken) is None
    with pytest.raises(FloatingPointError, match='out-of-range keys'):
        tr.assemble_stencil(broken)


def test_nonfinite_weights_and_entry_budget_raise_as_before():
    tr, st = _transfer('shell', torch.float64)
    g = st.rule.groups[0]
    weights = g.weights.clone()
    weights[1, 0] = float('inf')
    rule = InteractionRule((QuadratureGroup(g.cells, g.values, weights, g.order), *st.rule.groups[1:]), st.rule.orders,
                           st.rule.point_count)
    with pytest.raises(FloatingPointError, match='nonfinite'):
        tr.assemble_stencil(SharedAdaptiveStencil(st.base, st.phi, rule))
    total = tr.assemble_stencil(st).assembly['total_nnz']
    tr.max_entries = total - 1
    with pytest.raises(RuntimeError, match='budget exceeded'):
        tr.assemble_stencil(st)
    tr.max_entries = total
    assert tr.assemble_stencil(st).assembly['total_nnz'] == total
