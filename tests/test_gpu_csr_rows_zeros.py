"""Entries whose contributions cancel exactly, in the row assembly of P1 operators (B200).

Two points of one cell with the same rows and opposite shape values leave nothing in
a node's row.  The hash form skips a cell's zero sums and FP64 rows skip the zero sum of
one origin's points; FP32 rows add point by point and keep the entry, a zero.  The
operators' products are the same.
"""
import pytest
import torch
from afsi_gpu_b200 import synthetic
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.p1_csr import P1CSRTransfer
from afsi_gpu_b200.p2_cuda_transfer import SharedAdaptiveStencil
from afsi_gpu_b200.quadrature import InteractionRule, QuadratureGroup

pytestmark = pytest.mark.gpu
DEV = 'cuda'


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_exact_cancellation_leaves_explicit_zeros_at_most(dtype):
    X, cells = synthetic.prolate_shell(1, 4, 6, inner=(.125, .075, .075), outer=(.16, .11, .11))
    x, cells = torch.as_tensor(X, device=DEV, dtype=dtype), torch.as_tensor(cells[:1], device=DEV)
    tr = P1CSRTransfer(MACGrid((32, 32, 32), (1., 1., 1.)), x, cells, max_order=22)
    st = tr.prepare_tables(x)
    g = st.rule.groups[0]
    base, phi, values, weights = st.base.clone(), st.phi.clone(), g.values.clone(), g.weights.clone()
    base[:, 1], weights[0, 1] = base[:, 0], weights[0, 0]
    phi[:, :2] = .25  # exact products: fused sums leave no rounding of theirs
    values[:, 2] = 0
    values[0, 2], values[1, 2] = .25, -.25
    rule = InteractionRule((QuadratureGroup(g.cells, values, weights, g.order),), st.rule.orders, st.rule.point_count)
    st = SharedAdaptiveStencil(base, phi, rule)
    rows, table = tr._assemble_rows(st), tr._assemble_hash(st)
    node = int(g.cells[0, 2])
    coef = torch.randn((x.shape[0], 3), device=DEV, dtype=dtype)
    for a, b in zip(rows.gather, table.gather):
        count = int(a.crow[node + 1] - a.crow[node])
        assert count == (0 if dtype == torch.float64 else 64)
        assert not a.val[a.crow[node]:a.crow[node + 1]].any()
        assert a.nnz == b.nnz + count
    eps = torch.finfo(dtype).eps
    for a, b in zip(tr.spread(coef, rows), tr.spread(coef, table)):
        assert float((a - b).abs().max()) <= 64 * eps * float(b.abs().max())
