"""Table rows at the ends of the 64-bit range are outside the grid (B200).

Points binned without the support check can lie anywhere: coordinates beyond the
integers give the largest base, where base + 3 wraps to a negative number.  Such a
row is skipped and flagged as every other row outside is.
"""
import pytest
import torch
from afsi_gpu_b200 import cuda_ib, synthetic
from afsi_gpu_b200 import _lib
from afsi_gpu_b200._lib import call, dtype_code, ptr, status_word, stream
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.p1_csr import P1CSRTransfer
from afsi_gpu_b200.p2_cuda_transfer import SharedAdaptiveStencil

pytestmark = pytest.mark.gpu
DEV = 'cuda'
TOP = 2 ** 63 - 1
FAR = (TOP, TOP - 1, TOP - 2, TOP - 3, -TOP - 1)


def _cloud(points=200):
    g = torch.Generator(device=DEV).manual_seed(1)
    grid = MACGrid((16, 20, 12), (1., 1., 1.))
    x = .3 + .4 * torch.rand((points, 3), device=DEV, dtype=torch.float64, generator=g)
    return grid, x, torch.randn((points, 3), device=DEV, dtype=torch.float64, generator=g)


def _flagged():
    with pytest.raises(RuntimeError, match='outside the MAC grid'):
        cuda_ib.check()


@pytest.mark.parametrize('far', FAR)
@pytest.mark.parametrize('axis', [0, 1, 2])
def test_compact_rows_far_outside_are_skipped(far, axis):
    grid, x, force = _cloud()
    st = cuda_ib.compact_prepare(grid, x)
    vel = tuple(torch.randn(grid.face_shape(c), device=DEV, dtype=torch.float64) for c in range(3))
    base = st.base.clone()
    base[:, 7, axis] = far
    broken = cuda_ib.CompactStencil(base, st.phi)
    lists = cuda_ib.CompactStencil(list(base), list(st.phi))  # component by component
    without = force.clone()
    without[7] = 0
    want = cuda_ib.compact_spread(grid, without, st)
    gathered = cuda_ib.compact_gather(grid, vel, st)
    gathered[7] = 0
    for form in (broken, lists):
        for a, b in zip(cuda_ib.compact_spread(grid, force, form), want):
            assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())  # atomics in another order
        _flagged()
        assert torch.equal(cuda_ib.compact_gather(grid, vel, form), gathered)
        _flagged()
    out = [torch.empty(grid.face_shape(c), device=DEV, dtype=torch.float64) for c in range(3)]
    need = _lib.load().afsi_b200_compact_binned_bytes(base.shape[1], *grid.shape)
    work = torch.empty(need, device=DEV, dtype=torch.uint8)
    call('afsi_b200_compact_spread3_binned', ptr(force), ptr(base), ptr(st.phi), base.shape[1], *grid.shape,
         float(grid.volume), *(ptr(u) for u in out), ptr(work), need, ptr(status_word(force.device)),
         dtype_code(force.dtype), stream(force.device))
    for a, b in zip(out, want):
        assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())
    _flagged()


@pytest.mark.parametrize('value', [1e30, float('inf'), -1e30, float('nan')])
def test_points_beyond_the_integers_without_the_support_check(value):
    grid, x, force = _cloud()
    x[7, 1] = value
    st = cuda_ib.compact_prepare(grid, x, check_support=False)
    status_word(x.device).zero_()  # the prepare's own support flag
    out = cuda_ib.compact_spread(grid, torch.ones_like(force), st)
    _flagged()
    # all points but one, each of unit force spread with weights that sum to one
    for c, u in enumerate(out):
        assert float(u.sum()) * grid.volume == pytest.approx(199, rel=1e-12)
    vel = tuple(torch.ones(grid.face_shape(c), device=DEV, dtype=torch.float64) for c in range(3))
    got = cuda_ib.compact_gather(grid, vel, st)
    assert torch.equal(got[7], torch.zeros(3, device=DEV, dtype=torch.float64))
    assert float((got[torch.arange(200) != 7] - 1).abs().max()) <= 1e-14
    _flagged()


@pytest.mark.parametrize('far', FAR)
def test_assembly_and_deterministic_plan_refuse_far_rows(far):
    X, cells = synthetic.prolate_shell(1, 6, 8, inner=(.2, .12, .12), outer=(.26, .18, .18))
    x = torch.as_tensor(X, device=DEV)
    tr = P1CSRTransfer(MACGrid((24, 24, 24), (1., 1., 1.)), x, torch.as_tensor(cells, device=DEV))
    st = tr.prepare_tables(x)
    assert tr._assemble_rows(st) is not None
    points = st.rule.groups[0].values.shape[0]
    for lattice in range(2):
        base = st.base.clone()
        base[lattice, :points] = far  # a whole cell: a box of regular size, far outside
        assert tr._assemble_rows(SharedAdaptiveStencil(base, st.phi, st.rule)) is None
        total, code = base.shape[1], dtype_code(x.dtype)
        n = _lib.load().afsi_b200_det_plan_bytes(total, *tr.grid.shape, code)
        plan = torch.empty(n, device=DEV, dtype=torch.uint8)
        word = status_word(x.device)
        word.zero_()
        call('afsi_b200_det_plan', ptr(base), total, *tr.grid.shape, ptr(plan), n, ptr(word), code, stream(x.device))
        _flagged()
