"""Fused Arnoldi step and marching Helmholtz sweeps (csrc/fgmres.cu,
csrc/stokes.cu) against plain torch in 64 bits (B200).

Arnoldi: coefficients and the new row are sums of n products, within n u of the
exact ones; the second pass leaves the row orthogonal to some u.  Sweeps: the
same operations in the same order, so bitwise equal in FP64.
"""
import numpy as np
import pytest
import torch
from oracle import stokes as ostokes
from afsi_gpu_b200 import _lib
from afsi_gpu_b200.grid import MACGrid
from afsi_gpu_b200.helmholtz import HelmholtzKernels
from afsi_gpu_b200.stokes_fgmres import GMRESOptions, _Arnoldi, gmres

pytestmark = pytest.mark.gpu
DEV = 'cuda'


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('n,k', [(1, 1), (7, 3), (255, 4), (257, 5), (5000, 21), (200003, 9)])
def test_arnoldi_step(n, k, dtype):
    g = torch.Generator(device=DEV).manual_seed(n + k)
    rows = min(k, n)
    q = torch.linalg.qr(torch.randn((n, rows), device=DEV, dtype=torch.float64, generator=g))[0]
    V = torch.zeros((rows + 1, n), device=DEV, dtype=dtype)
    V[:rows] = q.t().to(dtype)
    w = torch.randn(n, device=DEV, dtype=torch.float64, generator=g).to(dtype)
    kept = w.clone()
    column = _Arnoldi(V).step(rows - 1, w)
    assert torch.equal(w, kept)
    B, x = V[:rows].double(), w.double()
    c = B @ x
    y = x - B.t() @ c
    d = B @ y
    z = y - B.t() @ d
    u = torch.finfo(dtype).eps
    tol = 4 * u * float(x.norm()) * max(1., rows ** .5)
    ref = (c + d).tolist()
    assert len(column) == rows + 2
    assert max(abs(a - b) for a, b in zip(column, ref)) <= tol
    assert abs(column[-2] - float(z.norm())) <= tol and abs(column[-1] - float(x.norm())) <= tol
    if n > 2 * rows:
        assert float((V[rows].double() - z / z.norm()).abs().max()) <= 8 * u
        assert float((B @ V[rows].double()).abs().max()) <= 8 * u


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_gmres_solves_on_either_side_and_leaves_the_action_alone(dtype):
    n = 300
    A = torch.randn((n, n), dtype=torch.float64, generator=torch.Generator().manual_seed(2)) / n ** .5 + 3 * torch.eye(n)
    b = torch.randn(n, dtype=torch.float64, generator=torch.Generator().manual_seed(3))
    opts = GMRESOptions(rtol=1e-10 if dtype == torch.float64 else 1e-4, restart=40, max_iterations=200)
    infos = []
    for dev in (DEV, 'cpu'):
        M, r = A.to(dev, dtype), b.to(dev, dtype)
        x, info = gmres(lambda v: M @ v, r, options=opts)
        assert float((M @ x - r).norm()) <= info['tolerance'] * (1 + 1e-6)
        infos.append(info['iterations'])
    assert infos[0] == infos[1]
    # an action that returns its argument: the basis must not be written through it
    r = b.to(DEV, dtype)
    x, info = gmres(lambda v: v, r, options=opts)
    assert info['iterations'] == 1 or torch.allclose(x, r)
    assert torch.allclose(x, r, rtol=1e-4)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('shape,lengths', [((4, 4, 4), (1., 1., 1.)), ((5, 9, 17), (1., .7, 1.3)),
                                          ((33, 4, 31), (1., 1., 1.)), ((16, 32, 8), (1., 2., .5)),
                                          ((130, 12, 15), (2., 1., 1.))])
def test_helmholtz_columns(shape, lengths, dtype):
    grid = MACGrid(shape, lengths)
    rng = np.random.default_rng(3)
    npt = np.float64 if dtype == torch.float64 else np.float32
    b = [rng.standard_normal(grid.face_shape(c)).astype(npt) for c in range(3)]
    p = rng.standard_normal(shape).astype(npt)
    alpha, scale = 3e-4, .25
    diag = [d.astype(npt) for d in ostokes.cn_diagonal(shape, grid.spacing, alpha)]
    rhs, u = ostokes.helmholtz_initialize(b, p, diag, scale, grid.spacing)
    t = lambda a: tuple(torch.as_tensor(v, device=DEV) for v in a)
    k = HelmholtzKernels()
    R, A, B = (tuple(torch.empty_like(v) for v in t(b)) for _ in range(3))
    D = t(diag)
    param = torch.tensor([alpha, scale], device=DEV, dtype=dtype)
    k.initialize(t(b), torch.as_tensor(p, device=DEV), D, R, A, param, grid)
    for _ in range(2):
        u = ostokes.helmholtz_sweep(u, rhs, diag, alpha, grid.spacing)
        k.sweep(A, R, D, B, param, grid)
        A, B = B, A
    for c in range(3):
        if dtype == torch.float64:
            assert np.array_equal(R[c].cpu().numpy(), rhs[c]) and np.array_equal(A[c].cpu().numpy(), u[c])
        else:
            np.testing.assert_allclose(A[c].cpu().numpy(), u[c], rtol=2e-6, atol=2e-6 * np.abs(u[c]).max())


def test_krylov_argument_errors():
    lib = _lib.load()
    assert lib.afsi_b200_krylov_scratch_bytes(0) == -1 and lib.afsi_b200_krylov_scratch_bytes(1025) == -1
    with pytest.raises(RuntimeError, match='invalid Krylov step'):
        _lib.call('afsi_b200_krylov_step', 1, 10, 0, 1, 2, 1, 1, 1 << 20, _lib.F64, None)
