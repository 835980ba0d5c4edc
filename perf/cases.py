"""The work that a user of this library has it do, as timed cases.

A case is one pass through public entry points: the binning, spread and
gather of a time step, an adaptive finite-element transfer, a pressure, mass
or Stokes solve, a batch of channel instances.  ``listed`` names the cases,
``draw`` gives more of the same ranges, ``prepare`` makes what a program has in
hand before the call (inputs from the seed, and the transfer or solver object
that it keeps), ``run`` makes one pass, ``exact`` computes the same results in
64 bits with plain torch and numpy.
"""
from functools import lru_cache
from math import ceil, log, pi, prod

import numpy as np
import torch

from afsi_gpu_b200 import cuda_ib
from afsi_gpu_b200.batch import BatchedChannels, Schedule
from afsi_gpu_b200.grid import ChannelGrid, MACGrid
from afsi_gpu_b200.mass import MassSolver, SolverOptions
from afsi_gpu_b200.multigrid import ChannelMultigrid, GeometricMultigrid
from afsi_gpu_b200.p1_csr import P1CSRTransfer
from afsi_gpu_b200.p2_cuda_transfer import P1Transfer, P2Transfer
from afsi_gpu_b200.stokes_fgmres import CNStokes

F64 = torch.float64
DTYPES = {'float32': torch.float32, 'float64': torch.float64}
CHANNEL_SHAPES = ((128, 32), (256, 64), (384, 96), (512, 128))


def listed():
    return [
        # a 2D step's transfers: closed ellipse of markers in a 256x64 channel; launches and latency
        dict(name='ib2d_256x64', kind='ib2d', shape='256x64', points=20000, dtype='float64'),
        # the same step's pressure: one small 2D multigrid solve, periodic in x
        dict(name='pressure2d_256x64', kind='pressure2d', shape='256x64', periodic=True),
        # a served 3D step's transfers: marker cloud of a shell, bins and weights made for each step
        dict(name='ib3d_64_400k', kind='ib3d', shape='64x64x64', points=400000, dtype='float64'),
        # an FSI step on a quadratic shell with stencil tables (the drop-in form of the reference's transfer)
        dict(name='p2_tables_64', kind='p2', form='tables', shape='64x64x64', nr=3, ntheta=40, nphi=64,
             dtype='float64', deterministic=False),
        # the same step without tables, the form that a program of this library uses
        dict(name='p2_free_64', kind='p2', form='free', shape='64x64x64', nr=3, ntheta=40, nphi=64,
             dtype='float64', deterministic=False),
        # linear shell on a fine grid, operators assembled for each configuration and applied both ways
        dict(name='p1_csr_128', kind='p1csr', shape='128x128x128', nr=2, ntheta=80, nphi=160, dtype='float64'),
        # the same shell matrix-free in the precision form: FP64 positions, FP32 weights and transfers
        dict(name='p1_free_128_f32', kind='p1', shape='128x128x128', nr=2, ntheta=80, nphi=160, dtype='float32',
             deterministic=False),
        # the pressure solve of a 3D step, ordinary and large
        dict(name='pressure3d_64', kind='pressure3d', shape='64x64x64'),
        dict(name='pressure3d_128', kind='pressure3d', shape='128x128x128'),
        # the consistent-mass solve around every finite-element transfer, three columns at once
        dict(name='mass_p2_shell', kind='mass', nr=3, ntheta=40, nphi=64, check_every=4),
        # the coupled velocity-pressure solve of a Crank-Nicolson step
        dict(name='stokes_64', kind='stokes', shape='64x64x64', precision='fp64'),
        # 60 independent channel instances stepped together to the FP64 tolerance
        dict(name='batch_60', kind='batch', count=60, points_lo=5000, points_hi=40000, layout_seed=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(log(lo), log(hi)))))


def _box(rng, sizes):
    n = rng.choice(sizes)
    flat = rng.choice((n, n, n // 2))
    return 'x'.join(str(v) for v in rng.choice(((n, n, n), (n, n, flat), (n, flat, n))))


def _shell(rng, n, theta, phi):
    """Shell divisions for a grid of n cells per axis, as multiples of n."""
    return dict(ntheta=max(6, int(n * rng.uniform(*theta))), nphi=2 * max(4, int(n * rng.uniform(*phi) / 2)))


def draw(rng):
    kind = rng.choice(('ib2d', 'pressure2d', 'ib3d', 'ib3d', 'p2', 'p2', 'p1csr', 'p1', 'pressure3d', 'pressure3d',
                       'mass', 'stokes', 'batch'))
    dtype = rng.choice(('float64', 'float64', 'float32'))
    if kind == 'ib2d':
        nx, ny = rng.choice(CHANNEL_SHAPES + ((250, 61), (97, 40)))
        return dict(kind=kind, shape=f'{nx}x{ny}', points=_log_int(rng, 1000, 200000), dtype=dtype)
    if kind == 'pressure2d':
        nx, ny = rng.choice(CHANNEL_SHAPES + ((160, 48), (192, 96)))
        return dict(kind=kind, shape=f'{nx}x{ny}', periodic=rng.random() < .5, layout_seed=rng.randrange(1 << 20))
    if kind == 'ib3d':
        return dict(kind=kind, shape=_box(rng, (32, 45, 48, 64, 96)), points=_log_int(rng, 20000, 400000), dtype=dtype)
    if kind == 'p2':
        n = rng.choice((32, 40, 48, 64))
        det = rng.random() < .25
        # coarse elements reach rules of hundreds of points; on the fine grid, and for
        # the deterministic spread's bounded boxes, elements stay near one cell
        size = ((.55, .625), (.85, 1.)) if det or n == 64 else ((.4, .625), (.7, 1.))
        return dict(kind=kind, form=rng.choice(('tables', 'free', 'free')), shape=f'{n}x{n}x{n}',
                    nr=3 if n == 64 else rng.choice((2, 3)), dtype=dtype, deterministic=det, **_shell(rng, n, *size))
    if kind in ('p1csr', 'p1'):
        n = rng.choice((32, 48, 64, 96))
        d = dict(kind=kind, shape=f'{n}x{n}x{n}', nr=rng.choice((1, 2)), dtype=dtype,
                 **_shell(rng, n, (.4, .65), (.7, 1.2)))
        return d if kind == 'p1csr' else dict(d, deterministic=rng.random() < .25)
    if kind == 'pressure3d':
        return dict(kind=kind, shape=_box(rng, (32, 48, 64, 80, 96, 128)), layout_seed=rng.randrange(1 << 20))
    if kind == 'mass':
        return dict(kind=kind, nr=rng.choice((1, 2, 3)), ntheta=rng.randrange(10, 40), nphi=2 * rng.randrange(8, 32),
                    check_every=rng.choice((1, 4, 5)))
    if kind == 'stokes':
        return dict(kind=kind, shape=_box(rng, (32, 48, 64)), precision=rng.choice(('fp64', 'fp32-preconditioner')),
                    layout_seed=rng.randrange(1 << 20))
    lo = _log_int(rng, 500, 5000)
    return dict(kind=kind, count=rng.randrange(3, 49), points_lo=lo, points_hi=lo + _log_int(rng, 1000, 30000),
                layout_seed=rng.randrange(1 << 20))


# ------------------------------------------------------------------- inputs

def _shape(case):
    return tuple(int(v) for v in case['shape'].split('x'))


def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _normal(shape, g, dtype=F64):
    return torch.randn(shape, generator=g, device='cuda', dtype=F64).to(dtype)


def _uniform(shape, g, lo, hi):
    return torch.rand(shape, generator=g, device='cuda', dtype=F64) * (hi - lo) + lo


def _faces(shape, c):
    return tuple(n + (a == c) for a, n in enumerate(shape))


def _smooth_faces(shape, lengths, g, dtype=F64, modes=8):
    """One face array per component: a sum of `modes` Fourier modes."""
    out = []
    for c in range(len(shape)):
        total = 0.
        for _ in range(modes):
            amp = _normal((1,), g)
            for a, (n, length) in enumerate(zip(_faces(shape, c), lengths)):
                x = (torch.arange(n, device='cuda', dtype=F64) + .5 * (a != c)) * (length / shape[a])
                k = torch.randint(1, 6, (1,), generator=g, device='cuda')
                wave = torch.sin(2 * pi * k * x / length + _uniform((1,), g, 0., 2 * pi))
                amp = amp[..., None] * wave
            total = total + amp[0]
        out.append(total.to(dtype).contiguous())
    return tuple(out)


def _mean_free(shape, g, dtype=F64):
    r = _normal(shape, g)
    return (r - r.mean()).to(dtype)


def _ellipse(points, g, lengths, h):
    t = torch.arange(points, device='cuda', dtype=F64) * (2 * pi / points)
    a, b = .3 * lengths[0], .4 * lengths[1]
    r = 1 + _uniform((points,), g, -.2 * h, .2 * h) / torch.hypot(a * torch.cos(t), b * torch.sin(t))
    return torch.stack((.5 * lengths[0] + a * r * torch.cos(t), .5 * lengths[1] + b * r * torch.sin(t)), -1)


def _cloud(points, g):
    """Markers of a truncated prolate shell in the unit box, in no order."""
    th, ph = _uniform((points,), g, .12 * pi, .72 * pi), _uniform((points,), g, 0., 2 * pi)
    s = _uniform((points,), g, 0., 1.)
    a, b = .25 + .07 * s, .15 + .07 * s
    return torch.stack((.5 - a * torch.cos(th), .5 + b * torch.sin(th) * torch.cos(ph),
                        .5 + b * torch.sin(th) * torch.sin(ph)), -1)


@lru_cache(maxsize=8)
def _mesh(nr, ntheta, nphi, inner, outer, quadratic):
    """Tetrahedra of a truncated prolate shell: five per cell of a (radial,
    polar, azimuthal) lattice, the two mirror splits in a checkerboard; with
    one shared midpoint per edge for quadratic elements."""
    s, t = np.linspace(0, 1, nr + 1), np.linspace(.12 * pi, .72 * pi, ntheta + 1)
    f = np.arange(nphi) * (2 * pi / nphi)
    S, T, P = np.meshgrid(s, t, f, indexing='ij')
    a, b = (inner[k] + S * (outer[k] - inner[k]) for k in (0, 1))
    X = np.stack((.5 - a * np.cos(T), .5 + b * np.sin(T) * np.cos(P), .5 + b * np.sin(T) * np.sin(P)), -1)
    I, J, K = np.meshgrid(np.arange(nr), np.arange(ntheta), np.arange(nphi), indexing='ij')
    corner = np.stack([((I + (v & 1)) * (ntheta + 1) + J + ((v >> 1) & 1)) * nphi + (K + (v >> 2)) % nphi
                       for v in range(8)], -1).reshape(-1, 8)
    splits = np.array([[(0, 3, 5, 6)] + [(v, v ^ 1, v ^ 2, v ^ 4) for v in (1, 2, 4, 7)],
                       [(1, 2, 4, 7)] + [(v, v ^ 1, v ^ 2, v ^ 4) for v in (0, 3, 5, 6)]])
    odd = ((I + J + K) % 2).reshape(-1)
    cells = np.take_along_axis(corner[:, None, :], splits[odd].reshape(-1, 20)[:, None, :], -1).reshape(-1, 4)
    X = X.reshape(-1, 3)
    if quadratic:
        edges = np.array(((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)))
        ends = np.sort(cells[:, edges].reshape(-1, 2), 1)
        keys, inverse = np.unique(ends[:, 0] * len(X) + ends[:, 1], return_inverse=True)
        cells = np.concatenate((cells, len(X) + inverse.reshape(-1, 6)), 1)
        X = np.concatenate((X, X[np.stack((keys // len(X), keys % len(X)), 1)].mean(1)))
    return X, cells.astype(np.int64)


def _structure(case, seed):
    """Reference positions, connectivity and this seed's positions: the shell
    moved and slightly deformed, as between the steps of a run."""
    quadratic = case['kind'] in ('p2', 'mass')
    walls = dict(inner=(.25, .15), outer=(.32, .22)) if quadratic else dict(inner=(.214, .144), outer=(.224, .154))
    X, cells = _mesh(case['nr'], case['ntheta'], case['nphi'], quadratic=quadratic, **walls)
    X = torch.as_tensor(X, device='cuda')
    g = _generator(seed)
    amp = _uniform((3,), g, -.004, .004)
    phase = _uniform((3,), g, 0., 2 * pi)
    x = X + _uniform((3,), g, -.02, .02) + amp * torch.sin(2 * pi * X.roll(1, 1) + phase)
    return X, torch.as_tensor(cells, device='cuda'), x, g


def _fe_inputs(case, seed):
    X, cells, x, g = _structure(case, seed)
    dtype = DTYPES[case['dtype']]
    coef = _normal(X.shape, g, dtype) if case['kind'] == 'p2' else _uniform(X.shape, g, -1., 1.).to(dtype)
    vel = _smooth_faces(_shape(case), (1., 1., 1.), g, dtype)
    return X, cells, x, coef, vel


def _mass_matrix(case, seed):
    """Consistent quadratic mass matrix of the deformed shell (degree-5 rule):
    (rows, cols, values) of the coalesced matrix, and its diagonal."""
    _, cells, x, g = _structure(case, seed)
    q, w = _keast()
    N = torch.as_tensor(_tabulate(q, True), device='cuda')
    W = _volumes(x, cells)[:, None] * torch.as_tensor(w, device='cuda')
    local = torch.einsum('eq,qa,qb->eab', W, N, N)
    ij = torch.stack((cells[:, :, None].expand_as(local).reshape(-1), cells[:, None, :].expand_as(local).reshape(-1)))
    M = torch.sparse_coo_tensor(ij, local.reshape(-1), (len(x), len(x))).coalesce()
    diag = torch.zeros(len(x), device='cuda', dtype=F64).index_add_(
        0, cells.reshape(-1), local.diagonal(dim1=-2, dim2=-1).reshape(-1))
    return M, diag, _normal((len(x), 3), g)


def _divergence_free(shape, g):
    """Face field with zero discrete divergence and no flux through the walls."""
    h = [1. / n for n in shape]
    pot = []
    for c in range(3):
        a = _normal(tuple(n + (k != c) for k, n in enumerate(shape)), g)
        for k in range(3):
            if k != c:
                a.select(k, 0).zero_()
                a.select(k, shape[k]).zero_()
        pot.append(a)
    return tuple((torch.diff(pot[(c + 2) % 3], dim=(c + 1) % 3) / h[(c + 1) % 3]
                  - torch.diff(pot[(c + 1) % 3], dim=(c + 2) % 3) / h[(c + 2) % 3]).contiguous() for c in range(3))


def _batch_inputs(case, seed):
    layout = np.random.default_rng(case['layout_seed'])
    sizes = [(CHANNEL_SHAPES[int(layout.integers(4))], int(layout.integers(case['points_lo'], case['points_hi'] + 1)))
             for _ in range(case['count'])]
    g = _generator(seed)
    out = []
    for shape, points in sizes:
        s = _uniform((points,), g, 0., 1.)
        lower = torch.arange(points, device='cuda') < points // 2
        x = 4. * torch.where(lower, .35, .45) + .32 * s * s + _uniform((points,), g, -.25, .25) * (4. / shape[0])
        y = torch.where(lower, .02 + .4 * s, .98 - .4 * s)
        out.append((shape, torch.stack((x, y), -1), _normal((points, 2), g), _smooth_faces(shape, (4., 1.), g),
                    _mean_free(shape, g)))
    return out


STOKES = dict(dt=1e-3, rho=1., mu=.01)
BATCH_SCHEDULE = dict(streams=1, order='given', smoother='jacobi', cycles=5, vcycles='batched', refined=True)


def prepare(case, seed):
    kind = case['kind']
    g = _generator(seed)
    if kind == 'ib2d':
        shape = _shape(case)
        dtype = DTYPES[case['dtype']]
        grid = ChannelGrid(shape, (1., .25))
        x = _ellipse(case['points'], g, grid.lengths, grid.spacing[0]).to(dtype)
        return dict(case=case, grid=grid, x=x, force=_normal(x.shape, g, dtype),
                    vel=_smooth_faces(shape, grid.lengths, g, dtype))
    if kind == 'pressure2d':
        grid = ChannelGrid(_shape(case), (1., .25), periodic=case['periodic'])
        return dict(case=case, solver=ChannelMultigrid(grid), rhs=_mean_free(grid.shape, g))
    if kind == 'ib3d':
        shape = _shape(case)
        dtype = DTYPES[case['dtype']]
        x = _cloud(case['points'], g).to(dtype)
        return dict(case=case, grid=MACGrid(shape, (1., 1., 1.)), x=x, force=_normal(x.shape, g, dtype),
                    vel=_smooth_faces(shape, (1., 1., 1.), g, dtype))
    if kind in ('p2', 'p1', 'p1csr'):
        grid = MACGrid(_shape(case), (1., 1., 1.))
        X, cells, x, coef, vel = _fe_inputs(case, seed)
        kw = {} if kind == 'p1csr' else dict(deterministic=case['deterministic'])
        cls = {'p2': P2Transfer, 'p1': P1Transfer, 'p1csr': P1CSRTransfer}[kind]
        tr = cls(grid, X, cells, max_order=22, transfer_dtype=DTYPES[case['dtype']], **kw)
        return dict(case=case, transfer=tr, x=x, coef=coef, vel=vel)
    if kind == 'pressure3d':
        grid = MACGrid(_shape(case), (1., 1., 1.))
        return dict(case=case, solver=GeometricMultigrid(grid), rhs=_mean_free(grid.shape, g))
    if kind == 'mass':
        M, diag, rhs = _mass_matrix(case, seed)
        solver = MassSolver(M.to_sparse_csr(), diag[:, None].expand(-1, 3),
                            SolverOptions(rtol=1e-12, atol=1e-13, max_iterations=500,
                                          check_every=case['check_every']))
        return dict(case=case, solver=solver, rhs=rhs)
    if kind == 'stokes':
        grid = MACGrid(_shape(case), (1., 1., 1.))
        return dict(case=case, flow=CNStokes(grid, precision=case['precision'], **STOKES),
                    b=_divergence_free(grid.shape, g))
    rows = _batch_inputs(case, seed)
    cpu = [(s, x.cpu(), f.cpu(), [v.cpu() for v in vel], r.cpu()) for s, x, f, vel, r in rows]
    batch = BatchedChannels([ChannelGrid(r[0], (4., 1.)) for r in cpu], *([r[k] for r in cpu] for k in range(1, 5)),
                            transfer_dtype=F64, schedule=Schedule(**BATCH_SCHEDULE))
    batch.use(batch.schedule)
    return dict(case=case, batch=batch)


# ---------------------------------------------------------------------- run

def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'ib2d':
        st = cuda_ib.prepare2d(state['grid'], state['x'])
        u, v = cuda_ib.spread2d(state['grid'], state['force'], st)
        return dict(u=u, v=v, velocity=cuda_ib.gather2d(state['vel'], st), ids0=st.indices[0], ids1=st.indices[1],
                    weights0=st.weights[0], weights1=st.weights[1])
    if kind == 'ib3d':
        st = cuda_ib.compact_prepare(state['grid'], state['x'])
        u, v, w = cuda_ib.compact_spread(state['grid'], state['force'], st)
        return dict(u=u, v=v, w=w, velocity=cuda_ib.compact_gather(state['grid'], state['vel'], st), base=st.base,
                    phi=st.phi)
    if kind in ('pressure2d', 'pressure3d'):
        return dict(p=state['solver'].solve(state['rhs'])[0])
    if kind in ('p2', 'p1'):
        tr = state['transfer']
        if kind == 'p2' and case['form'] == 'tables':
            st = tr.prepare(state['x'])
            u, v, w = tr.spread(state['coef'], st)
            return dict(u=u, v=v, w=w, rhs=tr.assemble_velocity(state['vel'], st))
        pending = tr.prepare_table_free(state['x'])
        u, v, w = tr.spread(state['coef'], pending.stencil)
        rhs = tr.assemble_velocity(state['vel'], pending.stencil)
        tr.note_transfers(pending)
        tr.confirm(pending)
        return dict(u=u, v=v, w=w, rhs=rhs)
    if kind == 'p1csr':
        tr = state['transfer']
        st = tr.prepare(state['x'])
        u, v, w = tr.spread(state['coef'], st)
        out = dict(u=u, v=v, w=w, rhs=tr.interpolate_rhs(state['vel'], st))
        # the operators' row pointers; their entries, whose number changes with x, are in the responses
        for c in range(3):
            out.update({f'gather{c}': st.gather[c].crow, f'spread{c}': st.spread[c].crow})
        return out
    if kind == 'mass':
        return dict(x=state['solver'].solve(state['rhs'])[0])
    if kind == 'stokes':
        res = state['flow'].stokes(state['b'])
        return dict(u=res.velocity[0], v=res.velocity[1], w=res.velocity[2], p=res.pressure)
    b = state['batch']
    b.replay()
    out = dict(u=b.u, v=b.v, velocity=b.gathered)
    for i in range(len(b.grids)):
        out[f'p{i}'] = b.pressure(i)
    return out


# --------------------------------------------------------------- work, error

def work(case):
    """Inputs read once and results written once; operations of the contraction
    or of the sweeps that the solve is made of."""
    kind = case['kind']
    if kind in ('ib2d', 'ib3d'):
        shape, P = _shape(case), case['points']
        d, s = len(shape), 4 if case['dtype'] == 'float32' else 8
        faces = sum(prod(_faces(shape, c)) for c in range(d))
        table = P * d * (16 * (8 + s) if d == 2 else 3 * (8 + 4 * s))
        return dict(bytes=3 * P * d * s + 2 * faces * s + table, flops=P * d * (4 ** d) * 2 * 3)
    if kind in ('pressure2d', 'pressure3d'):
        n = prod(_shape(case))
        sweeps = 12 * (8 + 2) * (8 / 7 if kind == 'pressure3d' else 4 / 3)
        return dict(bytes=2 * n * 8, flops=n * sweeps * (17 if kind == 'pressure3d' else 12))
    if kind in ('p2', 'p1', 'p1csr', 'mass'):
        hexes = case['nr'] * case['ntheta'] * case['nphi']
        corners = (case['nr'] + 1) * (case['ntheta'] + 1) * case['nphi']
        E, npc = 5 * hexes, 10 if kind in ('p2', 'mass') else 4
        nodes = corners if npc == 4 else corners + 6 * hexes + 4 * corners // 2
        if kind == 'mass':
            nnz = 25 * nodes
            return dict(bytes=nnz * 12 + nodes * (8 + 2 * 24), flops=60 * nodes * (25 * 6 + 3 * 14))
        s = 4 if case['dtype'] == 'float32' else 8
        shape = _shape(case)
        faces = sum(prod(_faces(shape, c)) for c in range(3))
        # points per element at density 2 for elements of about a grid spacing
        q = 64 if npc == 10 else 8
        nbytes = E * (8 * npc + q * s) + nodes * (24 + 2 * 3 * s) + 2 * faces * s
        if kind == 'p1csr':
            nbytes += 3 * 2 * (nodes * 130 * 16 + 8 * faces // 3)
        return dict(bytes=nbytes, flops=E * q * 3 * (2 * 64 * 2 + npc * 4 + 60))
    if kind == 'stokes':
        n = prod(_shape(case))
        return dict(bytes=2 * 4 * n * 8, flops=n * 7 * (3 * 14 * 22 + 2 * 11.5 * 17 + 4 * 24))
    cells = case['count'] * 256 * 75
    P = case['count'] * (case['points_lo'] + case['points_hi']) // 2
    return dict(bytes=P * 2 * 3 * 8 + cells * 8 * 6, flops=P * 2 * 16 * 6 + cells * 12 * 10 * 4 / 3 * 12)


def tolerance(case):
    """Transfers: rounding of the data type in sums of another order (atomic
    additions: 2e-15 and 4.5e-14 the largest seen between two runs in
    FP64, 4.4e-7 and 1.3e-5 in FP32).  Solves: the stopping rule leaves a relative
    residual of up to 1e-10 (1e-12 for the mass solve), and with it an error of
    the solution of that order (1.4e-10 to 2.4e-10 for the pressures, 4e-13 for
    the mass solve, 1e-11 to 6e-9 for the coupled pressure, whose Krylov loop
    stops between checks)."""
    kind = case['kind']
    if kind in ('ib2d', 'ib3d', 'p2', 'p1', 'p1csr'):
        return dict(rel=2e-6, max=6e-5) if case['dtype'] == 'float32' else dict(rel=1e-14, max=4e-13)
    return {'mass': dict(rel=2e-12, max=5e-11), 'stokes': dict(rel=3e-8, max=1e-6),
            'batch': dict(rel=3e-10, max=1e-8)}.get(kind, dict(rel=1e-9, max=2e-8))


# -------------------------------------------------------------------- exact

def _peskin(r):
    r = r.abs()
    a, b = r.clamp(max=1.), r.clamp(min=1., max=2.)
    inner = (3 - 2 * a + torch.sqrt(1 + 4 * a - 4 * a * a)) / 8
    outer = (5 - 2 * b - torch.sqrt((-7 + 12 * b - 4 * b * b).clamp(min=0.))) / 8
    return torch.where(r < 1, inner, torch.where(r < 2, outer, torch.zeros_like(r)))


def _bins(x, start, h):
    """Lower support index and the four weights of every coordinate."""
    scaled = (x - start) / h
    lower = torch.floor(scaled - 1)
    k = torch.arange(4, device=x.device, dtype=x.dtype)
    return lower.long(), _peskin(scaled[..., None] - (lower[..., None] + k))


def _stencil3(x, shape, c):
    """Flat face indices (P,64) and weights (P,64) of component c."""
    n = _faces(shape, c)
    bins = [_bins(x[:, a], 0. if a == c else .5 / shape[a], 1. / shape[a]) for a in range(3)]
    k = torch.arange(4, device=x.device)
    i = [b[0][:, None] + k for b in bins]
    flat = (i[0][:, :, None, None] * n[1] + i[1][:, None, :, None]) * n[2] + i[2][:, None, None, :]
    w = bins[0][1][:, :, None, None] * bins[1][1][:, None, :, None] * bins[2][1][:, None, None, :]
    return flat.reshape(len(x), 64), w.reshape(len(x), 64)


def _transfer3(x, force, vel, shape):
    """Spread and gather of a point set in chunks: fields and point velocities."""
    vol = 1. / prod(shape)
    fields, out = [], torch.empty(x.shape, device=x.device, dtype=F64)
    for c in range(3):
        f = torch.zeros(prod(_faces(shape, c)), device=x.device, dtype=F64)
        for lo in range(0, len(x), 1 << 18):
            s = slice(lo, lo + (1 << 18))
            ids, w = _stencil3(x[s], shape, c)
            f.index_add_(0, ids.reshape(-1), (w * force[s, c, None] / vol).reshape(-1))
            out[s, c] = (vel[c].reshape(-1)[ids] * w).sum(1)
        fields.append(f.view(_faces(shape, c)))
    return fields, out


def _exact_ib3d(case, seed):
    st = prepare(case, seed)
    x, force, vel = st['x'].double(), st['force'].double(), [v.double() for v in st['vel']]
    shape = _shape(case)
    (u, v, w), velocity = _transfer3(x, force, vel, shape)
    phi = torch.stack([torch.stack([_bins(x[:, a], 0. if a == c else .5 / shape[a], 1. / shape[a])[1]
                                    for a in range(3)], 1) for c in range(3)])
    # bins of 32-bit coordinates are the 32-bit arithmetic's own
    return dict(u=u, v=v, w=w, velocity=velocity, base=None, phi=phi if case['dtype'] == 'float64' else None)


def _stencil2(x, shape, lengths, c):
    h = [length / n for length, n in zip(lengths, shape)]
    (bx, wx), (by, wy) = (_bins(x[:, a], 0. if a == c else .5 * h[a], h[a]) for a in range(2))
    k = torch.arange(4, device=x.device)
    ny = shape[1]
    y = by[:, None] + k
    if c == 0:
        r, out = torch.where(y < 0, -y - 1, torch.where(y >= ny, 2 * ny - y - 1, y)), (y < 0) | (y >= ny)
    else:
        r, out = torch.where(y < 0, -y, torch.where(y > ny, 2 * ny - y, y)), (y < 0) | (y > ny)
    ids = (bx[:, None] + k)[:, :, None] * (ny + c) + r[:, None, :]
    w = wx[:, :, None] * torch.where(out, -wy, wy)[:, None, :]
    return ids.reshape(len(x), 16), w.reshape(len(x), 16)


def _transfer2(x, force, vel, shape, lengths):
    vol = prod(length / n for length, n in zip(lengths, shape))
    fields, velocity, tables = [], [], []
    for c in range(2):
        ids, w = _stencil2(x, shape, lengths, c)
        f = torch.zeros(prod(_faces(shape, c)), device=x.device, dtype=F64)
        f.index_add_(0, ids.reshape(-1), (w * force[:, c, None] / vol).reshape(-1))
        fields.append(f.view(_faces(shape, c)))
        velocity.append((vel[c].reshape(-1)[ids] * w).sum(1))
        tables.append(w)
    return fields, torch.stack(velocity, 1), tables


def _exact_ib2d(case, seed):
    st = prepare(case, seed)
    (u, v), velocity, w = _transfer2(st['x'].double(), st['force'].double(), [a.double() for a in st['vel']],
                                     _shape(case), st['grid'].lengths)
    if case['dtype'] == 'float32':
        w = [None, None]
    return dict(u=u, v=v, velocity=velocity, ids0=None, ids1=None, weights0=w[0], weights1=w[1])


def _keast():
    """Keast's 15-point rule of degree 5 on the unit tetrahedron."""
    from itertools import permutations
    a = .4334498464263357
    orbits = (((.25,) * 4, .030283678097089182), ((0., 1 / 3, 1 / 3, 1 / 3), .006026785714285717),
              ((8 / 11, 1 / 11, 1 / 11, 1 / 11), .011645249086028967), ((a, a, .5 - a, .5 - a), .010949141561386449))
    rows = [(p[1:], w) for orbit, w in orbits for p in sorted(set(permutations(orbit)))]
    return np.array([r[0] for r in rows]), np.array([r[1] for r in rows])


def _collapsed(n):
    """Collapsed Gauss-Jacobi product rule with n points per direction."""
    def rule(alpha):
        k = np.arange(n, dtype=float)
        diag = np.zeros(n) if not alpha else -alpha ** 2 / ((2 * k + alpha) * (2 * k + alpha + 2))
        j = np.arange(1, n, dtype=float)
        m = 2 * j + alpha
        off = np.sqrt(4 * (j * (j + alpha)) ** 2 / (m * m * (m * m - 1)))
        t, V = np.linalg.eigh(np.diag(diag) + np.diag(off, 1) + np.diag(off, -1))
        return (t + 1) / 2, V[0] ** 2 / (alpha + 1)
    (u, a), (v, b), (w, c) = (rule(al) for al in (2, 1, 0))
    U, V, W = np.meshgrid(u, v, w, indexing='ij')
    pts = np.stack((U, (1 - U) * V, (1 - U) * (1 - V) * W), -1).reshape(-1, 3)
    return pts, np.einsum('i,j,k->ijk', a, b, c).reshape(-1)


def _tabulate(q, quadratic):
    L = np.concatenate((1 - q.sum(1, keepdims=True), q), 1)
    if not quadratic:
        return L
    i, j = np.array((0, 0, 0, 1, 1, 2)), np.array((1, 2, 3, 2, 3, 3))
    return np.concatenate((L * (2 * L - 1), 4 * L[:, i] * L[:, j]), 1)


def _volumes(X, cells):
    v = X[cells[:, :4]]
    return torch.linalg.det(v[:, 1:] - v[:, :1]).abs()


def _orders(x, cells, dx, quadratic):
    p = x[cells]
    if quadratic:
        i, j = (0, 0, 0, 1, 1, 2), (1, 2, 3, 2, 3, 3)
        p = torch.cat((p[:, :4], 2 * p[:, 4:] - .5 * (p[:, i] + p[:, j])), 1)
    d = torch.cdist(p, p, compute_mode='donot_use_mm_for_euclid_dist').amax((1, 2))
    return torch.ceil(2. * d / dx).long().clamp(min=3 if quadratic else 2)


def _exact_fe(case, seed):
    """Quadrature transfer of the elements, group by group, in chunks."""
    quadratic = case['kind'] == 'p2'
    X, cells, x, coef, vel = _fe_inputs(case, seed)
    coef, vel, shape = coef.double(), [v.double() for v in vel], _shape(case)
    dets = _volumes(X, cells)
    orders = _orders(x, cells, 1. / max(shape), quadratic)
    fields = [torch.zeros(_faces(shape, c), device='cuda', dtype=F64) for c in range(3)]
    rhs = torch.zeros(X.shape, device='cuda', dtype=F64)
    for n in orders.unique().tolist():
        q, w = _keast() if n == 3 else _collapsed(n)
        N = torch.as_tensor(_tabulate(q, quadratic), device='cuda')
        ids = torch.where(orders == n)[0]
        step = max(1, (1 << 18) // len(w))
        for lo in range(0, len(ids), step):
            e = ids[lo:lo + step]
            W = dets[e, None] * torch.as_tensor(w, device='cuda')
            pos = torch.einsum('qa,ead->eqd', N, x[cells[e]]).reshape(-1, 3)
            force = torch.einsum('qa,ead->eqd', N, coef[cells[e]]) * W[..., None]
            part, U = _transfer3(pos, force.reshape(-1, 3), vel, shape)
            for f, add in zip(fields, part):
                f += add
            local = torch.einsum('qa,eq,eqd->ead', N, W, U.view(len(e), -1, 3))
            rhs.index_add_(0, cells[e].reshape(-1), local.reshape(-1, 3))
    return dict(u=fields[0], v=fields[1], w=fields[2], rhs=rhs)


def _exact_p1csr(case, seed):
    return dict(_exact_fe(case, seed), **{f'{name}{c}': None for c in range(3) for name in ('gather', 'spread')})


def _axis(n, h, kind):
    """1D operator -d2/dx2 of one axis as a dense symmetric matrix.  kind: 'wall'
    (zero flux), 'wrap', 'outlet' (zero flux, then zero value half a cell past
    the end), 'odd' (zero value half a cell past both ends), 'node' (interior
    nodes between two zero end nodes)."""
    A = torch.zeros((n, n), dtype=F64)
    i = torch.arange(n - 1)
    A[i, i + 1] = A[i + 1, i] = -1.
    A[range(n), range(n)] = 2.
    if kind in ('wall', 'outlet'):
        A[0, 0] = 1.
        A[-1, -1] = 1. if kind == 'wall' else 3.
    elif kind == 'wrap':
        A[0, -1] += -1.
        A[-1, 0] += -1.
    elif kind == 'odd':
        A[0, 0] = A[-1, -1] = 3.
    return (A / h ** 2).cuda()


class _Separable:
    """(shift + scale * sum of 1D operators)^-1 through their eigenvectors; a
    zero eigenvalue of the sum (pure zero-flux or periodic) maps to zero."""

    def __init__(self, axes, shift=0., scale=1.):
        pairs = [torch.linalg.eigh(A) for A in axes]
        self.V = [p[1] for p in pairs]
        total = shift
        for a, (lam, _) in enumerate(pairs):
            total = total + scale * lam.reshape([-1 if k == a else 1 for k in range(len(axes))])
        self.inverse = torch.where(total.abs() > 1e-9 * total.abs().max(), 1 / total, torch.zeros_like(total))

    def __call__(self, r):
        for a, V in enumerate(self.V):
            r = torch.tensordot(V.t(), r, dims=([1], [a])).movedim(0, a)
        r = r * self.inverse
        for a, V in enumerate(self.V):
            r = torch.tensordot(V, r, dims=([1], [a])).movedim(0, a)
        return r.contiguous()


def _exact_pressure(case, seed):
    shape = _shape(case)
    if len(shape) == 2:
        kinds, lengths = ('wrap' if case['periodic'] else 'outlet', 'wall'), (1., .25)
    else:
        kinds, lengths = ('wall',) * 3, (1.,) * 3
    inverse = _Separable([_axis(n, length / n, k) for n, length, k in zip(shape, lengths, kinds)])
    p = inverse(_mean_free(shape, _generator(seed)))
    return dict(p=p if kinds[0] == 'outlet' else p - p.mean())


def _exact_mass(case, seed):
    """Jacobi-preconditioned conjugate gradients, far past the stated tolerance."""
    M, diag, b = _mass_matrix(case, seed)
    M, d = M.to_sparse_csr(), diag[:, None]
    x = torch.zeros_like(b)
    for _ in range(3):  # restarted from the true residual
        r = b - M @ x
        z = r / d
        p, rz = z.clone(), (r * z).sum()
        for _ in range(70):
            Ap = M @ p
            alpha = rz / (p * Ap).sum()
            x, r = x + alpha * p, r - alpha * Ap
            z = r / d
            new = (r * z).sum()
            p, rz = z + (new / rz) * p, new
            if float(new) == 0.:
                break
    return dict(x=x)


def _exact_stokes(case, seed):
    """Pressure Schur complement of the coupled system by conjugate gradients,
    the velocity operator inverted through its eigenvectors."""
    shape = _shape(case)
    h = [1. / n for n in shape]
    b = _divergence_free(shape, _generator(seed))
    scale, alpha = STOKES['dt'] / STOKES['rho'], STOKES['dt'] * STOKES['mu'] / (2 * STOKES['rho'])
    H = [_Separable([_axis(n - 1 if a == c else n, h[a], 'node' if a == c else 'odd') for a, n in enumerate(shape)],
                    1., alpha) for c in range(3)]
    L = _Separable([_axis(n, d, 'wall') for n, d in zip(shape, h)])

    def grad(p):
        return [torch.diff(p, dim=c) / h[c] for c in range(3)]

    def div(u):
        out = 0.
        for c, v in enumerate(u):
            wall = torch.zeros_like(v.narrow(c, 0, 1))
            out = out + torch.diff(torch.cat((wall, v, wall), c), dim=c) / h[c]
        return out

    def velocity(p):
        return [inv(v.narrow(c, 1, shape[c] - 1) - scale * q) for c, (inv, v, q) in enumerate(zip(H, b, grad(p)))]

    def schur(p):  # -D H^-1 scale G
        return -div([inv(scale * q) for inv, q in zip(H, grad(p))])

    def smooth(r):  # (H on pressures) applied to the scaled Poisson inverse
        z = L(r)
        return (z + alpha * (r - r.mean())) / scale

    p = torch.zeros(shape, device='cuda', dtype=F64)
    for _ in range(2):
        r = -div(velocity(p))
        r = r - r.mean()
        z = smooth(r)
        d, rz = z.clone(), (r * z).sum()
        for _ in range(80):
            if not float(rz) > 0.:
                break
            Ad = schur(d)
            a = rz / (d * Ad).sum()
            p, r = p + a * d, r - a * Ad
            z = smooth(r)
            new = (r * z).sum()
            d, rz = z + (new / rz) * d, new
    u = [torch.nn.functional.pad(v, [n for k in (2, 1, 0) for n in ((1, 1) if k == c else (0, 0))])
         for c, v in enumerate(velocity(p))]
    return dict(u=u[0], v=u[1], w=u[2], p=p - p.mean())


def _exact_batch(case, seed):
    u, v, velocity, pressures = [], [], [], {}
    solvers = {}
    for i, (shape, x, force, vel, rhs) in enumerate(_batch_inputs(case, seed)):
        fields, U, _ = _transfer2(x, force, vel, shape, (4., 1.))
        u.append(fields[0].reshape(-1))
        v.append(fields[1].reshape(-1))
        velocity.append(U)
        if shape not in solvers:
            solvers[shape] = _Separable([_axis(shape[0], 4. / shape[0], 'outlet'), _axis(shape[1], 1. / shape[1], 'wall')])
        pressures[f'p{i}'] = solvers[shape](rhs)
    return dict(u=torch.cat(u), v=torch.cat(v), velocity=torch.cat(velocity), **pressures)


def exact(case, seed):
    kind = case['kind']
    if kind in ('pressure2d', 'pressure3d'):
        return _exact_pressure(case, seed)
    return {'ib2d': _exact_ib2d, 'ib3d': _exact_ib3d, 'p2': _exact_fe, 'p1': _exact_fe, 'p1csr': _exact_p1csr,
            'mass': _exact_mass, 'stokes': _exact_stokes, 'batch': _exact_batch}[kind](case, seed)
