"""Drop-in counterparts of ``afsi_torch.mac.cuda_ib`` on the B200 kernels.

Same function names, argument meaning, output ownership and error behaviour as
``afsi_torch/mac/cuda_ib.py:38-112`` and the ``afsi_ib_cuda`` operator schemas
(``mac/csrc/transfer.cpp:48-57``): outputs of the gathers/spreads are freshly
allocated, tensors are made contiguous, kernels run on PyTorch's current CUDA
stream, and a CPU tensor is rejected (no silent CPU fallback,
``mac/cuda_ib.py:63-66``).  Stencil indices that leave the grid do not trap
the device (the reference uses ``CUDA_KERNEL_ASSERT``); the kernels set a bit in
the device status word, which :func:`check` turns into a ``RuntimeError``.

Beyond the reference operators this module exposes the binning kernels
(:func:`compact_prepare`, :func:`prepare2d`), which the reference runs as torch
expressions.
"""
import threading
from dataclasses import dataclass
from math import prod
import torch
from . import _lib
from ._lib import call, ptr, stream, dtype_code


def build(*, verbose=False):
    """Compile (if needed) and load the native library; call before graph capture."""
    if torch.cuda.is_available() and torch.cuda.is_current_stream_capturing():
        raise RuntimeError('build the B200 IB library before CUDA Graph capture')
    from .build import build as _build
    _build(verbose=verbose)
    _lib.load()


def require_cuda(tensor):
    _lib.require_cuda(tensor)


def check(device=None, *, clear=True):
    """Raise if a kernel flagged an out-of-range stencil or support violation.

    Synchronises with the device (reads the status word)."""
    word = _lib.status_word(device if device is not None else torch.cuda.current_device())
    value = int(word.item())
    if clear:
        word.zero_()
    if value & _lib.FLAG_INDEX:
        raise RuntimeError('IB stencil index outside the MAC grid or node range')
    if value & _lib.FLAG_SUPPORT:
        raise ValueError('MAC IB support reaches a wall or is nonfinite; enlarge/refine the fluid box')
    return value


def _field(t):
    if t.dtype not in (torch.float32, torch.float64):
        raise RuntimeError('IB supports float32/float64')
    return t


def _same(t, like, dtype):
    if not t.is_cuda or t.device != like.device:
        raise RuntimeError('IB transfer requires one CUDA device')
    if t.dtype != dtype:
        raise RuntimeError('IB transfer requires contiguous matching tensors')
    if t.requires_grad:
        raise RuntimeError('IB forward transfer does not register autograd')
    return t.contiguous()


# ------------------------------------------------------------- raw operators
# Schemas of afsi_ib_cuda.{indexed_gather, indexed_spread, compact_gather,
# compact_spread} (mac/csrc/transfer.cpp:48-57) and their checks (:9-41).

def op_indexed_gather(field, indices, weights):
    field = _same(_field(field), field, field.dtype)
    indices, weights = _same(indices, field, torch.int64), _same(weights, field, field.dtype)
    if field.dim() != 2 or field.shape[1] == 0:
        raise RuntimeError('IB indexed field must be N x C')
    if indices.dim() != 2 or indices.shape[1] == 0 or indices.shape != weights.shape:
        raise RuntimeError('IB indexed stencil shape mismatch')
    if field.shape[0] == 0:
        raise RuntimeError('empty IB grid')
    P, K = indices.shape
    out = torch.empty((P, field.shape[1]), device=field.device, dtype=field.dtype)
    call('afsi_b200_indexed_gather', ptr(field), field.shape[0], field.shape[1], ptr(indices), ptr(weights),
         P, K, ptr(out), ptr(_lib.status_word(field.device)), dtype_code(field.dtype), stream(field.device))
    return out


def op_indexed_spread(field, indices, weights, size, volume):
    field = _same(_field(field), field, field.dtype)
    indices, weights = _same(indices, field, torch.int64), _same(weights, field, field.dtype)
    if field.dim() != 2 or field.shape[1] == 0:
        raise RuntimeError('IB indexed field must be N x C')
    if indices.dim() != 2 or indices.shape[1] == 0 or indices.shape != weights.shape:
        raise RuntimeError('IB indexed stencil shape mismatch')
    if not (size > 0 and volume > 0 and volume == volume and volume != float('inf')):
        raise RuntimeError('invalid IB output size/volume')
    if field.shape[0] != indices.shape[0]:
        raise RuntimeError('IB spread point count mismatch')
    out = torch.zeros((size, field.shape[1]), device=field.device, dtype=field.dtype)
    call('afsi_b200_indexed_spread', ptr(field), field.shape[0], field.shape[1], ptr(indices), ptr(weights),
         indices.shape[1], size, float(volume), ptr(out), ptr(_lib.status_word(field.device)),
         dtype_code(field.dtype), stream(field.device))
    return out


def _compact_checks(field, base, phi, nx, ny, nz, volume, spread):
    field = _same(_field(field), field, field.dtype)
    base, phi = _same(base, field, torch.int64), _same(phi, field, field.dtype)
    if field.dim() != 1 or base.dim() != 2 or base.shape[1] != 3:
        raise RuntimeError('invalid compact IB field/base')
    if phi.dim() != 3 or phi.shape[0] != base.shape[0] or phi.shape[1] != 3 or phi.shape[2] != 4:
        raise RuntimeError('invalid compact IB weights')
    if not (nx > 0 and ny > 0 and nz > 0 and volume > 0):
        raise RuntimeError('invalid compact grid/volume')
    if field.numel() != (base.shape[0] if spread else nx * ny * nz):
        raise RuntimeError('compact IB field length mismatch')
    return field, base, phi


def op_compact_gather(field, base, phi, nx, ny, nz):
    field, base, phi = _compact_checks(field, base, phi, nx, ny, nz, 1., False)
    out = torch.empty(base.shape[0], device=field.device, dtype=field.dtype)
    call('afsi_b200_compact_gather', ptr(field), ptr(base), ptr(phi), base.shape[0], nx, ny, nz, ptr(out),
         ptr(_lib.status_word(field.device)), dtype_code(field.dtype), stream(field.device))
    return out


def op_compact_spread(field, base, phi, nx, ny, nz, volume):
    field, base, phi = _compact_checks(field, base, phi, nx, ny, nz, volume, True)
    out = torch.zeros(nx * ny * nz, device=field.device, dtype=field.dtype)
    call('afsi_b200_compact_spread', ptr(field), ptr(base), ptr(phi), base.shape[0], nx, ny, nz, float(volume),
         ptr(out), ptr(_lib.status_word(field.device)), dtype_code(field.dtype), stream(field.device))
    return out


# ----------------------------------------------------- Python-level wrappers
# afsi_torch/mac/cuda_ib.py:69-90

def indexed_gather(field, indices, weights):
    require_cuda(field)
    return op_indexed_gather(field.contiguous(), indices.contiguous(), weights.contiguous())


def indexed_spread(field, indices, weights, size, volume=1.):
    require_cuda(field)
    return op_indexed_spread(field.contiguous(), indices.contiguous(), weights.contiguous(), size, float(volume))


def _component_tables(grid, values, stencil, like):
    """(base, phi) of a stencil with one contiguous table per component, for
    the one-launch transfers; None for any other (lists, views, other types),
    which takes the per-component operators and their checks."""
    base, phi = stencil.base, stencil.phi
    if not (torch.is_tensor(base) and torch.is_tensor(phi) and base.dim() == 3 and base.shape[0] == 3
            and base.shape[2] == 3 and phi.shape == (*base.shape, 4) and base.dtype == torch.int64
            and phi.dtype == like.dtype and like.dtype in (torch.float32, torch.float64)
            and base.is_contiguous() and phi.is_contiguous()
            and all(t.device == like.device and not t.requires_grad for t in (base, phi, *values))
            and all(grid.face_shape(c) == tuple(n + (a == c) for a, n in enumerate(grid.shape)) for c in range(3))
            and min(grid.shape) > 0):
        return None
    return base, phi


# The binned spread wins where many points share a cell.  What it saves grows with
# the points and with how many share one; what it costs is a fixed 30 us of binning
# and, per cell of the grid, two words that are cleared and scanned.  One B200, points
# per occupied cell from which it is the faster form (a thin shell's cloud in any order,
# both spreads with all their launches and scratch), FP64: 60,000 points 20 on 64^3 and
# 30 on 128^3; 100,000 14 and 20; 200,000 below 12 and 14; 256^3 50 at 200,000, 15 at
# 400,000, 4 at a million; 512^3 none up to a million (60,000: 840 against 490 us and
# 1.1 GB of scratch).  In FP32 the plain form's reductions cost less and the sums on
# chip have no tensor cores: 60,000 points 20 on 32^3, 50 on 64^3 and none on 128^3;
# 100,000 40; 200,000 22 on 64^3, 25 on 128^3, 38 on 192^3; more points 16 to 22 up to
# 192^3; 256^3 none at any.  How many share a cell is sampled once, when the points are
# binned (bin_density_kernel), and read with the support flag; the sample counts by
# points, so a cloud whose cells are unevenly full reads denser than its mean, a thin
# shell by a third.  With the lines below, over 748 clouds of each type, thin and thick,
# 3 to 96 per cell, 60,000 to a million points on 32^3 to 256^3, the form taken is 0.5 %
# (FP64) and 0.7 % (FP32) slower than the faster one on average, where 12 per cell on
# every grid was 2.7 and 10.7 % slower.
_BINNED_POINTS = 60000
# points at which `even` per cell break even: on the smallest grid, more up to 64^3 cells (FP32, where the plain
# form's reductions meet less), and a fiftieth of the cells; even (in proportion to the points), the least per cell,
# the most cells per point, the most cells
_BINNED = {torch.float64: (64000, 0, 16., 9., 96, 1 << 62), torch.float32: (40000, 60000, 32., 22., 40, 1 << 23)}


def _binned_per_cell(points, shape, dtype):
    """Points per occupied cell from which a cloud takes the binned spread, or None."""
    if points < _BINNED_POINTS or dtype not in _BINNED:
        return None
    base, more, even, least, widest, most = _BINNED[dtype]
    cells = prod(shape)
    if cells > min(widest * points, most):
        return None
    return max(least, even * (base + more * min(cells / 64 ** 3, 1.) + cells / 50) / points)


def _binned_bytes(grid, stencil, points, phi):
    """Scratch of the binned spread where it is the faster form, else 0."""
    if (not getattr(stencil, 'dense', False) or phi.data_ptr() % 16
            or _binned_per_cell(points, grid.shape, phi.dtype) is None):
        return 0
    return max(int(_lib.load().afsi_b200_compact_binned_bytes(points, *grid.shape)), 0)


def compact_gather(grid, velocity, stencil):
    require_cuda(velocity[0])
    tables = _component_tables(grid, velocity, stencil, velocity[0]) if len(velocity) == 3 else None
    if tables is not None and all(u.dtype == velocity[0].dtype and u.numel() == prod(grid.face_shape(c))
                                  for c, u in enumerate(velocity)):
        base, phi = tables
        u = [u.contiguous() for u in velocity]
        out = torch.empty((base.shape[1], 3), device=base.device, dtype=phi.dtype)
        call('afsi_b200_compact_gather3', *(ptr(t) for t in u), ptr(base), ptr(phi), base.shape[1], *grid.shape,
             ptr(out), ptr(_lib.status_word(base.device)), dtype_code(phi.dtype), stream(base.device))
        return out
    return torch.stack([op_compact_gather(u.contiguous().view(-1), stencil.base[c].contiguous(),
                                          stencil.phi[c].contiguous(), *grid.face_shape(c))
                        for c, u in enumerate(velocity)], -1)


def compact_spread(grid, force, stencil):
    require_cuda(force)
    tables = _component_tables(grid, (force,), stencil, force)
    if tables is not None and force.shape == (tables[0].shape[1], 3) and grid.volume > 0:
        base, phi = tables
        force = force.contiguous()
        fields = tuple(torch.empty(grid.face_shape(c), device=force.device, dtype=force.dtype) for c in range(3))
        scratch = _binned_bytes(grid, stencil, base.shape[1], phi)
        if scratch > 0:
            work = torch.empty(scratch, device=force.device, dtype=torch.uint8)
            call('afsi_b200_compact_spread3_binned', ptr(force), ptr(base), ptr(phi), base.shape[1], *grid.shape,
                 float(grid.volume), *(ptr(f) for f in fields), ptr(work), scratch,
                 ptr(_lib.status_word(force.device)), dtype_code(force.dtype), stream(force.device))
            return fields
        call('afsi_b200_compact_spread3', ptr(force), ptr(base), ptr(phi), base.shape[1], *grid.shape,
             float(grid.volume), *(ptr(f) for f in fields), ptr(_lib.status_word(force.device)),
             dtype_code(force.dtype), stream(force.device))
        return fields
    return tuple(op_compact_spread(force[:, c].contiguous(), stencil.base[c].contiguous(),
                                   stencil.phi[c].contiguous(), *grid.face_shape(c),
                                   float(grid.volume)).view(grid.face_shape(c)) for c in range(3))


# ------------------------------------------------------------------ binning

@dataclass(frozen=True)
class CompactStencil:
    """base (L,P,3) int64 and phi (L,P,3,4); L=3 component tables
    (``mac/compact_transfer.py:11-18``) or L=2 shared face/centre tables
    (``mac/shared_stencil.py:8-19``)."""
    base: torch.Tensor
    phi: torch.Tensor
    layout: str = 'component'
    dense: bool = False  # many points share a cell: the spread bins them first

    @property
    def storage_bytes(self):
        return self.base.numel() * self.base.element_size() + self.phi.numel() * self.phi.element_size()

    def expanded(self):
        if self.layout != 'shared':
            return self
        base = torch.stack([torch.stack([self.base[int(a != c), :, a] for a in range(3)], -1) for c in range(3)])
        phi = torch.stack([torch.stack([self.phi[int(a != c), :, a, :] for a in range(3)], 1) for c in range(3)])
        return CompactStencil(base, phi, 'component')


_ROWS = 256
_rows, _rows_lock = {}, threading.Lock()


def _own_words(device):
    """Two zeroed int32 words of one call's own, read by the host before the call
    returns: rows of a block per device, each given out once.  The block is cleared
    and waited for when it is made, so its rows serve every stream (a fill per call
    cost 3 us of the 165 that 84,000 points on 32 x 32 x 16 take)."""
    with _rows_lock:
        block, given = _rows.get(device.index, (None, _ROWS))
        if given == _ROWS:
            block, given = torch.zeros((_ROWS, 2), device=device, dtype=torch.int32), 0
            torch.cuda.current_stream(device).synchronize()
        _rows[device.index] = block, given + 1
    return block[given]


def compact_prepare(grid, points, *, layout='component', phi_form='clamped', check_support=True):
    """Binning + weights of ``mac/compact_transfer.py:21-26`` (``from_points``),
    with the support screen of ``compact_transfer.py:94-96`` fused.

    ``phi_form='clamped'`` is the torch kernel (``ib.py:57-67``); ``'radical'``
    the shared radical of the reference CUDA/Triton prepares.  Raises
    ``ValueError`` (after a device sync) when a point's support leaves the grid.
    """
    require_cuda(points)
    points = points.contiguous()
    if points.dim() != 2 or points.shape[1] != 3:
        raise ValueError('points must be (P,3)')
    P = points.shape[0]
    if layout == 'component':
        origins = [grid.face_origin(c) for c in range(3)]
    elif layout == 'shared':
        origins = [grid.origin, tuple(o + .5 * h for o, h in zip(grid.origin, grid.spacing))]
    else:
        raise ValueError('layout must be component or shared')
    L = len(origins)
    base = torch.empty((L, P, 3), device=points.device, dtype=torch.int64)
    phi = torch.empty((L, P, 3, 4), device=points.device, dtype=points.dtype)
    word = _lib.status_word(points.device)
    # a cloud whose density is asked for has two words of its own, the support flag and the answer, read in one copy:
    # the stream's word holds violations only, and other callers raise on any bit of it
    per_cell = _binned_per_cell(P, grid.shape, points.dtype) if check_support and layout == 'component' else None
    ask = per_cell is not None
    if ask:
        own = _own_words(points.device)
    else:
        own = word.zero_() if check_support else word
    call('afsi_b200_compact_prepare', ptr(points), P, L, _lib.doubles(sum(map(list, origins), [])),
         _lib.doubles(grid.spacing), _lib.doubles(grid.origin), _lib.int64s(grid.shape),
         _lib.PHI_RADICAL if phi_form == 'radical' else _lib.PHI_CLAMPED, ptr(base), ptr(phi), ptr(own),
         dtype_code(points.dtype), stream(points.device))
    dense = False
    if ask:
        word.zero_()  # as every checked prepare does; queued behind the kernel, which the host need not wait for
        call('afsi_b200_compact_density', ptr(base), P, per_cell, 1, ptr(own[1:]), stream(points.device))
        flags, dense = own.tolist()
    else:
        flags = int(word.item()) if check_support and P else 0
    if flags & _lib.FLAG_SUPPORT:
        if not ask:
            word.zero_()
        raise ValueError('MAC IB support reaches a wall or is nonfinite; enlarge/refine the fluid box')
    return CompactStencil(base, phi, layout, bool(dense))


@dataclass(frozen=True)
class Stencil2D:
    """Reflected 2D stencils (``mac2d/transfer.py:12-15``): per component ids
    (P,16) int64 and signed weights (P,16)."""
    indices: tuple
    weights: tuple


def prepare2d(grid, points, *, check_support=True):
    """``TriangleTransfer._prepare`` (``mac2d/transfer.py:61-81``) with the
    support screen of ``mac2d/transfer.py:97-101`` fused."""
    require_cuda(points)
    points = points.contiguous()
    if points.dim() != 2 or points.shape[1] != 2:
        raise ValueError('points must be (P,2)')
    P = points.shape[0]
    ids = torch.empty((2, P, 16), device=points.device, dtype=torch.int64)
    w = torch.empty((2, P, 16), device=points.device, dtype=points.dtype)
    word = _lib.status_word(points.device)
    if check_support:
        word.zero_()
    hx, hy = grid.spacing
    call('afsi_b200_indexed_prepare2d', ptr(points), P, grid.shape[0], grid.shape[1], hx, hy,
         grid.lengths[0], grid.lengths[1], ptr(ids), ptr(w), ptr(word), dtype_code(points.dtype),
         stream(points.device))
    if check_support and P and int(word.item()) & _lib.FLAG_SUPPORT:
        word.zero_()
        raise ValueError('valve IB points leave the channel support region')
    return Stencil2D((ids[0], ids[1]), (w[0], w[1]))


def _pair_tables(stencil, like, values):
    """The two components' (ids, weights) when the one-launch 2D transfers take
    them: 16 taps per point, contiguous tables of matching types; else None."""
    if len(stencil.indices) != 2 or len(stencil.weights) != 2 or like.dtype not in (torch.float32, torch.float64):
        return None
    shape = stencil.indices[0].shape
    if len(shape) != 2 or shape[1] != 16:
        return None
    for ids, w in zip(stencil.indices, stencil.weights):
        if not (ids.shape == shape and w.shape == shape and ids.dtype == torch.int64 and w.dtype == like.dtype
                and ids.is_contiguous() and w.is_contiguous() and ids.device == like.device and w.device == like.device
                and not w.requires_grad):
            return None
    if any(t.requires_grad or t.device != like.device or t.dtype != like.dtype for t in values):
        return None
    return (*stencil.indices, *stencil.weights)


def spread2d(grid, force, stencil):
    """``TriangleTransfer._spread`` CUDA branch (``mac2d/transfer.py:108-112``):
    point forces (P,2) -> (u, v) face fields divided by the cell area."""
    sizes = [grid.face_shape(c)[0] * grid.face_shape(c)[1] for c in range(2)]
    if torch.is_tensor(force) and force.is_cuda and force.dim() == 2 and force.shape[1] >= 2:
        tables = _pair_tables(stencil, force, (force,))
        if (tables is not None and tables[0].shape[0] == force.shape[0] and min(sizes) > 0
                and 0 < grid.volume < float('inf')):
            force = force.contiguous()
            u, v = (torch.empty(grid.face_shape(c), device=force.device, dtype=force.dtype) for c in range(2))
            call('afsi_b200_indexed_spread2', ptr(force), force.shape[1], *(ptr(t) for t in tables), force.shape[0],
                 *sizes, float(grid.volume), ptr(u), ptr(v), ptr(_lib.status_word(force.device)),
                 dtype_code(force.dtype), stream(force.device))
            return u, v
    return tuple(indexed_spread(force[:, c:c + 1], stencil.indices[c], stencil.weights[c], sizes[c], grid.volume)
                 .reshape(grid.face_shape(c)) for c in range(2))


def gather2d(velocity, stencil):
    """``TriangleTransfer._gather`` CUDA branch (``mac2d/transfer.py:122-124``)."""
    if len(velocity) == 2 and all(torch.is_tensor(u) and u.is_cuda and u.numel() > 0 for u in velocity):
        tables = _pair_tables(stencil, velocity[0], velocity)
        if tables is not None:
            u, v = (t.contiguous() for t in velocity)
            out = torch.empty((tables[0].shape[0], 2), device=u.device, dtype=u.dtype)
            call('afsi_b200_indexed_gather2', ptr(u), ptr(v), u.numel(), v.numel(), *(ptr(t) for t in tables),
                 out.shape[0], ptr(out), ptr(_lib.status_word(u.device)), dtype_code(u.dtype), stream(u.device))
            return out
    return torch.cat([indexed_gather(u.reshape(-1, 1), ids, w)
                      for u, ids, w in zip(velocity, stencil.indices, stencil.weights)], -1)


def contract(stencil, group, component, offset, low, width, prefix, count, face_shape, workspace, cache=None):
    """``mac/cuda_ib.py:93-106``: P1 box-site contraction into the hash table."""
    from .p1_csr import contract as _contract
    _contract(stencil, group, component, offset, low, width, prefix, count, face_shape, workspace, cache)


def hash_accumulate(keys, values, workspace):
    """``mac/cuda_ib.py:109-112``: insert a (key, value) stream into the table."""
    from .p1_csr import hash_accumulate as _accumulate
    _accumulate(keys, values, workspace)
