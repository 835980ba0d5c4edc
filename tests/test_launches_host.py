"""How the library launches its kernels, seen by a CUDA runtime without a GPU
(fake_cudart.cc, CPU): the test program loads it before the library, whose
launches then reach it instead of a device.
"""
import subprocess
import sys
from pathlib import Path
import pytest
from afsi_gpu_b200.build import build, nvcc

HERE = Path(__file__).resolve().parent
PRELUDE = '''
import ctypes, importlib.util, sys, types
sys.modules['torch'] = types.ModuleType('torch')  # torch brings the real runtime along
fake = ctypes.CDLL({fake!r}, ctypes.RTLD_GLOBAL)
spec = importlib.util.spec_from_file_location('binding', {binding!r})
L = importlib.util.module_from_spec(spec)
spec.loader.exec_module(L)
HOOK = ctypes.CFUNCTYPE(None, ctypes.c_char_p, ctypes.c_int, ctypes.c_uint, ctypes.c_size_t,
                        ctypes.POINTER(ctypes.c_void_p))
log = []
hook = HOOK(lambda name, device, blocks, smem, args: log.append((name.decode(), device, blocks, smem, look(name.decode(), args))))
look = lambda name, args: None
L.load()
fake.fake_hook(hook)
ONE, GEO, P = L.doubles([1.] * 3), L.doubles([0.] * 3), 4096  # P: a pointer that nothing reads

def plan(shape, bc, levels, dtype=L.F64):
    p = L.MGPlan(dim=len(shape), bc=bc, levels=levels, smooth=2, dtype=dtype, coarse_dtype=L.F64, coarse_inverse=P,
                 scratch=P)
    for l in range(levels):
        for a in range(3):
            p.level[l].shape[a] = shape[a] >> l if a < len(shape) else 1
            p.level[l].h2[a] = p.level[l].inv_h2[a] = 1.
        p.level[l].p = p.level[l].ping = p.level[l].rhs = P
    return p
'''


@pytest.fixture(scope='module')
def run(tmp_path_factory):
    build()
    fake = tmp_path_factory.mktemp('fake') / 'fake_cudart.so'
    include = Path(nvcc()).resolve().parents[1] / 'include'
    subprocess.run(['g++', '-std=c++17', '-shared', '-fPIC', '-O1', '-I', str(include), '-o', str(fake),
                    str(HERE / 'fake_cudart.cc')], check=True)
    prelude = PRELUDE.format(fake=str(fake), binding=str(HERE.parent / 'afsi_gpu_b200' / '_lib.py'))

    def program(code):
        r = subprocess.run([sys.executable, '-c', prelude + code], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout
    return program


def test_every_kernel_is_configured_on_the_device_that_launches_it(run):
    """Function attributes belong to a device: a process that uses a second one
    gets the same launches there, kernels above the default shared memory too."""
    out = run('''
def everything():
    for npc, nq in ((4, 8), (4, 200), (10, 15), (10, 64)):
        for pos, dt in ((L.F64, L.F64), (L.F64, L.F32), (L.F32, L.F32)):
            for elements in (100, 5000):
                head = (npc, P, 50, P, elements, P, P, nq, P)
                L.call('afsi_b200_fe_fused_spread', *head, P, GEO, ONE, ONE, P, P, P, 32, 32, 32, 1., P, pos, dt, None)
                for f in ('afsi_b200_fe_fused_gather', 'afsi_b200_fe_fused_gather_local'):
                    L.call(f, *head, P, P, P, GEO, ONE, ONE, P, 32, 32, 32, P, pos, dt, None)
                n = L.load().afsi_b200_fe_det_spread_bytes(elements, 32, 32, 32, dt)
                L.call('afsi_b200_fe_det_spread', *head, P, GEO, ONE, ONE, P, P, P, 32, 32, 32, 1., P, n, P, pos, dt, None)
    for dt in (L.F64, L.F32):
        n = L.load().afsi_b200_det_plan_bytes(5000, 32, 32, 32, dt)
        L.call('afsi_b200_det_spread', P, P, P, 5000, 32, 32, 32, P, n, P, P, P, dt, None)
        n = L.load().afsi_b200_compact_binned_bytes(70000, 32, 32, 32)
        L.call('afsi_b200_compact_spread3_binned', P, P, P, 70000, 32, 32, 32, 1., P, P, P, P, n, P, dt, None)
        table = (L.RowsGroup * 1)(L.RowsGroup(P, P, 0, 0, 8))
        L.call('afsi_b200_p1_rows_fill', P, P, 800, table, 1, P, P, 50, P, P, 32, 32, 32, 4000, P, P, P, P, dt, None)
        for shape, bc, levels in (((64, 64, 64), L.BC_NEUMANN, 5), ((64, 64, 64), L.BC_DIRICHLET, 5),
                                  ((256, 64), L.BC_CHANNEL, 5), ((256, 64), L.BC_PERIODIC, 5)):
            p = plan(shape, bc, levels, dt)
            L.call('afsi_b200_mg_vcycles', ctypes.byref(p), 1, None)
            L.call('afsi_b200_mg_persistent', ctypes.byref(p), 1, 0, 1, 0., P, P, None)
            p.smoother = 1
            L.call('afsi_b200_mg_vcycles', ctypes.byref(p), 1, None)
seen = []
for device in (0, 1, 0):
    assert fake.cudaSetDevice(device) == 0
    log.clear()
    everything()
    seen.append([(name, blocks, smem) for name, at, blocks, smem, _ in log if at == device])
    assert len(seen[-1]) == len(log)
assert seen[0] == seen[1] == seen[2]
print(len(seen[0]), max(smem for _, _, smem in seen[0]))
''')
    launches, largest = map(int, out.split())
    assert launches > 100 and largest > 48 * 1024


def test_no_consumer_adds_thousands_of_partials(run):
    """Pending means: every block of a consumer adds all partials of its producer,
    so grids of thousands of blocks must leave one finished sum instead; and what a
    consumer reads is what the producer of that field left."""
    run('''
MOST = 1200  # kPendingMost

class Pending(ctypes.Structure):
    _fields_ = [('part', ctypes.c_void_p), ('count', ctypes.c_int)]

class Site(ctypes.Structure):
    _fields_ = [('partial', ctypes.c_void_p), ('counter', ctypes.c_void_p), ('result', ctypes.c_void_p)]

READS = {'sweep_kernel': (4, 5), 'sweep_columns_kernel': (4,), 'residual_restrict_zpair_kernel': (5,),
         'residual_restrict_kernel': (5,), 'prolong_kernel': (5, 6), 'prolong_octet_kernel': (5, 6),
         'shift_kernel': (3,), 'coarse_kernel': (1,), 'cluster_kernel': (1,)}
LEAVES = {'sweep_kernel': (6, 8), 'sweep_columns_kernel': (5, 8), 'residual_restrict_zpair_kernel': (6, 7),
          'residual_restrict_kernel': (6, 7), 'level_sum_kernel': (2, None)}  # site, flag (none: always)
of = lambda args, i, kind: ctypes.cast(args[i], ctypes.POINTER(kind))[0]

def look(name, args):
    kernel = [k for k in sorted({**READS, **LEAVES}, key=len, reverse=True) if f'{len(k)}{k}I' in name]
    if not kernel:
        return None
    k = kernel[0]
    reads = [(p.part, p.count) for p in (of(args, i, Pending) for i in READS.get(k, ())) if p.part]
    site, mode = None, 0
    if k in LEAVES:
        at, i = LEAVES[k]
        site = of(args, at, Site)
        if i is None or of(args, i, ctypes.c_int):
            mode = 2 if i is None or 'Lb1EE' in name else 1  # the last template argument: finished by the producer
        site = site.partial, site.result
    return k, reads, site, mode

for shape, bc, levels in (((256, 128), L.BC_PERIODIC, 5), ((1024, 512), L.BC_PERIODIC, 7), ((2048, 512), L.BC_PERIODIC, 7),
                          ((4096, 4096), L.BC_PERIODIC, 9), ((64, 64, 64), L.BC_NEUMANN, 5),
                          ((256, 256, 256), L.BC_NEUMANN, 6), ((64, 512, 512), L.BC_NEUMANN, 6),
                          ((128, 1024, 512), L.BC_NEUMANN, 7)):
    for smoother in (0, 1):
        for dt in (L.F64, L.F32):
            p = plan(shape, bc, levels, dt)
            p.smoother = smoother
            log.clear()
            L.call('afsi_b200_mg_vcycles', ctypes.byref(p), 2, None)
            left, read = {}, 0
            for name, device, blocks, smem, seen in log:
                if seen is None:
                    continue
                kernel, reads, site, mode = seen
                for part, count in reads:
                    assert count <= MOST, (shape, kernel, count)
                    assert left[part] == count, (shape, kernel)
                    read += 1
                if mode:
                    left.pop(site[0], None), left.pop(site[1], None)
                    left[site[0 if mode == 1 else 1]] = blocks if mode == 1 else 1
            assert read, shape
''')
