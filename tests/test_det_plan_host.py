"""The deterministic table spread's plan belongs to its stencil (CPU, launches played).

A time loop prepares into the same buffers, or into memory that the allocator hands
out again: the new stencil has other rows at the old address.
"""
import types
import torch
from afsi_gpu_b200 import p2_cuda_transfer as p2t
from afsi_gpu_b200.grid import MACGrid


def test_every_stencil_gets_a_plan_of_its_own(monkeypatch):
    built = []

    def call(name, base, total, nx, ny, nz, plan, nbytes, *rest):
        built.append((name, base))
    monkeypatch.setattr(p2t, 'call', call)
    monkeypatch.setattr(p2t, 'stream', lambda device: 0)
    monkeypatch.setattr(p2t._lib, 'status_word', lambda device: torch.zeros((), dtype=torch.int32))
    transfer = p2t.P2Transfer.__new__(p2t.P2Transfer)
    transfer.grid = MACGrid((16, 16, 16), (1., 1., 1.))
    base = torch.zeros((2, 40, 3), dtype=torch.int64)
    phi = torch.zeros((2, 40, 3, 4), dtype=torch.float64)
    rule = types.SimpleNamespace(groups=())
    first, second = (p2t.SharedAdaptiveStencil(base, phi, rule) for _ in range(2))
    a = transfer.det_plan(first)
    assert transfer.det_plan(first) is a and len(built) == 1
    b = transfer.det_plan(second)  # the same buffers, prepared again
    assert b is not a and len(built) == 2
    base.add_(1)  # rows changed in place
    assert transfer.det_plan(second) is not b and len(built) == 3
    transfer.grid = MACGrid((16, 16, 24), (1., 1., 1.))
    transfer.det_plan(second)
    assert len(built) == 4 and len(second.plans) == 1
