"""Host side of the fused Arnoldi step (CPU)."""
import torch
from afsi_gpu_b200 import stokes_fgmres


def test_the_step_launches_on_the_device_of_its_vectors(monkeypatch):
    """gmres takes vectors of any device, as the torch operations did that the step
    replaced; a launch goes to the current device, which need not be theirs."""
    active, seen = [], []

    class Device:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            active.append(self.device)

        def __exit__(self, *_):
            active.pop()

    V = torch.zeros((4, 10), dtype=torch.float64)
    arnoldi = stokes_fgmres._Arnoldi(V)
    arnoldi.column.zero_()
    monkeypatch.setattr(torch.cuda, 'device', Device)
    monkeypatch.setattr(stokes_fgmres, 'stream', lambda device: 0)
    monkeypatch.setattr(stokes_fgmres, 'call', lambda name, *args: seen.append((name, tuple(active))))
    assert arnoldi.step(1, torch.ones(10, dtype=torch.float64)) == [0.] * 4
    assert seen == [('afsi_b200_krylov_step', (V.device,))] and not active
