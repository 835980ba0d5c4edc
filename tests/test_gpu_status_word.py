"""The stream's status word holds violations only (B200).

Host threads of one stream share the word, and several of its readers raise on any
bit: the binning of a dense cloud neither sets a bit that is none, nor takes back
what another caller's kernel set meanwhile.  The other caller is played between the
launch of the density question and its reading.
"""
import pytest
import torch
from afsi_gpu_b200 import cuda_ib
from afsi_gpu_b200 import _lib
from afsi_gpu_b200.grid import MACGrid

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _dense():
    g = torch.Generator(device=DEV).manual_seed(2)
    x = .3 + .3 * torch.rand((70000, 3), device=DEV, dtype=torch.float64, generator=g)
    return MACGrid((40, 36, 32), (1., 1., 1.)), x


def _between(monkeypatch, act):
    real = cuda_ib.call

    def call(name, *args):
        rc = real(name, *args)
        if name == 'afsi_b200_compact_density':
            act()
        return rc
    monkeypatch.setattr(cuda_ib, 'call', call)


def test_a_dense_cloud_sets_no_bit_that_others_would_raise(monkeypatch):
    grid, x = _dense()
    seen = []
    _between(monkeypatch, lambda: seen.append(int(_lib.status_word(x.device).item())))
    assert cuda_ib.compact_prepare(grid, x).dense
    assert seen == [0]


def test_a_dense_cloud_keeps_the_flags_of_others(monkeypatch):
    grid, x = _dense()
    word = _lib.status_word(x.device)
    _between(monkeypatch, lambda: word.bitwise_or_(_lib.FLAG_INDEX))
    assert cuda_ib.compact_prepare(grid, x).dense
    with pytest.raises(RuntimeError, match='outside the MAC grid'):
        cuda_ib.check()
    _between(monkeypatch, lambda: word.bitwise_or_(_lib.FLAG_SUPPORT))
    assert cuda_ib.compact_prepare(grid, x).dense  # another's violation is not this cloud's
    word.zero_()
    monkeypatch.undo()
    x[5, 0] = -.1
    with pytest.raises(ValueError, match='support'):
        cuda_ib.compact_prepare(grid, x)
    assert cuda_ib.check() == 0


def test_no_pair_of_words_is_given_out_twice():
    """Rows of used-up blocks are not zeroed again: every call gets a fresh one, on every stream."""
    grid, x = _dense()
    streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    held = [cuda_ib._own_words(x.device) for _ in range(2 * cuda_ib._ROWS)]
    assert len({w.data_ptr() for w in held}) == len(held) and not any(bool(w.any()) for w in held)
    sparse = .1 + .8 * torch.rand((70000, 3), device=DEV, dtype=torch.float64)
    bad = x.clone()
    bad[3, 1] = float('nan')
    torch.cuda.synchronize()
    for k in range(cuda_ib._ROWS + 10):
        with torch.cuda.stream(streams[k % 3]):
            if k % 50 == 7:
                with pytest.raises(ValueError, match='support'):
                    cuda_ib.compact_prepare(grid, bad)
            else:
                assert cuda_ib.compact_prepare(grid, x if k % 2 else sparse).dense == bool(k % 2)
