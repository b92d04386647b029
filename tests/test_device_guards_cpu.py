"""Launches that follow their tensors' device and refuse what does not fit, without a GPU: the library is a recorder."""
import types

import pytest
import torch

from dgi_b200 import _lib, mixer_ops, ops


@pytest.fixture
def recorded(monkeypatch):
    """``[(device of the guard, entry name)]`` of the launches made."""
    made, inside = [], []

    class Guard:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            inside.append(self.device)

        def __exit__(self, *exc):
            inside.pop()

    class Library:
        def __getattr__(self, name):
            return lambda *a: made.append((inside[-1] if inside else None, name)) or 0

    monkeypatch.setattr(torch.cuda, "device", Guard)
    monkeypatch.setattr(mixer_ops, "_lib_", Library)
    monkeypatch.setattr(ops, "_lib", types.SimpleNamespace(load=Library, check=_lib.check, B200LibraryError=_lib.B200LibraryError))
    for m in (mixer_ops, ops):
        monkeypatch.setattr(m, "_need_cuda", lambda *a: None)
        monkeypatch.setattr(m, "_stream", lambda: 0)
    return made


def test_zeroed_blocks_follow_their_pools(recorded):
    pools = [torch.ones(4, 2, 8), torch.ones(3, 16)]
    mixer_ops.zero_blocks(pools, [0, 2])
    assert recorded == [(torch.device("cpu"), "b200_zero_blocks")]
    mixer_ops.zero_blocks([], [0])
    mixer_ops.zero_blocks(pools, [])
    for bad, slots, error in ((pools, [3], IndexError), (pools, [-1], IndexError), ([pools[0], pools[1].t()], [0], ValueError),
                              ([pools[0], torch.ones(4, 8, device="meta")], [0], ValueError)):
        with pytest.raises(error):
            mixer_ops.zero_blocks(bad, slots)
    assert len(recorded) == 1


def test_zeroed_blocks_are_on_a_gpu():
    with pytest.raises(_lib.B200LibraryError):
        mixer_ops.zero_blocks([torch.ones(4, 2, 8)], [0])


def test_rope_tables_follow_their_positions(recorded):
    pos, freqs = torch.zeros(2, 3, dtype=torch.int64), torch.ones(4)
    cos, sin = ops.rope_tables(pos, freqs, torch.bfloat16, 1.0)
    assert cos.shape == sin.shape == (2, 3, 8) and recorded == [(torch.device("cpu"), "b200_rope_tables")]
    for bad in (freqs.view(2, 2), freqs.double(), torch.ones(4, device="meta")):
        with pytest.raises(ValueError):
            ops.rope_tables(pos, bad, torch.bfloat16, 1.0)
