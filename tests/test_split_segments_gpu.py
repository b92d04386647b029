"""Recurrences in chunks whose sequences are cut into segments: portions around a segment's end, more heads than the workspace holds at
once, sequences that share tokens, and heads whose values cannot be split."""
import pytest
import torch

from dgi_b200 import mixer_ops
from test_column_scan_gpu import F64, _inputs
from test_split_scan_gpu import _exact, _run

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _chunks(monkeypatch):
    monkeypatch.setattr(mixer_ops, "split_scan_pays", lambda *_: True)


@pytest.mark.parametrize("group", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("segment", [1, 2, 5])
@pytest.mark.parametrize("shape", [(64, 128, 3, [1, 97, 16, 160, 33]), (61, 70, 2, [200, 1, 80])], ids=["64x128", "61x70"])
@pytest.mark.parametrize("rule", ["gated", "retention"])
def test_segments_against_float64(rule, shape, segment, dtype, group, monkeypatch):
    dk, dv, H, lens = shape
    monkeypatch.setattr(mixer_ops, "split_scan_segment", lambda *_: segment)
    if group:       # one head's operands at a time
        monkeypatch.setattr(mixer_ops, "SPLIT_SCAN_WORKSPACE", 1)
    parts, state, consts, seqs, rows = _inputs(dk, dv, H, H, lens, dtype, False)
    want, want_state = _exact(rule, parts, consts, state, rows, H, H)
    got = _run(rule, parts, consts, state, seqs, H, H, max(lens))
    # the bound of the chunks in one piece: a segment's end enters the next by one fp32 product and sum
    for x, y in ((got, want), (state, want_state)):
        assert (x.to(F64) - y).abs().max() <= 1e-5 * y.abs().max() + 1e-7


@pytest.mark.parametrize("where", [0, 1, 2, "state"])
@pytest.mark.parametrize("rule", ["gated", "retention"])
def test_values_that_cannot_be_split(rule, where, monkeypatch):
    """A head with an infinity in its last segment (or its first state) walks token by token from its first on; the others keep their bits."""
    dk, dv, H, lens = 64, 72, 3, [40, 101, 20]
    monkeypatch.setattr(mixer_ops, "split_scan_segment", lambda *_: 2)
    parts, state, consts, seqs, _rows = _inputs(dk, dv, H, H, lens, torch.bfloat16, False)
    clean_state = state.clone()
    clean = _run(rule, parts, consts, clean_state, seqs, H, H, 101)
    if where == "state":
        state[3, 1, 5, 7] = float("inf")           # sequence 0 has slot 3
    else:
        parts[where][40 + 99, 1 * (dk if where < 2 else dv) + 3] = float("inf")
    by_token = state.clone()
    monkeypatch.setattr(mixer_ops, "split_scan_pays", lambda *_: False)
    want = _run(rule, parts, consts, by_token, seqs, H, H, 1)
    monkeypatch.setattr(mixer_ops, "split_scan_pays", lambda *_: True)
    got = _run(rule, parts, consts, state, seqs, H, H, 101)
    assert torch.equal(got.isfinite(), want.isfinite()) and torch.equal(state.isfinite(), by_token.isfinite())
    keep, (first, last) = [0, 2], (0, 40) if where == "state" else (40, 141)
    assert torch.equal(got[:, keep], clean[:, keep])
    assert torch.equal(got[:first], clean[:first]) and torch.equal(got[last:], clean[last:])


@pytest.mark.parametrize("rule", ["gated", "retention"])
def test_sequences_that_share_tokens(rule, monkeypatch):
    """More segments than the tokens have: those beyond the workspace walk token by token."""
    monkeypatch.setattr(mixer_ops, "split_scan_segment", lambda *_: 1)
    dk, dv, H, n = 64, 72, 2, 41
    parts, state, consts, _, _ = _inputs(dk, dv, H, H, [n], torch.bfloat16, False)
    state = state[:1].repeat(6, 1, 1, 1)
    alone = state.clone()
    want = _run(rule, parts, consts, alone, torch.tensor([(0, n, 1, 0)], dtype=torch.int32, device="cuda"), H, H, n)
    seqs = torch.tensor([(0, n, i, 0) for i in range(1, 6)], dtype=torch.int32, device="cuda")
    got = _run(rule, parts, consts, state, seqs, H, H, n)
    assert (got - want).abs().max() <= 2e-5 * want.abs().max() and (state[1:] - alone[1]).abs().max() <= 2e-5 * alone[1].abs().max()
    assert torch.equal(state[0], alone[0])


def test_without_room_for_the_ends(monkeypatch):
    """No memory for the segments' ends: the sequences run in one piece."""
    dk, dv, H, lens = 64, 48, 2, [170, 20]
    parts, state, consts, seqs, _ = _inputs(dk, dv, H, H, lens, torch.bfloat16, False)
    other = state.clone()
    want = _run("gated", parts, consts, state, seqs, H, H, max(lens))
    monkeypatch.setattr(mixer_ops, "split_scan_segment", lambda *_: 2)
    real = torch.empty

    def empty(*size, **kw):
        if kw.get("dtype") == torch.float32 and isinstance(size[0], int):
            raise torch.OutOfMemoryError("no memory")
        return real(*size, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    assert torch.equal(_run("gated", parts, consts, other, seqs, H, H, max(lens)), want) and torch.equal(other, state)
