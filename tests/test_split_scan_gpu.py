"""The recurrences in chunks of 16 tokens on the tensor cores: portions around a chunk, key and value sizes that are padded, rows that
cannot be moved in words, heads in groups, and values that cannot be split."""
import pytest
import torch

from dgi_b200 import mixer_ops
from test_column_scan_gpu import F64, _inputs, _walk

pytestmark = pytest.mark.gpu

# (key size, value size, heads, heads of q and k, portions)
SHAPES = [(64, 128, 3, 3, [1, 97, 16, 15]), (64, 130, 4, 2, [100, 17, 2]), (61, 40, 2, 1, [113]), (30, 5, 1, 1, [31, 33, 96]), (1, 72, 2, 2, [99]),
          (64, 64, 2, 2, [112, 1, 1, 48])]


@pytest.fixture(autouse=True)
def _chunks_from_their_first_token_count_on(monkeypatch):
    """These sizes are too small for chunks to be ahead."""
    monkeypatch.setattr(mixer_ops, "split_scan_pays", lambda rule, longest, *_: longest >= mixer_ops.SPLIT_SCAN_FROM[rule])


def _run(rule, parts, consts, state, seqs, H, G, max_count):
    (q, k, v, chan, head), (c1, c2, c3) = parts, consts
    if rule == "gated":
        return mixer_ops.gated_scan(q, k, v, c1, c2, state, seqs, H, max_count=max_count)
    if rule == "retention":
        return mixer_ops.retention_scan(q, k, v, (1 - 0.2 * c3.float()).contiguous(), 0.3, state, seqs, max_count=max_count)
    a, bias = (chan, c1) if rule == "delta" else (head, c1[:H].contiguous())
    return mixer_ops.delta_scan(q, k, v, head, a, bias, c3, state, seqs, G, 1e-6, 0.5, max_count=max_count)


def _exact(rule, parts, consts, state, rows, H, G):
    (q, k, v, chan, head), (c1, c2, c3) = [x.to(F64) for x in parts], [x.to(F64) for x in consts]
    n, dk = q.shape[0], state.shape[2]
    q, k = (x.reshape(n, G, dk).repeat_interleave(H // G, dim=1) for x in (q, k))
    v = v.reshape(n, H, -1)
    beta = torch.ones(n, H, dtype=F64, device="cuda")
    if rule == "gated":
        low = c2.view(H, dk)
        f = low + (1 - low) * torch.sigmoid(k + c1.view(H, dk))
        q, k = q * torch.sigmoid(q), 1 - f
    elif rule == "retention":
        f, k = (1 - 0.2 * c3)[None, :, None].expand(n, H, dk), 0.3 * k
    else:
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        a, bias = (chan, c1) if rule == "delta" else (head, c1[:H])
        f = torch.exp(-torch.exp(c3)[:, None] * torch.nn.functional.softplus((a + bias).view(n, H, -1), threshold=60).expand(n, H, dk))
        q, beta = q * 0.5, torch.sigmoid(head)

    def step(S, i):
        S = f[i][:, :, None] * S
        u = v[i] - (k[i][:, None] @ S)[:, 0] if rule.startswith("delta") else v[i]
        S = S + k[i][:, :, None] * (beta[i][:, None] * u)[:, None]
        return S, (q[i][:, None] @ S)[:, 0]
    return _walk(rows, state, step)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "-".join(map(str, s[:4])))
@pytest.mark.parametrize("rule", ["gated", "delta", "delta_fp16_head", "retention"])
def test_chunks_against_float64(rule, shape, dtype, odd, monkeypatch):
    dk, dv, H, G, lens = shape
    if not rule.startswith("delta"):
        G = H
    if rule == "delta_fp16_head" and dtype == torch.bfloat16:
        pytest.skip("one decay per head in bf16 has a kernel of its own")
    monkeypatch.setattr(mixer_ops, "SPLIT_SCAN_FROM", (1, 1, 1))
    if odd and H > 2:       # one head's operands at a time
        monkeypatch.setattr(mixer_ops, "SPLIT_SCAN_WORKSPACE", 1)
    parts, state, consts, seqs, rows = _inputs(dk, dv, H, G, lens, dtype, odd)
    want, want_state = _exact(rule, parts, consts, state, rows, H, G)
    got = _run(rule, parts, consts, state, seqs, H, G, max(lens))
    # fp32 sums of dk and 16 products per chunk: 16 units of 2^-24 per level leave 1e-5 of the largest entry, as token by token
    for x, y in ((got, want), (state, want_state)):
        assert (x.to(F64) - y).abs().max() <= 1e-5 * y.abs().max() + 1e-7


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e30], ids=["nan", "inf", "large"])
@pytest.mark.parametrize("where", [0, 1, 2, "state"])
@pytest.mark.parametrize("rule", ["gated", "delta", "retention"])
def test_values_that_cannot_be_split(rule, where, value):
    """One such value in q, k, v or the state of one head: the same entries are finite as token by token, other heads and sequences
    keep their bits."""
    dk, dv, H, lens = 64, 72, 3, [40, 101, 20]
    parts, state, consts, seqs, _rows = _inputs(dk, dv, H, H, lens, torch.bfloat16, False)
    clean_state = state.clone()
    clean = _run(rule, parts, consts, clean_state, seqs, H, H, 101)
    if where == "state":
        state[1 + 1, 1, 5, 7] = value       # sequence 1 has slot 2 and is fresh: not read
        state[3, 1, 5, 7] = value           # sequence 0 has slot 3
    else:
        parts[where][40 + 33, 1 * (dk if where < 2 else dv) + 3] = value
    by_token = state.clone()
    want = _run(rule, parts, consts, by_token, seqs, H, H, 1)
    got = _run(rule, parts, consts, state, seqs, H, H, 101)
    assert torch.equal(got.isfinite(), want.isfinite()) and torch.equal(state.isfinite(), by_token.isfinite())
    # A large value stands beside its head's others: sums round in units of the row's (the head's) largest entry.  Decays of up to 28
    # tokens, both sides' with two roundings each (2^-24 x 28 x 2 = 3.3e-6), in a sum of 64 channels whose terms may be 16 times the sum: 5e-5
    for x, y, dims in ((got, want, (2,)), (state, by_token, (2, 3))):
        x, y = (torch.where(t.isfinite(), t, 0.0).to(F64) for t in (x, y))
        assert ((x - y).abs() <= 5e-5 * y.abs().amax(dims, keepdim=True) + 1e-5).all()
    keep = [0, 2]
    first, last = (0, 40) if where == "state" else (40, 141)
    assert torch.equal(got[:, keep], clean[:, keep])
    assert torch.equal(got[:first], clean[:first]) and torch.equal(got[last:], clean[last:])


@pytest.mark.parametrize("rule", ["gated", "delta", "retention"])
def test_sequences_that_share_tokens(rule, monkeypatch):
    """Five states over the same tokens have more chunks than the tokens have: the read-outs and every state are a sequence's alone."""
    monkeypatch.setattr(mixer_ops, "SPLIT_SCAN_FROM", (1, 1, 1))
    dk, dv, H, n = 64, 72, 2, 41
    parts, state, consts, _, _ = _inputs(dk, dv, H, H, [n], torch.bfloat16, False)
    state = state[:1].repeat(6, 1, 1, 1)
    alone = state.clone()
    want = _run(rule, parts, consts, alone, torch.tensor([(0, n, 1, 0)], dtype=torch.int32, device="cuda"), H, H, n)
    seqs = torch.tensor([(0, n, i, 0) for i in range(1, 6)], dtype=torch.int32, device="cuda")
    got = _run(rule, parts, consts, state, seqs, H, H, n)
    # some in chunks, some token by token: fp32 sums of dk and 16 products, as above
    assert (got - want).abs().max() <= 2e-5 * want.abs().max() and (state[1:] - alone[1]).abs().max() <= 2e-5 * alone[1].abs().max()
    assert torch.equal(state[0], alone[0])


@pytest.mark.parametrize("rule", ["gated", "delta", "retention"])
def test_a_hint_beyond_the_step_is_no_portion(rule):
    """160 single tokens without a usable hint walk token by token (in chunks of 16 each would be a chunk): the same bits."""
    parts, state, consts, seqs, _ = _inputs(64, 48, 2, 2, [1] * 160, torch.bfloat16, False)
    other = state.clone()
    want = _run(rule, parts, consts, state, seqs, 2, 2, 1)
    assert torch.equal(_run(rule, parts, consts, other, seqs, 2, 2, 1 << 20), want) and torch.equal(other, state)


@pytest.mark.parametrize("room", [2, 1, 0], ids=["two_heads", "one_head", "none"])
@pytest.mark.parametrize("rule", ["gated", "delta", "retention"])
def test_without_memory_for_the_workspace(rule, room, monkeypatch):
    """Heads in smaller groups keep their bits; without room for one head's operands the scan walks token by token."""
    dk, dv, H, lens = 64, 48, 4, [170, 20]
    parts, state, consts, seqs, _ = _inputs(dk, dv, H, H, lens, torch.bfloat16, False)
    states = [state.clone() for _ in range(2)]
    want = _run(rule, parts, consts, states[0], seqs, H, H, max(lens) if room else 1)
    one = mixer_ops._lib_().b200_split_scan_workspace(1 if rule == "delta" else 0, sum(lens), len(lens), 1)
    real, asked = torch.empty, []

    def empty(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            asked.append(size[0])
            if size[0] > room * one:
                raise torch.OutOfMemoryError("no memory")
        return real(*size, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    got = _run(rule, parts, consts, states[1], seqs, H, H, max(lens))
    assert asked == [h * one for h in ((4, 2, 1) if room < 2 else (4, 2))]
    assert torch.equal(got, want) and torch.equal(states[1], states[0])
