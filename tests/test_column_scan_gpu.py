"""The token-by-token recurrences at the edges of their tiles: key sizes around the register tile's, value sizes that fill no
group of columns, portions around a stage of eight tokens, one and many columns per lane, rows that cannot be moved in words."""
import pytest
import torch

from dgi_b200 import mixer_ops

pytestmark = pytest.mark.gpu

F64 = torch.float64
# (key size, value size, heads, heads of q and k, portions): 40 heads x 128 columns take four columns per lane, the rest fewer
SHAPES = [(64, 128, 40, 40, [9]), (64, 128, 40, 20, [17, 8, 1]), (128, 126, 40, 40, [7]), (30, 130, 40, 40, [8]), (64, 48, 2, 1, [1, 7, 8, 9, 65]),
          (61, 33, 3, 3, [16, 15]), (1, 1, 1, 1, [3]), (129, 17, 2, 2, [20]), (256, 64, 2, 2, [11]), (300, 5, 1, 1, [10, 2])]


def _inputs(dk, dv, H, G, lens, dtype, odd):
    """q | k | v | channel logits | head logits as slices of one tensor whose rows start on odd elements when ``odd``."""
    gen = torch.Generator(device="cuda").manual_seed(dk * 1000 + dv)
    n, sizes = sum(lens), (G * dk, G * dk, H * dv, H * dk, H)
    wide = torch.randn(n, sum(sizes) + (-sum(sizes) % 8) + (9 if odd else 8), generator=gen, device="cuda").to(dtype)
    parts, at = [], 1 if odd else 0
    for s in sizes:
        parts.append(wide[:, at:at + s])
        at += s
    state = torch.randn(len(lens) + 1, H, dk, dv, generator=gen, device="cuda")
    consts = [torch.rand(m, generator=gen, device="cuda").to(dtype) for m in (H * dk, H * dk, H)]
    first, rows = 0, []
    for i, c in enumerate(lens):
        rows.append((first, c, len(lens) - i, i % 2))       # slots in reverse, every second sequence fresh
        first += c
    return parts, state, consts, torch.tensor(rows, dtype=torch.int32, device="cuda"), rows


def _walk(rows, state, step):
    outs, state = [], state.to(F64)
    for first, count, slot, fresh in rows:
        S = torch.zeros_like(state[slot]) if fresh else state[slot]
        for i in range(first, first + count):
            S, o = step(S, i)
            outs.append(o)
        state[slot] = S
    return torch.stack(outs), state


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "-".join(map(str, s[:4])))
@pytest.mark.parametrize("rule", ["gated", "delta", "delta_head", "retention"])
def test_recurrence_edges(rule, shape, dtype, odd):
    dk, dv, H, G, lens = shape
    if rule.startswith("delta") and dk > 256:
        pytest.skip("the delta rule's key sizes end at 256")
    if not rule.startswith("delta"):
        G = H
    (q, k, v, chan, head), state, (c1, c2, c3), seqs, rows = _inputs(dk, dv, H, G, lens, dtype, odd)
    n, before = q.shape[0], state.clone()
    Q, K = (x.to(F64).view(n, G, dk).repeat_interleave(H // G, dim=1) for x in (q, k))
    V = v.to(F64).view(n, H, dv)
    if rule == "gated":
        got = mixer_ops.gated_scan(q, k, v, c1, c2, state, seqs, H, max_count=max(lens))
        Q = Q * torch.sigmoid(Q)
        low = c2.to(F64).view(H, dk)
        f = low + (1 - low) * torch.sigmoid(K + c1.to(F64).view(H, dk))
        step = lambda S, i: (lambda s: (s, (Q[i][:, None] @ s)[:, 0]))(f[i][:, :, None] * S + (1 - f[i])[:, :, None] * V[i][:, None])  # noqa: E731
    elif rule == "retention":
        decay = 1 - torch.rand(H, device="cuda") * 0.2
        got = mixer_ops.retention_scan(q, k, v, decay, 0.3, state, seqs)
        step = lambda S, i: (lambda s: (s, (Q[i][:, None] @ s)[:, 0]))(decay.to(F64)[:, None, None] * S + 0.3 * K[i][:, :, None] * V[i][:, None])  # noqa: E731
    else:
        a, bias = (chan, c1) if rule == "delta" else (head, c1[:H])
        got = mixer_ops.delta_scan(q, k, v, head, a, bias.contiguous(), c3, state, seqs, G, 1e-6, 0.5)
        Q, K = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (Q, K))
        Q = Q * 0.5
        g = torch.exp(-torch.exp(c3.to(F64))[:, None] * torch.nn.functional.softplus(
            (a.to(F64) + bias.to(F64)).view(n, H, -1), threshold=60).expand(n, H, dk))
        beta = torch.sigmoid(head.to(F64))

        def step(S, i):
            S = g[i][:, :, None] * S
            S = S + K[i][:, :, None] * (beta[i][:, None] * (V[i] - (K[i][:, None] @ S)[:, 0]))[:, None]
            return S, (Q[i][:, None] @ S)[:, 0]
    want, want_state = _walk(rows, before, step)
    # fp32 sums of dk products, at most 65 tokens deep: 16 units of 2^-24 per level of a sum of 256 leave 1e-5 of the largest entry
    for x, y in ((got, want), (state, want_state)):
        assert (x.to(F64) - y).abs().max() <= 1e-5 * y.abs().max() + 1e-7


@pytest.mark.parametrize("rule", ["gated", "retention"])
def test_a_sequence_of_nans_stays_its_own(rule):
    gen = torch.Generator(device="cuda").manual_seed(3)
    H, dk, dv, counts = 2, 64, 40, (19, 30, 1)
    n = sum(counts)
    x = torch.randn(n, H * (2 * dk + dv), generator=gen, device="cuda")
    seqs = torch.tensor([(sum(counts[:i]), c, i, 0) for i, c in enumerate(counts)], dtype=torch.int32, device="cuda")
    state = torch.randn(3, H, dk, dv, generator=gen, device="cuda")
    bias, lower, decay = torch.randn(H * dk, generator=gen, device="cuda"), torch.rand(H * dk, device="cuda") * 0.9, torch.tensor([0.9, 0.99], device="cuda")

    def run(rows):
        s = state.clone()
        a, b, v = rows[:, :H * dk], rows[:, H * dk:2 * H * dk], rows[:, 2 * H * dk:]
        o = mixer_ops.gated_scan(a, b, v, bias, lower, s, seqs, H) if rule == "gated" else mixer_ops.retention_scan(a, b, v, decay, 0.1, s, seqs)
        return o, s

    bad = x.clone()
    bad[19 + 11] = float("nan")
    (o, s), (o0, s0) = run(bad), run(x)
    clean = [t for t in range(n) if not 30 <= t < 49]
    assert torch.equal(o[clean], o0[clean]) and torch.equal(s[[0, 2]], s0[[0, 2]])
    assert o[30:49].isnan().all() and s[1].isnan().all()
