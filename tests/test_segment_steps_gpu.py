"""Recurrences whose sequences the dispatch itself cuts into segments: long portions alone and beside short ones, decays near one, whose state is
the segments' ends, and the mixers around them."""
import math

import pytest
import torch

from dgi_b200 import mixer_ops
from dgi_b200.fibirax_layer import ParallelMixer
from dgi_b200.paged_layer import RaggedBatchState, RaggedLayerCache
from dgi_b200.petipel_layer import GatedLinearRecurrence
from oracle import fibirax_ref
from test_fibirax_gpu import left, right

pytestmark = pytest.mark.gpu

F64, DEV, DK, DV = torch.float64, "cuda", 64, 128


@pytest.fixture
def cuts(monkeypatch):
    """Chunks per segment of every scan that follows (0: in one piece)."""
    seen, segment, wait = [], mixer_ops.split_scan_segment, mixer_ops.split_segments_wait

    def note(*a):
        seen.append(segment(*a))
        return seen[-1]

    def or_wait(*a):
        if wait(*a):
            seen[-1] = 0
        return wait(*a)

    monkeypatch.setattr(mixer_ops, "split_scan_segment", note)
    monkeypatch.setattr(mixer_ops, "split_segments_wait", or_wait)
    return seen


def _steps(rows, f, k, v, q, state):
    """Token by token in 64 bits: S <- f S + k v^T, o = S^T q."""
    out, state = torch.empty(v.shape, dtype=F64, device=DEV), state.to(F64)
    for first, count, slot, fresh in rows:
        S = torch.zeros_like(state[slot]) if fresh else state[slot]
        for i in range(first, first + count):
            S = f[i][:, :, None] * S + k[i][:, :, None] * v[i][:, None]
            out[i] = torch.einsum("hkv,hk->hv", S, q[i])
        state[slot] = S
    return out, state


def _rows(lens):
    """Slots in reverse; the first sequence goes on from a state, every second one starts."""
    return [(sum(lens[:i]), n, len(lens) - i, i % 2) for i, n in enumerate(lens)]


def _close(got, want):
    # fp32 sums of 64 keys and 16 tokens per chunk, as in one piece; a segment's end enters the next by one product and sum
    assert (got.to(F64) - want).abs().max() <= 1e-5 * want.abs().max() + 1e-7


@pytest.mark.parametrize("slow", [False, True], ids=["decays", "near_one"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rule,H,lens", [("gated", 4, [1300]), ("gated", 4, [2048, 40, 1]), ("gated", 8, [1153, 1000]), ("gated", 16, [900]),
                                         ("retention", 4, [2047]), ("retention", 8, [1300, 17, 1301]), ("retention", 16, [1150])])
def test_long_walks_against_float64(rule, H, lens, dtype, slow, cuts):
    gen = torch.Generator(device=DEV).manual_seed(H + len(lens))
    n, rows = sum(lens), _rows(lens)
    wide = torch.randn(n, H * (2 * DK + DV) + 8, generator=gen, device=DEV).to(dtype)
    a, b, v = wide[:, :H * DK], wide[:, H * DK:2 * H * DK], wide[:, 2 * H * DK:H * (2 * DK + DV)]
    state = torch.randn(len(lens) + 1, H, DK, DV, generator=gen, device=DEV)
    before, seqs = state.clone(), torch.tensor(rows, dtype=torch.int32, device=DEV)
    Q, B, V = a.to(F64).view(n, H, DK), b.to(F64).view(n, H, DK), v.to(F64).reshape(n, H, DV)
    if rule == "gated":
        bias, low = torch.randn(H * DK, generator=gen, device=DEV).to(dtype), torch.rand(H * DK, generator=gen, device=DEV)
        low = (0.98 + 0.015 * low if slow else low).to(dtype)
        got = mixer_ops.gated_scan(a, b, v, bias, low, state, seqs, H, max_count=max(lens))
        lo = low.to(F64).view(H, DK)
        f = lo + (1 - lo) * torch.sigmoid(B + bias.to(F64).view(H, DK))
        want, want_state = _steps(rows, f, 1 - f, V, Q * torch.sigmoid(Q), before)
    else:
        decay = 1 - torch.rand(H, generator=gen, device=DEV) * (0.002 if slow else 0.2)
        got = mixer_ops.retention_scan(a, b, v, decay, 0.125, state, seqs, max_count=max(lens))
        want, want_state = _steps(rows, decay.to(F64)[None, :, None].expand(n, H, DK), 0.125 * B, V, Q, before)
    assert cuts[-1] > 0
    _close(got, want)
    _close(state, want_state)


def _state_of(rows, lens, past):
    spans = [(first, n, b, 0 if fresh else past) for b, (first, n, _slot, fresh) in enumerate(rows)]
    pos = torch.cat([torch.arange(p, p + n) for _f, n, _b, p in spans])
    row = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens))
    pages = (past + max(lens) + 15) // 16
    tables = torch.randperm(len(lens) * pages, generator=torch.Generator().manual_seed(1)).view(len(lens), pages)
    slots = tables[row, pos // 16] * 16 + pos % 16
    return RaggedBatchState(tok_pos=pos.to(torch.int32).to(DEV), slot_mapping=slots.to(DEV), block_tables=tables.to(torch.int32).to(DEV),
                            scan_seqs=torch.tensor(rows, dtype=torch.int32).to(DEV), spans=spans, tok_row=row.to(torch.int32).to(DEV), scan_host=rows)


@pytest.mark.parametrize("H,lens", [(4, [1301]), (8, [1153, 1000])])
def test_a_gated_mixer(H, lens, cuts):
    gen = torch.Generator(device=DEV).manual_seed(H)
    rnd = lambda *s, by=1.0: (torch.randn(*s, generator=gen, device=DEV) * by).to(torch.bfloat16)  # noqa: E731
    W, n, rows = 128, sum(lens), _rows(lens)
    t = dict(q=rnd(H * DK, W, by=W ** -0.5), f=rnd(H * DK, W, by=W ** -0.5), v=rnd(H * DV, W, by=W ** -0.5), norm=rnd(DV), o=rnd(W, H * DV, by=(H * DV) ** -0.5))
    t["f.b"], t["lower"] = rnd(H * DK), torch.rand(H * DK, generator=gen, device=DEV).to(torch.bfloat16)
    mixer = GatedLinearRecurrence(dict(heads=H, dim=DK, vdim=DV), t, 1e-6, DEV, torch.bfloat16)
    state = torch.randn(len(lens) + 1, H, DK, DV, generator=gen, device=DEV)
    before, h = state.clone(), rnd(n, W)
    with torch.no_grad():
        got = mixer(h, RaggedLayerCache(None, None, state, _state_of(rows, lens, 30)))
        proj = torch.nn.functional.linear(h, mixer.w_in).to(F64)          # what the recurrence reads, rounded as the mixer rounds it
    assert cuts[-1] > 0
    q, f, v = (x.reshape(n, H, -1) for x in proj.split([H * DK, H * DK, H * DV], dim=1))
    low = t["lower"].to(F64).view(H, DK)
    f = low + (1 - low) * torch.sigmoid(f + t["f.b"].to(F64).view(H, DK))
    o, want_state = _steps(rows, f, 1 - f, v, q * torch.sigmoid(q), before)
    _close(state, want_state)
    want = (o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-6) * t["norm"].to(F64)).view(n, H * DV) @ t["o"].to(F64).T
    assert (got.to(F64) - want).norm() <= 1.5 * 2.0 ** -8 * want.norm()      # two roundings to 8 bits


def test_attention_beside_retention(cuts):
    """One fresh portion, beyond the line from which such a step is cut: both mixers against their statements, the state against 64 bits."""
    gen = torch.Generator().manual_seed(7)
    rnd = lambda *s, by=1.0: (torch.randn(*s, generator=gen) * by).to(torch.bfloat16)  # noqa: E731
    H, W, n = 4, 128, 2001
    spec = dict(left=left(4, 2, 64, 64, 100, 16), right=right(H, DK, DV, [0.9, 0.99, 0.999, 0.5]), left_scale=1.0, right_scale=1.0)
    t = {"left.q": rnd(4 * 64, W, by=W ** -0.5), "left.k": rnd(2 * 64, W, by=W ** -0.5), "left.v": rnd(2 * 64, W, by=W ** -0.5), "left.o": rnd(W, 4 * 64, by=1 / 16),
         "right.q": rnd(H * DK, W, by=W ** -0.5), "right.k": rnd(H * DK, W, by=W ** -0.5), "right.v": rnd(H * DV, W, by=W ** -0.5),
         "right.g": rnd(H * DV, W, by=W ** -0.5), "right.o": rnd(W, H * DV, by=(H * DV) ** -0.5)}
    mixer = ParallelMixer(spec, t, 1e-6, DEV, torch.bfloat16)
    rows, h = [(0, n, 0, 1)], rnd(n, W)
    st = _state_of(rows, [n], 0)
    pools = [torch.zeros(st.block_tables.numel(), 2, 16, 64, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    state = torch.randn(1, H, DK, DV, generator=gen).to(DEV)
    with torch.no_grad():
        got = mixer(h.to(DEV), RaggedLayerCache(*pools, state, st))
        proj = torch.nn.functional.linear(h.to(DEV), mixer.w_in).to(F64)
    assert cuts[-1] > 0
    q, k, v = (proj[:, mixer.cuts[i]:mixer.cuts[i] + w].reshape(n, H, -1) for i, w in ((3, H * DK), (4, H * DK), (5, H * DV)))
    decay = mixer.decay.to(F64)[None, :, None].expand(n, H, DK)
    o, want_state = _steps(rows, decay, k * DK ** -0.5, v, q, torch.zeros_like(state))
    _close(state, want_state)
    parts = {s: {key[len(s) + 1:]: x.to(F64) for key, x in t.items() if key.startswith(s)} for s in ("left", "right")}
    gate = h.to(F64) @ parts["right"]["g"].T
    normed = (o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-6)).view(n, H * DV).cpu()
    want = fibirax_ref.window_sink_attention(h.to(F64), spec["left"], parts["left"], 1e-6) + (normed * gate * torch.sigmoid(gate)) @ parts["right"]["o"].T
    # projections, q / k rows, weights, gated rows and the result are each rounded to 8 bits
    assert (got.cpu().to(F64) - want).norm() <= math.sqrt(5) * 2.0 ** -8 * want.norm()
