"""A Llama layer's decode step in one call: batches around the tiles of eight sequences, both head sizes, contractions that fill no round of
the warps, RoPE tables given or made, divided contexts; and who is left to the separate launches."""
import math

import pytest
import torch

from dgi_b200 import ops
from dgi_b200.paged_layer import PagedBatchState, PagedLayerKV, PagedLlamaDecoderLayer, rope_tables
from dgi_b200.testing import LlamaShapeConfig

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _case(W, heads, kv, ff, B, dtype, seed=0, context=70, head_dim=None):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    cfg = LlamaShapeConfig(hidden_size=W, num_attention_heads=heads, num_key_value_heads=kv, intermediate_size=ff, vocab_size=64, num_hidden_layers=1,
                           head_dim=head_dim)
    layer = PagedLlamaDecoderLayer(cfg, 0, "cuda", dtype)
    D = layer.head_dim
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn(p.shape, generator=gen, device="cuda") * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (p.dim() == 1))
    lens = [1 + (context * (b + 3) * 7) % context for b in range(B)]
    need = [(n + 15) // 16 for n in lens]
    order = torch.randperm(sum(need), generator=gen, device="cuda").to(torch.int32)
    tables = torch.zeros(B, max(need), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = order[at:at + n]
        at += n
    k, v = (torch.randn(sum(need), kv, 16, D, generator=gen, device="cuda").to(dtype) for _ in range(2))
    x = torch.randn(B, 1, W, generator=gen, device="cuda").to(dtype)
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    pos = (ctx.to(torch.int64) - 1)[:, None].contiguous()
    slots = tables.gather(1, (pos // 16)).squeeze(1).to(torch.int64) * 16 + pos.squeeze(1) % 16
    return layer, x, pos, k, v, PagedBatchState(block_tables=tables, context_lens=ctx, slot_mapping=slots, max_context_len=max(lens)), lens


def _exact(layer, x, pos, k, v, st, lens):
    H, G, D = layer.num_heads, layer.num_kv_heads, layer.head_dim
    w = {n: p.detach().to(F64) for n, p in layer.named_parameters()}
    x, k, v = x[:, 0].to(F64), k.to(F64).clone(), v.to(F64).clone()

    def norm(a, g):
        return a / torch.sqrt((a * a).mean(-1, keepdim=True) + layer.eps) * g

    def turn(a, p):
        ang = p.to(F64)[:, None, None] * torch.cat([layer.inv_freq.to(F64)] * 2)
        half = torch.cat([-a[..., D // 2:], a[..., :D // 2]], -1)
        return a * ang.cos() + half * ang.sin()
    y = norm(x, w["input_layernorm.weight"])
    B = x.shape[0]
    q = turn((y @ w["self_attn.q_proj.weight"].T).view(B, H, D), pos[:, 0])
    kn = turn((y @ w["self_attn.k_proj.weight"].T).view(B, G, D), pos[:, 0])
    vn = (y @ w["self_attn.v_proj.weight"].T).view(B, G, D)
    att = torch.empty(B, H * D, dtype=F64, device="cuda")
    for b, n in enumerate(lens):
        blk, off = st.block_tables[b, (n - 1) // 16].long(), (n - 1) % 16
        k[blk, :, off], v[blk, :, off] = kn[b], vn[b]
        t = st.block_tables[b, :(n + 15) // 16].long()
        kk, vv = (p[t].transpose(1, 2).reshape(-1, G, D)[:n].repeat_interleave(H // G, dim=1) for p in (k, v))
        s = torch.einsum("hd,nhd->hn", q[b], kk) / math.sqrt(D)
        att[b] = torch.einsum("hn,nhd->hd", s.softmax(-1), vv).reshape(-1)
    h = x + att @ w["self_attn.o_proj.weight"].T
    y = norm(h, w["post_attention_layernorm.weight"])
    act = torch.nn.functional.silu(y @ w["mlp.gate_proj.weight"].T) * (y @ w["mlp.up_proj.weight"].T)
    return h + act @ w["mlp.down_proj.weight"].T, k, v


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("W,heads,kv,ff,B,context", [(256, 4, 1, 704, 1, 30), (512, 8, 2, 1408, 8, 300), (512, 4, 4, 96, 9, 17), (128, 2, 2, 32, 17, 5),
                                                     (1024, 8, 1, 1408, 32, 90), (2048, 16, 4, 4096, 3, 4000), (64, 1, 1, 160, 16, 33)])
def test_layer_against_float64(W, heads, kv, ff, B, context, given, dtype, monkeypatch):
    layer, x, pos, k, v, st, lens = _case(W, heads, kv, ff, B, dtype, context=context)
    want, want_k, want_v = _exact(layer, x, pos, k, v, st, lens)
    if given:
        st.cos, st.sin = rope_tables(pos, layer.inv_freq, dtype)
    calls = []
    real = ops.llama_decode_layer
    monkeypatch.setattr(ops, "llama_decode_layer", lambda *a, **kw: calls.append(1) or real(*a, **kw))
    with torch.no_grad():
        got, _ = layer(x, position_ids=pos, past_key_value=PagedLayerKV(k, v, st))
    assert calls and got.shape == x.shape
    # eight roundings to the storage type in a row (unit 2^-9 / 2^-12 each), of parts as large as the result
    unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    for a, b in ((got[:, 0], want), (k, want_k), (v, want_v)):
        assert (a.to(F64) - b).norm() <= 3 * unit * b.norm()


def test_who_keeps_the_separate_launches(monkeypatch):
    layer, x, pos, k, v, st, _lens = _case(256, 4, 2, 704, 4, torch.bfloat16)
    calls = []
    real = ops.llama_decode_layer
    monkeypatch.setattr(ops, "llama_decode_layer", lambda *a, **kw: calls.append(1) or real(*a, **kw))

    def run(grad=False):
        with torch.set_grad_enabled(grad):
            return layer(x, position_ids=pos, past_key_value=PagedLayerKV(k.clone(), v.clone(), st))[0]
    one = run()
    assert len(calls) == 1
    seen = []
    hook = layer.mlp.down_proj.register_forward_hook(lambda m, a, o: seen.append(1))
    many = run()
    hook.remove()
    assert seen and len(calls) == 1
    assert (many.float() - one.float()).norm() <= 2.0 ** -7 * one.float().norm()      # two paths, each within 3 x 2^-9 of float64
    assert run(grad=True).requires_grad and len(calls) == 1
    layer.mlp.up_proj = torch.nn.utils.parametrizations.weight_norm(layer.mlp.up_proj)
    run()
    layer.mlp.up_proj = torch.nn.Linear(256, 704, bias=True, device="cuda", dtype=torch.bfloat16)
    run()
    assert len(calls) == 1


class _Callable(torch.nn.Module):
    """What a projection's place needs: a forward, no weight."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, x):
        return self.inner(x)


@pytest.mark.parametrize("group,name", PagedLlamaDecoderLayer._LINEARS)
def test_a_projection_need_only_be_callable(group, name, monkeypatch):
    layer, x, pos, k, v, st, lens = _case(256, 4, 2, 704, 4, torch.bfloat16)
    want, _, _ = _exact(layer, x, pos, k, v, st, lens)
    monkeypatch.setattr(ops, "llama_decode_layer", lambda *a, **kw: pytest.fail("a wrapped projection was passed by"))
    setattr(getattr(layer, group), name, _Callable(getattr(getattr(layer, group), name)))
    with torch.no_grad():
        got, _ = layer(x, position_ids=pos, past_key_value=PagedLayerKV(k, v, st))
    assert (got[:, 0].to(F64) - want).norm() <= 3 * 2.0 ** -9 * want.norm()      # as above


@pytest.mark.parametrize("W,heads,ff,B,head_dim", [(256, 2, 688, 4, None), (512, 4, 1000, 1, None), (128, 2, 344, 9, None), (144, 2, 704, 3, 64),
                                                   (256, 4, 8, 32, None)])
def test_sizes_that_are_no_multiples_of_32_keep_the_separate_launches(W, heads, ff, B, head_dim, monkeypatch):
    layer, x, pos, k, v, st, lens = _case(W, heads, heads // 2, ff, B, torch.bfloat16, head_dim=head_dim)
    want, want_k, want_v = _exact(layer, x, pos, k, v, st, lens)
    monkeypatch.setattr(ops, "llama_decode_layer", lambda *a, **kw: pytest.fail("these sizes are not served"))
    with torch.no_grad():
        got, _ = layer(x, position_ids=pos, past_key_value=PagedLayerKV(k, v, st))
    for a, b in ((got[:, 0], want), (k, want_k), (v, want_v)):
        assert (a.to(F64) - b).norm() <= 3 * 2.0 ** -9 * b.norm()                # as above
