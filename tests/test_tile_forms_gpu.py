"""The forms of the tile attention kernel that a launch's size and its operands' places choose: one CTA of 128 rows per SM or two, queries by
the copy engine or in pieces (partial tiles, groups of heads that do not divide 128 rows), rows that leave through shared memory or not."""
import pytest
import torch

from dgi_b200 import mixer_ops
from test_tile_attention_gpu import F64, _case, _reference

pytestmark = pytest.mark.gpu

# H, G, key size, value size, value heads per key head
LAYOUTS = {"4x128": (8, 2, 128, 128, 1), "4x64": (8, 2, 64, 64, 1), "6x128": (6, 1, 128, 128, 1), "1x64": (4, 4, 64, 64, 1)}


@pytest.mark.parametrize("out", ["16", "32", "off"], ids=["half", "float", "off_16_bytes"])
@pytest.mark.parametrize("mode", ["plain", "bias", "cap"])
@pytest.mark.parametrize("many", [False, True], ids=["one_per_sm", "two_per_sm"])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_forms(layout, many, mode, out):
    H, G, dk, dv, div = LAYOUTS[layout]
    cap = 128 // (H // G)
    # portions of one, two and a half tiles; with `many`, more CTAs than SMs
    portions = [(cap, 0), (2 * cap, 40), (cap + cap // 2, 100)] + ([(5, 70)] * (160 // G) if many else [])
    q, k_pool, v_pool, st, rnd = _case(LAYOUTS[layout], portions, 16, torch.bfloat16)
    n, scale = q.shape[0], dk ** -0.5
    bias = rnd(H, 150) if mode == "bias" else None
    kw = dict(softcap=4.0) if mode == "cap" else {}
    gate = rnd(n, H * dv if mode == "cap" else H).to(torch.bfloat16)
    wide = torch.full((n, H * dv + 4), 7.0, dtype=torch.float32 if out == "32" else torch.bfloat16, device="cuda")
    o = wide[:, 2:2 + H * dv].unflatten(1, (H, dv)) if out == "off" else torch.empty(n, H, dv, dtype=wide.dtype, device="cuda")
    tiles = st.prompt_tiles(1, cap)[0]
    assert (tiles.shape[0] * G > 148) is many
    mixer_ops.tile_attention(o, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, scale, rows=128, gate=gate, bias_lut=bias, **kw)
    want = _reference(q, k_pool, v_pool, st, dv, div, scale, bias=bias, gate=gate, **kw)
    # weights rounded to 8 bits and one rounding of the result, as in the tests of the options
    tol = 1.5 * 2.0 ** -8
    assert (o.to(F64) - want).norm() / want.norm() <= tol
    assert ((o.to(F64) - want).norm(dim=2) / want.norm(dim=2)).max() <= 8 * tol
    if out == "off":
        assert (wide[:, :2] == 7).all() and (wide[:, 2 + H * dv:] == 7).all()
    again = torch.empty_like(o)
    mixer_ops.tile_attention(again, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, scale, rows=128, gate=gate, bias_lut=bias, **kw)
    assert torch.equal(again, o)


@pytest.mark.parametrize("layout,rows", [("4x128", 128), ("4x128", 256), ("4x64", 128), ("6x128", 128)])
def test_gates_per_channel_come_last(layout, rows):
    """A row with gates per channel is the row without them times the gates: the same products in the same order, fp32, to the bit."""
    H, G, dk, dv, _div = LAYOUTS[layout]
    cap = rows // (H // G)
    q, k_pool, v_pool, st, rnd = _case(LAYOUTS[layout], [(cap, 0), (cap + cap // 3, 100)], 16, torch.bfloat16)
    n = q.shape[0]
    gate = rnd(n, H * dv).to(torch.bfloat16)
    plain, gated = (torch.empty(n, H, dv, dtype=torch.float32, device="cuda") for _ in range(2))
    args = q, k_pool, v_pool, st.block_tables, st.prompt_tiles(1, cap)[0], st.tok_pos, dk ** -0.5
    mixer_ops.tile_attention(plain, *args, rows=rows)
    mixer_ops.tile_attention(gated, *args, rows=rows, gate=gate)
    assert torch.equal(gated, plain * (1.0 / (1.0 + torch.exp(-gate.float()))).view(n, H, dv))


@pytest.mark.parametrize("n", [65535, 65536, 70001])
def test_more_tiles_than_a_grid_has_rows(n):
    """One token per tile: a grid's second dimension ends at 65535, the tiles behind it are another launch's."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    dk, page = 64, 16
    q = torch.randn(n, 1, dk, generator=gen, device="cuda").to(torch.bfloat16)
    pools = torch.randn(2, 3, 1, page, dk, generator=gen, device="cuda").to(torch.bfloat16)
    pos = torch.randint(0, 3 * page, (n,), generator=gen, device="cuda", dtype=torch.int32)
    tables = torch.tensor([[2, 0, 1]], dtype=torch.int32, device="cuda")
    tiles = torch.stack([torch.arange(n, device="cuda"), torch.ones(n, device="cuda", dtype=torch.int64), torch.zeros(n, device="cuda", dtype=torch.int64)], 1).to(torch.int32)
    out = torch.empty_like(q)
    mixer_ops.tile_attention(out, q, pools[0], pools[1], tables, tiles.contiguous(), pos, dk ** -0.5, rows=128)
    K, V = (p[tables[0].long(), 0].reshape(3 * page, dk).to(F64) for p in pools)
    s = (q[:, 0].to(F64) @ K.T * dk ** -0.5).masked_fill(torch.arange(3 * page, device="cuda")[None] > pos[:, None], float("-inf"))
    want = torch.softmax(s, 1) @ V
    assert ((out[:, 0].to(F64) - want).norm(dim=1) / want.norm(dim=1)).max() <= 12 * 2.0 ** -8      # as the rows above


@pytest.mark.parametrize("out", ["16", "32", "off"], ids=["half", "float", "off_16_bytes"])
@pytest.mark.parametrize("mode", ["plain", "bias", "cap"])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_forms_of_256_rows(layout, mode, out):
    """Full tiles, a second half with some rows, with one token and with none, one key tile and many."""
    H, G, dk, dv, div = LAYOUTS[layout]
    rep = H // G
    cap, half = 256 // rep, 128 // rep
    q, k_pool, v_pool, st, rnd = _case(LAYOUTS[layout], [(cap, 0), (2 * cap, 40), (half + half // 2, 100), (half + 1, 300), (half, 70), (half // 2, 0), (1, 9)], 16, torch.bfloat16)
    n, scale = q.shape[0], dk ** -0.5
    bias = rnd(H, 150) if mode == "bias" else None
    kw = dict(softcap=4.0) if mode == "cap" else {}
    gate = rnd(n, H * dv if mode == "cap" else H).to(torch.bfloat16)
    wide = torch.full((n, H * dv + 4), 7.0, dtype=torch.float32 if out == "32" else torch.bfloat16, device="cuda")
    o = wide[:, 2:2 + H * dv].unflatten(1, (H, dv)) if out == "off" else torch.empty(n, H, dv, dtype=wide.dtype, device="cuda")
    mixer_ops.tile_attention(o, q, k_pool, v_pool, st.block_tables, st.prompt_tiles(1, cap)[0], st.tok_pos, scale, rows=256, gate=gate, bias_lut=bias, **kw)
    want = _reference(q, k_pool, v_pool, st, dv, div, scale, bias=bias, gate=gate, **kw)
    tol = 1.5 * 2.0 ** -8       # as above
    assert (o.to(F64) - want).norm() / want.norm() <= tol
    assert ((o.to(F64) - want).norm(dim=2) / want.norm(dim=2)).max() <= 8 * tol
    if out == "off":
        assert (wide[:, :2] == 7).all() and (wide[:, 2 + H * dv:] == 7).all()


@pytest.mark.parametrize("rows", [128, 256])
def test_queries_by_heads(rows):
    """Queries whose heads lie further apart than their tokens: the same bits as side by side."""
    H, G, dk, dv, _div = LAYOUTS["4x128"]
    cap = rows // (H // G)
    q, k_pool, v_pool, st, _rnd = _case(LAYOUTS["4x128"], [(2 * cap, 0), (cap + 3, 50)], 16, torch.bfloat16)
    outs = []
    for x in (q.contiguous(), q.transpose(0, 1).contiguous().transpose(0, 1)):
        outs.append(torch.empty(q.shape[0], H, dv, dtype=torch.bfloat16, device="cuda"))
        mixer_ops.tile_attention(outs[-1], x, k_pool, v_pool, st.block_tables, st.prompt_tiles(1, cap)[0], st.tok_pos, dk ** -0.5, rows=rows)
    assert torch.equal(*outs)
