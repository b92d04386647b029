"""Prompt attention in tiles of 128 or 256 rows against float64: portions around the tiles' edges, contexts around the key tiles', every mask
and option the layers use, head layouts of each instantiation, page sizes that are no power of two, keys divided over CTAs."""
import pytest
import torch

from dgi_b200 import mixer_ops
from dgi_b200.paged_layer import RaggedBatchState

pytestmark = pytest.mark.gpu

F64 = torch.float64
#           H, G, key size, value size (0: the key rows' first 256 columns), value heads per key head
GROUPED, WIDE, NARROW, ONE, LATENT, LATENT_ROT, PAIRED = ((8, 2, 128, 128, 1), (16, 1, 128, 128, 1), (6, 2, 64, 64, 1), (3, 3, 128, 128, 1),
                                                          (8, 1, 256, 0, 1), (16, 1, 320, 0, 1), (8, 4, 128, 128, 2))
# portions as (new tokens, tokens before)
EDGES = [(32, 0), (33, 31), (31, 64), (64, 1), (65, 200), (130, 0), (1, 5)]


def _case(layout, portions, page, dtype):
    H, G, dk, dv, div = layout
    gen = torch.Generator(device="cuda").manual_seed(H * dk + len(portions))
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    need = [(n + past + page - 1) // page for n, past in portions]
    order = torch.randperm(sum(need) + 3, generator=gen, device="cuda").to(torch.int32)
    tables = torch.zeros(len(portions), max(need) + 1, dtype=torch.int32, device="cuda")
    lo, spans, pos, first = 0, [], [], 0
    for b, (n, past) in enumerate(portions):
        tables[b, :need[b]] = order[lo:lo + need[b]]
        lo += need[b]
        spans.append((first, n, b, past))
        pos += range(past, past + n)
        first += n
    k_pool = rnd(sum(need) + 3, G, page, dk).to(dtype)
    v_pool = k_pool if dv == 0 else rnd(sum(need) + 3, G // div, page, dv).to(dtype)
    q = (rnd(first, H * dk + 16) * 1.5).to(dtype)[:, 8:8 + H * dk].unflatten(1, (H, dk))    # rows of a wider projection
    st = RaggedBatchState(tok_pos=torch.tensor(pos, dtype=torch.int32, device="cuda"), slot_mapping=None, block_tables=tables,
                          scan_seqs=None, spans=spans)
    return q, k_pool, v_pool, st, rnd


def _reference(q, k_pool, v_pool, st, dv, div, scale, sink=None, window=0, keep_first=0, softcap=0.0, chunk=0, gate=None, bias=None, temp=None):
    n_all, H, dk = q.shape
    G, page = k_pool.shape[1], k_pool.shape[2]
    out = torch.empty(n_all, H, dv, dtype=F64, device=q.device)
    for first, n, b, past in st.spans:
        T = past + n
        j, i = torch.arange(T, device=q.device), torch.arange(past, T, device=q.device)[:, None]
        rows = lambda pool: pool[st.block_tables[b, j // page].long(), :, j % page].to(F64)  # noqa: E731
        K, V = rows(k_pool), rows(v_pool)[..., :dv]
        seen = j[None] <= i
        if window:
            seen &= (i - j[None] < window) | (j[None] < keep_first)
        if chunk:
            seen &= i // chunk == j[None] // chunk
        for h in range(H):
            g = h // (H // G)
            s = q[first:first + n, h].to(F64) @ K[:, g].T * scale
            if temp:
                s = s * (1 + temp[0] * torch.log(((i + 1) // temp[1] + 1).to(F64)))
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if bias is not None:
                s = s + bias[h].to(F64)[(i - j[None]).clamp(0, bias.shape[1] - 1)]
            s = s.masked_fill(~seen, float("-inf"))
            m = s.amax(1, keepdim=True) if sink is None else torch.maximum(s.amax(1, keepdim=True), sink[h].to(F64))
            e = torch.exp(s - m)
            out[first:first + n, h] = e @ V[:, g // div] / (e.sum(1, keepdim=True) + (0 if sink is None else torch.exp(sink[h].to(F64) - m)))
    if gate is not None:
        out = out * torch.sigmoid(gate.to(F64)).view(n_all, H, -1)
    return out


OPTIONS = {
    "plain": (GROUPED, {}),
    "window": (GROUPED, dict(window=40)),
    "kept": (GROUPED, dict(window=33, keep_first=5)),
    "cap_sink": (WIDE, dict(window=100, softcap=5.0, sink=True)),
    "gate": (LATENT, dict(gate="head")),
    "gates": (ONE, dict(window=70, gate="channel")),
    "narrow": (NARROW, dict(sink=True)),
    "rotated": (LATENT_ROT, dict(window=64, sink=True)),
    "blocks": (PAIRED, dict(chunk=50, fp32=True)),
    "bias": (GROUPED, dict(bias=90, temp=(0.3, 16), gate="head")),
    "bias_wide": (WIDE, dict(bias=3000, temp=(0.1, 8))),
    "bias_narrow": (NARROW, dict(bias=1)),
}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("portions,page", [(EDGES, 16), (EDGES, 7), ([(40, 900)], 16), ([(300, 0), (17, 300)], 32)], ids=["edges", "page7", "split", "long"])
@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("name", OPTIONS)
def test_tile_attention(name, rows, portions, page, dtype):
    layout, opt = OPTIONS[name]
    H, G, dk, dv, div = layout
    if rows > 128 and dk > 128:
        pytest.skip("wide heads have tiles of 128 rows")
    opt = dict(opt)
    q, k_pool, v_pool, st, rnd = _case(layout, portions, page, dtype)
    n, D, scale = q.shape[0], dv or 256, dk ** -0.5
    kw = {k: opt[k] for k in ("window", "keep_first", "softcap", "chunk") if k in opt}
    if opt.get("sink"):
        kw["sink"] = rnd(H)
    if "gate" in opt:
        kw["gate"] = rnd(n, H if opt["gate"] == "head" else H * D).to(dtype)
    bias = rnd(H, opt["bias"]) if "bias" in opt else None
    extra = dict(bias_lut=bias, temp_coef=opt["temp"][0], temp_every=opt["temp"][1]) if "temp" in opt else dict(bias_lut=bias)
    out = torch.full((n, H, D), 7.0, dtype=torch.float32 if opt.get("fp32") else dtype, device="cuda")
    tiles = st.prompt_tiles(2, rows // (H // G))[0]
    mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, scale, max_context=st.max_context(),
                             value_width=D, value_div=div, rows=rows, **kw, **extra)
    want = _reference(q, k_pool, v_pool, st, D, div, scale, bias=bias, temp=opt.get("temp"), **kw)
    ours = torch.cat([torch.arange(f, f + c) for f, c, _b, _p in st.spans if c > 1]).cuda()
    # weights rounded to 8 (bf16) or 11 bits, summed with random signs: one rounding of the result and a share of one per weight
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.5
    err = (out[ours].to(F64) - want[ours]).norm() / want[ours].norm()
    assert err <= tol, float(err)
    assert (out[ours].to(F64) - want[ours]).abs().max() <= 16 * tol * want[ours].square().mean().sqrt() + 8 * tol * want[ours].abs().max()
    left = [f for f, c, _b, _p in st.spans if c == 1]
    assert all((out[f] == 7.0).all() for f in left)       # rows outside the tiles are another launch's


def test_steep_scores_and_rescaling():
    """Maxima that grow by hundreds from key tile to key tile, and rows whose first visible key tile comes late."""
    q, k_pool, v_pool, st, rnd = _case((8, 2, 128, 128, 1), [(64, 500)], 16, torch.bfloat16)
    st.block_tables[0, :36] = torch.arange(36, dtype=torch.int32, device="cuda")
    k_pool[:36] *= torch.linspace(0.01, 12, 36, device="cuda").to(k_pool.dtype)[:, None, None, None]
    out = torch.empty(64, 8, 128, dtype=torch.bfloat16, device="cuda")
    for window, rows in ((0, 128), (60, 128), (0, 256), (60, 256)):
        tiles = st.prompt_tiles(2, rows // 4)[0]
        mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, 0.5, window=window, rows=rows)
        want = _reference(q, k_pool, v_pool, st, 128, 1, 0.5, window=window)
        assert (out.to(F64) - want).norm() / want.norm() <= 1.5 * 2.0 ** -8


@pytest.mark.parametrize("layout,rows,bias", [(GROUPED, 128, 0), (GROUPED, 256, 0), (GROUPED, 128, 4000), (GROUPED, 256, 4000), (WIDE, 256, 4000),
                                              (ONE, 256, 4000), (NARROW, 256, 4000), (LATENT, 128, 0), (LATENT_ROT, 128, 0)])
def test_walks_of_many_key_tiles(layout, rows, bias):
    """Every buffer, barrier and bias table is reused many times (no key splits); biases change sign and size from distance to distance,
    so that another tile's table shows.  Several calls are the same to the bit."""
    H, G, dk, dv, div = layout
    q, k_pool, v_pool, st, rnd = _case(layout, [(600, 1500), (2 * rows + 5, 1900)], 16, torch.bfloat16)
    lut = rnd(H, bias) * 3 if bias else None
    D, scale = dv or 256, dk ** -0.5
    out = torch.empty(q.shape[0], H, D, dtype=torch.bfloat16, device="cuda")
    tiles = st.prompt_tiles(2, rows // (H // G))[0]
    first = None
    for _ in range(20):
        out.fill_(7.0)
        mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, scale, value_width=D, rows=rows, bias_lut=lut)
        if first is None:
            first = out.clone()
            want = _reference(q, k_pool, v_pool, st, D, div, scale, bias=lut)
            assert (out.to(F64) - want).norm() / want.norm() <= 1.5 * 2.0 ** -8
            rows_err = (out.to(F64) - want).norm(dim=2) / want.norm(dim=2)
            assert rows_err.max() <= 8 * 2.0 ** -8          # a row of wrong biases is off by its own size
        assert torch.equal(out, first)


@pytest.mark.parametrize("layout,spread", [(GROUPED, 4.0), (GROUPED, 10.0), (NARROW, 10.0), (LATENT, 10.0)])
def test_weights_of_steep_rows(layout, spread):
    """fp32 outputs, so that only the weights are rounded (to 8 bits): the largest weight of a row is exact.  In float64 with weights rounded
    that way rows of scores of standard deviation 4 / 10 are 0.0005 / 0.0003 off; with the largest rounded like the others, 0.0013 / 0.0011."""
    H, G, dk, dv, div = layout
    q, k_pool, v_pool, st, rnd = _case(layout, [(64, 1984)], 16, torch.bfloat16)
    D = dv or 256
    q = rnd(64, H, dk).to(torch.bfloat16)
    scale = spread * dk ** -0.5
    out = torch.empty(64, H, D, dtype=torch.float32, device="cuda")
    for rows in (128, 256) if dk <= 128 else (128,):
        tiles = st.prompt_tiles(2, rows // (H // G))[0]
        mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, scale, value_width=D, rows=rows)
        want = _reference(q, k_pool, v_pool, st, D, div, scale)
        # 1.4: a sample of 64 x H rows, and scores summed in fp32
        assert (out.to(F64) - want).norm() / want.norm() <= 1.4 * (5e-4 if spread < 10 else 3.3e-4)


@pytest.mark.parametrize("layout,heads_as_rows", [(GROUPED, False), (WIDE, False), (WIDE, True), (LATENT, False), (PAIRED, False)])
@pytest.mark.parametrize("most", [1, 16])
def test_few_tokens_beside_a_prompt(layout, heads_as_rows, most):
    """The 16-row kernel over part of a step, keys divided over CTAs: its workspace has a place for each of its tiles' rows."""
    H, G, dk, dv, div = layout
    q, k_pool, v_pool, st, _ = _case(layout, [(300, 0), (1, 2500), (150, 40), (1, 17)], 16, torch.bfloat16)
    D, scale = dv or 256, dk ** -0.5
    q = q.contiguous()
    tiles = torch.tensor([(300, 1, 1), (451, 1, 3)], dtype=torch.int32, device="cuda")
    out = torch.full((q.shape[0], H, D), 7.0, dtype=torch.bfloat16, device="cuda")
    mixer_ops.mixed_prompt_attention(out, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, scale, max_context=2501, value_width=D,
                                     value_div=div, heads_as_rows=heads_as_rows, max_tile_tokens=most)
    want = _reference(q, k_pool, v_pool, st, D, div, scale)
    rows = torch.tensor([300, 451], device="cuda")
    assert ((out[rows].to(F64) - want[rows]).norm(dim=(1, 2)) / want[rows].norm(dim=(1, 2))).max() <= 1.5 * 2.0 ** -8
    left = torch.ones(q.shape[0], dtype=torch.bool, device="cuda")
    left[rows] = False
    assert (out[left] == 7).all()


@pytest.mark.parametrize("layout,rows", [(GROUPED, 128), (GROUPED, 256), (LATENT, 128)])
def test_a_query_of_nans_stays_its_own(layout, rows):
    H, G, dk, dv, div = layout
    q, k_pool, v_pool, st, _ = _case(layout, [(70, 300), (40, 0)], 16, torch.bfloat16)
    D = dv or 256
    tiles = st.prompt_tiles(2, rows // (H // G))[0]

    def run(x):
        out = torch.empty(q.shape[0], H, D, dtype=torch.bfloat16, device="cuda")
        mixer_ops.tile_attention(out, x, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, 0.1, value_width=D, rows=rows)
        return out

    bad = q.clone()
    bad[5, 1], bad[80] = float("nan"), float("inf")
    got, want = run(bad), run(q)
    hit = torch.zeros(q.shape[0], H, dtype=torch.bool, device="cuda")
    hit[5, 1], hit[80] = True, True
    assert torch.equal(got[~hit], want[~hit]) and got[hit].isnan().all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bias", [False, True])
def test_a_sequence_alone_in_a_step_and_in_portions(bias, dtype):
    """How the keys are divided, how many rows a tile has and which kernel takes a portion change with the step and the cut: a position's
    result changes by roundings of its weights and of itself, no more; without key splits it is the same to the bit."""
    H, G, dk, dv, _ = GROUPED
    q, k_pool, v_pool, st, rnd = _case(GROUPED, [(200, 400)] + [(90, 0)] * 3, 16, dtype)
    lut = rnd(H, 500) if bias else None

    def run(tokens, max_context, rows=128):      # the first sequence's tokens in portions of these sizes
        out = torch.full((q.shape[0], H, dk), 7.0, dtype=dtype, device="cuda")
        first = 0
        for n in tokens:
            cap = rows // (H // G)
            tiles = torch.tensor([(first + lo, min(cap, n - lo), 0) for lo in range(0, n, cap)], dtype=torch.int32, device="cuda")
            mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, tiles, st.tok_pos, 0.09, rows=rows, bias_lut=lut,
                                     max_context=max_context)
            first += n
        return out[:200]

    whole = run([200], 0)
    assert torch.equal(whole, run([200], 0, 256)) and torch.equal(whole, run([70, 1, 129], 0)) and torch.equal(whole, run([64] * 3 + [8], 0, 256))
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for other in (run([200], 600), run([70, 1, 129], 600), run([33, 167], 600, 256)):
        assert (other.to(F64) - whole.to(F64)).norm() / whole.to(F64).norm() <= 2 * eps
