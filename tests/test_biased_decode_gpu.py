"""Petipel's attention over few tokens with the keys divided over CTAs at multiples of 256: contexts around the borders, tiles of several
tokens across one, scores far below zero, and rows that do not depend on their neighbours."""
import pytest
import torch

from dgi_b200 import mixer_ops

pytestmark = pytest.mark.gpu

F64 = torch.float64


def _case(H, G, dk, dv, portions, dtype, far=300, level=0.0, page=16):
    """Portions as (new tokens, tokens before) over shuffled pages; ``level``: added to every distance bias."""
    gen = torch.Generator(device="cuda").manual_seed(H * dk + len(portions))
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    need = [(n + past + page - 1) // page for n, past in portions]
    order = torch.randperm(sum(need), generator=gen, device="cuda").to(torch.int32)
    tables = torch.zeros(len(portions), max(need), dtype=torch.int32, device="cuda")
    lo = first = 0
    spans, pos = [], []
    for b, (n, past) in enumerate(portions):
        tables[b, :need[b]] = order[lo:lo + need[b]]
        lo += need[b]
        spans.append((first, n, b, past))
        pos += range(past, past + n)
        first += n
    return dict(q=rnd(first, H * dk).to(dtype), gate=rnd(first, H).to(dtype), k=rnd(sum(need), G, page, dk).to(dtype),
                v=rnd(sum(need), G, page, dv).to(dtype), tables=tables, spans=spans, lut=rnd(H, far) + level, H=H, dv=dv,
                pos=torch.tensor(pos, dtype=torch.int32, device="cuda"))


def _run(c, max_context, rows=None):
    """``rows``: the spans served (all); the others' rows of the result keep 7."""
    spans = c["spans"] if rows is None else [c["spans"][i] for i in rows]
    tiles = torch.tensor([(f, n, b) for f, n, b, _p in spans], dtype=torch.int32, device="cuda")
    out = torch.full((c["q"].shape[0], c["H"] * c["dv"]), 7.0, dtype=c["q"].dtype, device="cuda")
    mixer_ops.biased_prompt_attention(out, c["q"], c["gate"], c["k"], c["v"], c["tables"], tiles, c["pos"], c["lut"], 0.1, 0.2, 16,
                                      c["H"], max_tile_tokens=max(n for _f, n, _b, _p in spans), max_context=max_context)
    return out


def _reference(c):
    H, page = c["H"], c["k"].shape[2]
    G, n_all = c["k"].shape[1], c["q"].shape[0]
    out = torch.empty(n_all, H, c["dv"], dtype=F64, device="cuda")
    for f, n, b, past in c["spans"]:
        j, i = torch.arange(past + n, device="cuda"), torch.arange(past, past + n, device="cuda")[:, None]
        K, V = (p[c["tables"][b, j // page].long(), :, j % page].to(F64) for p in (c["k"], c["v"]))
        temp = 1 + 0.2 * torch.log(((i + 1) // 16 + 1).to(F64))
        for h in range(H):
            s = c["q"][f:f + n].view(n, H, -1)[:, h].to(F64) @ K[:, h // (H // G)].T * 0.1 * temp
            s = s + c["lut"][h].to(F64)[(i - j).clamp(0, c["lut"].shape[1] - 1)]
            out[f:f + n, h] = torch.softmax(s.masked_fill(j > i, float("-inf")), 1) @ V[:, h // (H // G)]
    return (out * torch.sigmoid(c["gate"].to(F64))[..., None]).view(n_all, -1)


def _off(got, want):
    return ((got.to(F64) - want).norm(dim=-1) / want.norm(dim=-1)).max()


CONTEXTS = [(1, 0), (1, 254), (1, 255), (1, 256), (1, 511), (1, 512), (1, 1300)]
ACROSS = [(4, 254), (7, 250), (3, 0), (2, 255), (5, 508), (7, 1020)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("level", [0.0, -130.0, 200.0])
@pytest.mark.parametrize("H,G,dk,dv,portions", [(8, 2, 128, 128, CONTEXTS), (2, 2, 64, 24, CONTEXTS), (2, 2, 128, 128, ACROSS), (3, 3, 32, 48, ACROSS),
                                                (4, 2, 96, 64, ACROSS)])
def test_keys_divided_over_ctas(H, G, dk, dv, portions, level, dtype):
    c = _case(H, G, dk, dv, portions, dtype, level=level)
    most = max(p + n for n, p in portions)
    # weights and result rounded to 8 or 11 bits; scores of about `level` in fp32: 2^-24 of them in each exponent
    tol = 3 * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + abs(level) * 2.0 ** -23
    want = _reference(c)
    got = _run(c, most)
    assert _off(got, want) <= tol and _off(_run(c, 0), want) <= tol
    for i, (n, past) in enumerate(portions):        # alone, with its own bound of contexts: the same to the bit
        f = c["spans"][i][0]
        alone = _run(c, past + n, rows=[i])
        assert torch.equal(alone[f:f + n], got[f:f + n])
        assert (alone[:f] == 7).all() and (alone[f + n:] == 7).all()


@pytest.mark.parametrize("page", [16, 48, 64, 24])       # the last one is not whole tiles of 16
@pytest.mark.parametrize("H,G,dk,dv,portions", [(8, 1, 64, 128, CONTEXTS), (16, 1, 128, 64, CONTEXTS), (4, 2, 64, 64, [(8, 0), (1, 17), (3, 300), (2, 4000)]),
                                                (1, 1, 128, 128, [(1, 0), (16, 250), (9, 1015)])])
def test_page_sizes_row_counts_and_unwritten_rows(H, G, dk, dv, portions, page):
    c = _case(H, G, dk, dv, portions, torch.bfloat16, page=page)
    want = _reference(c)
    for f, n, b, past in c["spans"]:                  # what nobody wrote may hold anything
        j = torch.arange(past + n, -(-(past + n) // page) * page, device="cuda")
        for pool in (c["k"], c["v"]):
            pool[c["tables"][b, j // page].long(), :, j % page] = float("nan")
    most = max(p + n for n, p in portions)
    tol = 3 * 2.0 ** -8                               # weights and result rounded to 8 bits, scores within 2^-20
    assert _off(_run(c, most), want) <= tol and _off(_run(c, 0), want) <= tol


@pytest.mark.parametrize("form", ["expanded", "one_row_transposed", "columns_of_a_wider_one", "wider_than_contexts"])
def test_block_tables_whose_stride_is_not_their_width(form):
    """A table's stride finds its rows and is no bound of its columns."""
    c = _case(8, 2, 128, 128, [(1, 1300)] if form == "one_row_transposed" else CONTEXTS, torch.bfloat16)
    t = c["tables"]
    if form == "expanded":                          # every sequence reads the pages of the longest
        c["tables"] = t[-1:].contiguous().expand(t.shape[0], -1)
    elif form == "one_row_transposed":
        c["tables"] = t[0].contiguous()[:, None].t()
        assert c["tables"].stride() == (1, 1)
    elif form == "columns_of_a_wider_one":
        wide = torch.full((t.shape[0], t.shape[1] + 5), -1, dtype=torch.int32, device="cuda")
        wide[:, 5:] = t
        c["tables"] = wide[:, 5:]
    else:
        c["tables"] = torch.cat([t, torch.full_like(t, -1)], 1)
    most, want = max(p + n for _f, n, _b, p in c["spans"]), _reference(c)
    tol = 3 * 2.0 ** -8                             # as above
    assert _off(_run(c, most), want) <= tol and _off(_run(c, 0), want) <= tol
