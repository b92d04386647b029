"""Prompt attention on tcgen05: pages fetched whole and row by row, with garbage in every row that belongs to no token, and soft caps whose
scores lie within half the cap, beyond it, and on both sides."""
import pytest
import torch

from dgi_b200 import mixer_ops
from test_tile_attention_gpu import F64, GROUPED, LATENT, NARROW, _case, _reference

pytestmark = pytest.mark.gpu
TOL = {torch.bfloat16: 1.5 * 2.0 ** -8, torch.float16: 1.5 * 2.0 ** -11}     # as test_tile_attention


def _bury(pools, st, page):
    """NaN in every row of the pools that no sequence's tokens use."""
    for pool in pools:
        used = torch.zeros(pool.shape[0], page, dtype=torch.bool, device="cuda")
        for _first, n, b, past in st.spans:
            j = torch.arange(past + n, device="cuda")
            used[st.block_tables[b, j // page].long(), j % page] = True
        pool.masked_fill_(~used[:, None, :, None], float("nan"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("page", [8, 16, 24, 64])
@pytest.mark.parametrize("layout,rows,bias", [(GROUPED, 128, 0), (GROUPED, 256, 700), (NARROW, 256, 0), (LATENT, 128, 0)], ids=["rows128", "bias256", "narrow", "latent"])
def test_pages(layout, rows, bias, page, dtype):
    H, G, dk, dv, div = layout
    q, k_pool, v_pool, st, rnd = _case(layout, [(63, 64), (1, 127), (130, 0), (64, 64), (9, 311)], page, dtype)
    _bury((k_pool,) if dv == 0 else (k_pool, v_pool), st, page)
    lut = rnd(H, bias) if bias else None
    out = torch.zeros(q.shape[0], H, dv or 256, dtype=dtype, device="cuda")
    mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, st.prompt_tiles(1, rows // (H // G))[0], st.tok_pos, dk ** -0.5,
                             max_context=st.max_context(), value_width=dv or 256, value_div=div, rows=rows, bias_lut=lut)
    want = _reference(q, k_pool, v_pool, st, dv or 256, div, dk ** -0.5, bias=lut)
    assert (out.to(F64) - want).norm() <= TOL[dtype] * want.norm()


@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("cap", [0.5, 4.0, 9.0, 400.0])
def test_soft_caps(cap, rows):
    H, G, dk, _dv, _div = GROUPED
    q, k_pool, v_pool, st, _ = _case(GROUPED, [(150, 90)], 16, torch.float16)
    out = torch.zeros(q.shape[0], H, dk, dtype=torch.float16, device="cuda")
    mixer_ops.tile_attention(out, q, k_pool, v_pool, st.block_tables, st.prompt_tiles(1, rows // (H // G))[0], st.tok_pos, dk ** -0.5, rows=rows,
                             softcap=cap)
    want = _reference(q, k_pool, v_pool, st, dk, 1, dk ** -0.5, softcap=cap)
    assert (out.to(F64) - want).norm() <= TOL[torch.float16] * want.norm()
