"""How a packed step's portions are divided between the attention kernels, and what their key splits may allocate (host side only)."""
import pytest
import torch

from dgi_b200 import mixer_ops
from dgi_b200.paged_layer import RaggedBatchState


def _step(portions):
    spans, first = [], 0
    for b, (n, past) in enumerate(portions):
        spans.append((first, n, b, past))
        first += n
    return RaggedBatchState(tok_pos=torch.zeros(first, dtype=torch.int32), slot_mapping=None,
                            block_tables=torch.zeros(len(portions), 1, dtype=torch.int32), scan_seqs=None, spans=spans)


def test_portions_go_to_one_kernel_each_with_their_own_contexts():
    st = _step([(1, 30000), (500, 0), (1, 7), (2000, 100)])
    tiles, rest = st.attention_tiles(16, 4, 128, 16, True)
    assert tiles[2] == 2100 and rest[1:] == (1, 30001)
    served = sorted((f, n) for f, n, _row in tiles[0].tolist() + rest[0].tolist())
    assert served[0][0] == 0 and all(a + n == b for (a, n), (b, _) in zip(served, served[1:])) and sum(n for _f, n in served) == 2502
    assert rest[0].tolist() == [[0, 1, 0], [501, 1, 2]]
    tiles, rest = st.attention_tiles(16, 4, 128, 16, False)
    assert tiles is None and rest[1:] == (16, 30001)
    assert _step([(1, 5)]).attention_tiles(16, 4, 128, 16, True)[0] is None
    assert _step([(64, 5)]).attention_tiles(16, 4, 128, 16, True)[1] is None
    assert _step([]).attention_tiles(16, 4, 128, 16, True) == (None, None)


@pytest.mark.parametrize("H,G,bias,cut", [(16, 4, False, 2), (16, 4, True, 5), (16, 16, False, 8), (16, 16, True, 8), (8, 4, True, 9), (16, 1, True, 2),
                                          (6, 2, False, 2), (6, 2, True, 6)])
def test_short_portions_stay_with_the_16_row_kernels(H, G, bias, cut):
    assert mixer_ops.tile_attention_from(H, G, bias) == cut
    st = _step([(cut - 1, 900), (cut, 900), (1, 40)])
    tiles, rest = st.attention_tiles(H, G, 128, 16, True, bias)
    assert [n for _f, n, _b in tiles[0].tolist()] == [cut] and sorted(n for _f, n, _b in rest[0].tolist()) == sorted([cut - 1, 1])


@pytest.mark.parametrize("H,G,few,many", [(16, 4, 37, 38), (16, 16, 18, 19), (16, 8, 37, 38)])
def test_many_tiny_prompts_stay_with_the_16_row_kernel(H, G, few, many):
    for n, left in ((few, False), (many, True)):
        st = _step([(16, 16)] * n + [(17, 15), (12, 21), (100, 0)])       # one token or key too many, and a prompt
        tiles, rest = st.attention_tiles(H, G, 128, 16, True)
        assert (rest is not None and len(rest[0]) == n and rest[2] == 32) == left
        assert sum(c for _f, c, _b in tiles[0].tolist()) == 129 + (0 if left else 16 * n)
        assert st.attention_tiles(H, G, 128, 16, True, bias=True)[1] is None      # biases: by rows alone


@pytest.mark.parametrize("H,G", [(16, 1), (4, 1), (16, 2), (1, 1)])
def test_layouts_of_few_tiles_take_tiny_prompts_in_tiles(H, G):
    assert mixer_ops.tiny_to_tiles(1000, H, G)


class _Recorder:
    """Stands in for the library: sizes and rules are the real ones, launches are noted and not made."""

    def __init__(self, real):
        self.real, self.calls = real, []

    def __getattr__(self, name):
        if name in ("b200_biased_prompt_attn_ext", "b200_mixed_prompt_attn_ext3", "b200_tile_attn"):
            return lambda *a: self.calls.append(name) or 0
        return getattr(self.real, name)


@pytest.fixture
def workspaces(monkeypatch):
    """Bytes of every fp32 workspace allocated by the ops while no GPU is there."""
    lib, made, empty = _Recorder(mixer_ops._lib_()), [], torch.empty

    def recording(*a, **k):
        t = empty(*a, **{**k, "device": "meta"})
        made.append(t.numel() * t.element_size())
        return t

    monkeypatch.setattr(mixer_ops, "_lib_", lambda: lib)
    monkeypatch.setattr(mixer_ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(mixer_ops, "_stream", lambda: 0)
    monkeypatch.setattr(mixer_ops.torch, "empty", recording)
    return made


def _pools(n_rows, H, G, dk, dtype=torch.bfloat16):
    z = lambda *s, t=dtype: torch.zeros(*s, dtype=t)  # noqa: E731
    return dict(q=z(n_rows, H, dk), out=z(n_rows, H, dk), k=z(1, G, 16, dk), v=z(1, G, 16, dk))


@pytest.mark.parametrize("prompt", [0, 512, 8192])
def test_workspaces_hold_the_tiles_rows_not_the_steps(workspaces, prompt):
    """Two decoded tokens, one behind 32000 tokens, beside a prompt of any length: the prompt's rows and context add nothing."""
    H, G, dk = 16, 4, 128
    st = _step([(1, 32000), (1, 90)] + ([(prompt, 0)] if prompt else []))
    tiles, rest = st.attention_tiles(H, G, dk, 16, True)
    p = _pools(2 + prompt, H, G, dk)
    lut = torch.zeros(H, 8)
    mixer_ops.biased_prompt_attention(p["out"].flatten(1), p["q"].flatten(1), None, p["k"], p["v"], st.block_tables, rest[0], st.tok_pos, lut,
                                      1.0, 0.0, 1, H, max_tile_tokens=rest[1], max_context=rest[2])
    assert workspaces == [126 * 2 * H * (dk + 2) * 4]
    workspaces.clear()
    mixer_ops.mixed_prompt_attention(p["out"], p["q"], p["k"], p["v"], st.block_tables, rest[0], st.tok_pos, 1.0, max_tile_tokens=rest[1],
                                     max_context=rest[2])
    assert len(workspaces) == 1 and workspaces[0] <= 8 * 2 * H * (dk + 2) * 4
    workspaces.clear()
    if prompt:
        mixer_ops.tile_attention(p["out"], p["q"], p["k"], p["v"], st.block_tables, tiles[0], st.tok_pos, 1.0, max_context=tiles[2], rows=tiles[1])
        assert sum(workspaces) <= 16 * 148 * 128 * (dk + 2) * 4      # splits x tiles fill the chip once or twice


def test_a_workspace_beyond_its_bound_is_not_allocated(workspaces):
    """256 sequences, one at 200000 tokens: the keys stay undivided, as before there were splits."""
    H, G, dk, n = 32, 8, 128, 256
    st = _step([(1, 200000)] + [(1, 50)] * (n - 1))
    rest = st.attention_tiles(H, G, dk, 16, True)[1]
    p = _pools(n, H, G, dk)
    mixer_ops.biased_prompt_attention(p["out"].flatten(1), p["q"].flatten(1), None, p["k"], p["v"], st.block_tables, rest[0], st.tok_pos,
                                      torch.zeros(H, 8), 1.0, 0.0, 1, H, max_tile_tokens=rest[1], max_context=rest[2])
    assert workspaces == []


@pytest.mark.parametrize("page,rows", [(8, 128), (16, 128), (64, 128), (24, 256), (7, 256), (128, 256)])
def test_pages_that_come_row_by_row_share_wider_tiles(page, rows):
    """Plain attention: 128 rows where the copy engine fetches whole pages; where it cannot, 256 from three rounds of CTAs on.  Biases and
    caps: 256 from one round on, whatever the pages."""
    assert mixer_ops.tile_rows(16, 4, 128, 8000, page=page) == rows and mixer_ops.tile_rows(16, 4, 128, 7000, page=page) == 128
    assert mixer_ops.tile_rows(16, 4, 128, 2400, heavy=True, page=page) == 256 and mixer_ops.tile_rows(16, 4, 256, 8000, True, page) == 128
    st = _step([(1000, 0)] * 8)
    assert st.attention_tiles(16, 4, 128, 16, True, page=page)[0][1] == rows


@pytest.mark.parametrize("width,ff,most", [(256, 1024, 32), (512, 1408, 32), (512, 2048, 32), (1024, 1408, 32), (1024, 2816, 16), (512, 8192, 16),
                                           (1024, 8192, 16), (2048, 5632, 8), (2048, 8192, 8), (1024, 8224, 0), (4096, 1408, 0)])
def test_how_many_sequences_a_decode_layer_takes_in_one_call(width, ff, most):
    from dgi_b200 import ops
    assert ops.one_call_batch(width, ff) == most
