"""How the tile attention divides a walk over the keys: host arithmetic only."""
import pytest
import torch

import dgi_b200  # noqa: F401
from dgi_b200 import _lib


@pytest.mark.parametrize("n_tiles,key_tiles,G,dk,rows,splits", [
    # one CTA per SM, shares of 3 key tiles for few rows, of 8 otherwise
    (1, 17, 4, 128, 128, 5), (8, 17, 4, 128, 128, 4), (8, 16, 4, 128, 128, 4), (32, 16, 4, 128, 128, 1), (37, 40, 2, 64, 128, 2), (38, 16, 2, 64, 128, 1), (38, 40, 2, 64, 128, 3),
    # two per SM where that shortens a walk by more than the merge takes
    (16, 90, 4, 128, 128, 2), (16, 100, 4, 128, 128, 4), (16, 60, 4, 64, 128, 4), (32, 95, 4, 128, 128, 1), (32, 110, 4, 128, 128, 2), (38, 300, 4, 128, 128, 1),
    # forms that have an SM to themselves
    (16, 200, 4, 128, 256, 2), (32, 200, 4, 128, 256, 1), (63, 110, 1, 256, 128, 2), (74, 110, 1, 256, 128, 2), (75, 110, 1, 256, 128, 1),
    (0, 10, 4, 128, 128, 1), (1, 1, 1, 64, 128, 1), (1, 1000, 1, 64, 128, 16)])
def test_shares_of_a_walk(n_tiles, key_tiles, G, dk, rows, splits):
    lib = _lib.load_mixers()
    assert lib.b200_tile_attn_splits(n_tiles, key_tiles, G, dk, rows) == splits
    assert lib.b200_tile_attn_splits_ext(n_tiles, key_tiles, G, dk, rows, n_tiles * rows * G + 100000) == splits


@pytest.mark.parametrize("n_tiles,key_tiles,G,dk,live,splits", [
    # few tokens are soon merged: 20 x 4 behind 3000, 8 x 2 behind 8000, 16 x 8 behind 2000 of 4 heads with keys of their own; 16 x 64 are not
    (20, 47, 4, 128, 320, 3), (8, 126, 4, 128, 64, 9), (16, 32, 4, 128, 512, 4), (16, 33, 4, 128, 4096, 2), (20, 47, 4, 128, 10240, 1)])
def test_shares_of_tiles_that_are_not_full(n_tiles, key_tiles, G, dk, live, splits):
    assert _lib.load_mixers().b200_tile_attn_splits_ext(n_tiles, key_tiles, G, dk, 128, live) == splits


@pytest.mark.skipif(torch.cuda.is_available(), reason="the call must fail before anything is launched")
@pytest.mark.parametrize("dk", [64, 128])
def test_a_failed_register_query_is_reported_and_not_kept(dk):
    """Tiles of 256 rows ask what their kernel was built with: without a device that fails, with the runtime's error and not as a build's fault, and the
    row rule goes on without an answer."""
    lib, at = _lib.load_mixers(), 1 << 20        # an aligned address that nothing reads
    for _ in range(2):
        rc = lib.b200_tile_attn(at, 8 * dk, dk, at, 8 * dk, dk, None, 0, 0, at, 2 * at, at, 4, at, 200, 256, at, None, None, 0, 0.1, 0.0, 0.0, 1, 0, 0, 0, 8, 2,
                                dk, dk, dk, 1, 0, 16, 1, None, 2, None)
        assert rc > 0 and b"registers" not in lib.b200_mixers_last_error()
    assert lib.b200_tile_attn_rows_ext(4, 4, dk, 20000, 1) == 256
