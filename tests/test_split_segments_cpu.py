"""Which steps of the recurrences cut their sequences into segments: host arithmetic only."""
import pytest

import dgi_b200  # noqa: F401
from dgi_b200 import mixer_ops


@pytest.mark.parametrize("rule,heads,portions,dv,segment", [
    # (rule, heads, portions, value size, chunks per segment)
    (0, 4, [2048], 128, 4), (2, 4, [2048] * 8, 128, 10), (0, 8, [2048] * 8, 128, 0), (0, 16, [1780] + [1000] * 5, 128, 0), (2, 16, [1000] * 2, 128, 7),
    (1, 4, [2048], 128, 0), (0, 8, [700] * 6, 128, 0), (0, 16, [8192], 128, 17), (0, 32, [2048], 64, 7), (0, 4, [752], 128, 0), (0, 4, [753], 128, 4)])
def test_which_walks_are_cut_into_segments(rule, heads, portions, dv, segment):
    assert mixer_ops.split_scan_segment(rule, max(portions), sum(portions), len(portions), heads, dv) == segment
