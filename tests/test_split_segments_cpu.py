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


@pytest.mark.parametrize("rule,heads,portions,waits", [
    # around the lines: by the walk's length, by the tokens beside it, by the heads
    (0, 4, [1000], True), (0, 4, [1300], False), (0, 8, [1000], True), (0, 8, [1150], False), (0, 8, [1000, 1000], False), (0, 16, [760], True), (0, 16, [900], False),
    (0, 4, [843] + [525] * 7, True), (0, 4, [937] + [584] * 7, False), (2, 4, [1500], True), (2, 4, [2000], False), (2, 8, [1150] * 2, True), (2, 8, [1300] * 2, False),
    (2, 16, [1000], True), (2, 16, [1150], False), (2, 16, [1000] * 2, False),
    # shorter ones are not its business
    (0, 4, [752], False), (0, 4, [753], True)])
def test_which_steps_wait_for_the_host(rule, heads, portions, waits):
    assert mixer_ops.split_segments_wait(rule, max(portions), sum(portions), heads) is waits


def test_hardly_fewer_walks_than_multiprocessors_stay_whole():
    assert mixer_ops.split_scan_segment(0, 900, 1800, 2, 16, 128) == 0 and mixer_ops.split_scan_segment(0, 1000, 2000, 2, 16, 128) == 7
