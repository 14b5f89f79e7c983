"""The spread of a product's time stamps over its blocks, from a launch's buffer."""
import pytest

from dotllm_b200.kernels.microbench import TIMELINE_EVENTS, TIMELINE_SLOTS, TIMELINE_WARPS, timeline_spread


def test_spread_of_two_blocks():
    stamps = [0] * (len(TIMELINE_EVENTS) * TIMELINE_SLOTS)
    for e in range(len(TIMELINE_EVENTS)):
        for b in range(2):
            for w in range(3):
                stamps[e * TIMELINE_SLOTS + b * TIMELINE_WARPS + w] = 1000 + 100 * e + 10 * b + w
    spread = timeline_spread(stamps)
    assert spread["block_start"] == (0, 5, 10) and spread["block_end"] == (500, 505, 510)        # a block's first warp speaks for it
    assert spread["first_chunk_landed"] == (200, 206, 212)


def test_a_launch_without_stamps_says_so():
    with pytest.raises(SystemExit, match="no time stamps"):
        timeline_spread([0] * (len(TIMELINE_EVENTS) * TIMELINE_SLOTS))
