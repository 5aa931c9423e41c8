"""When a step's delta rule runs in blocks of tokens (calm_b200_seq_delta_blocks_pay): measured steps on both sides of the line, a long portion among many short ones among them."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

from calm_b200 import seqlib  # noqa: E402

SMS = 148
# heads, value columns, portions, us a layer in the scan and in blocks (both kernels, timed apart)
MEASURED = [
    (16, 128, [16], 17.8, 24.8), (16, 128, [24], 21.8, 26.5), (16, 128, [48], 37.4, 31.4), (16, 128, [2048], 1263.2, 598.4), (16, 128, [24] * 4, 26.8, 31.9), (16, 128, [48] * 4, 43.5, 39.5),
    (16, 128, [32] * 16, 97.1, 70.3), (16, 128, [128] * 16, 340.3, 211.1), (32, 128, [32] * 16, 161.3, 123.6), (16, 128, [700] * 3, 504.4, 312.6),
    (16, 128, [32] + [1] * 15, 39.9, 50.2), (16, 128, [128] + [1] * 15, 107.2, 91.0), (16, 128, [2048] + [1] * 15, 1464.5, 844.4),
    (8, 128, [32] + [1] * 15, 34.8, 37.7), (8, 128, [64] + [1] * 15, 56.2, 51.1), (16, 64, [32] + [1] * 15, 33.8, 38.9), (16, 64, [64] + [1] * 15, 56.4, 53.0),
    (32, 128, [32] + [1] * 15, 56.9, 81.5), (32, 128, [64] + [1] * 15, 81.4, 98.4), (32, 128, [300] + [1] * 15, 267.1, 216.8),
    (16, 128, [64] + [1] * 63, 100.1, 150.3), (16, 128, [300] + [1] * 63, 268.5, 256.5),
]


@pytest.mark.parametrize("heads,vdim,portions,scan,blocks", MEASURED)
def test_the_faster_one_is_taken(heads, vdim, portions, scan, blocks):
    few = sum(n < 32 for n in portions)
    assert bool(seqlib.load().calm_b200_seq_delta_blocks_pay(max(portions), few, heads, vdim, SMS)) == (blocks < scan)
