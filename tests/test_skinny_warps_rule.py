"""Warps of a CTA in the layer-list products of few tokens (calm_b200_seq_skinny_warps): measured products on both sides of the line, routed ones, most of whose CTAs find no row, among them."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

from calm_b200 import seqlib  # noqa: E402

SMS = 148
# weight rows, columns, matrices, rows over all groups (0: not grouped), us with 8 and with 16 warps
MEASURED = [
    (2048, 5632, 1, 0, 9.6, 7.1), (5632, 1024, 1, 0, 2.9, 6.0), (3216, 1024, 1, 0, 2.1, 3.8),
    (512, 2048, 8, 2, 4.47, 3.83), (512, 2048, 4, 2, 4.58, 3.39), (512, 1024, 8, 2, 3.11, 3.46), (2048, 1024, 8, 2, 4.39, 7.14), (2048, 4096, 8, 2, 9.69, 12.29),
    (4096, 2048, 8, 2, 10.10, 15.44), (512, 2048, 16, 4, 5.14, 5.36), (1024, 1024, 16, 2, 4.27, 6.25), (512, 2048, 64, 6, 7.28, 10.69), (1408, 2048, 64, 6, 13.01, 24.14),
    (768, 2048, 128, 8, 12.87, 23.47), (256, 1024, 32, 4, 3.36, 4.45), (512, 2048, 8, 8, 5.80, 6.88), (1024, 2048, 8, 8, 9.45, 12.37), (512, 2048, 64, 32, 14.92, 23.01), (128, 1024, 128, 4, 3.51, 5.96),
]


@pytest.mark.parametrize("m,k,groups,rows,eight,sixteen", MEASURED)
def test_the_faster_one_is_taken(m, k, groups, rows, eight, sixteen):
    assert seqlib.load().calm_b200_seq_skinny_warps(m, k, groups, rows, SMS) == (16 if sixteen < eight else 8)
