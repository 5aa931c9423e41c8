"""Which layer-list products run on pairs of CTAs (calm_b200_seq_pairs_pay): measured products on both sides of the line, for every epilogue that was measured on
both; where results are added to the stream by whole steps, in which most of a pair's start is hidden."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

from calm_b200 import seqlib  # noqa: E402

PAIRS = 74
EPI = {"f32": 0, "dyt": 2, "res": 3, "glu": 7}
# epilogue, rows, K, [(tokens, us with tiles of 128, us on pairs)] alone
MEASURED = [
    ("f32", 5712, 2048, [(64, 18.7, 16.4), (128, 22.2, 20.2), (1024, 40.0, 32.9), (2048, 57.5, 46.0)]),
    ("f32", 4176, 4096, [(64, 31.5, 24.0), (300, 35.3, 33.0), (2048, 69.2, 56.7)]),
    ("f32", 3072, 1024, [(256, 10.7, 13.2), (512, 11.0, 13.5)]),
    ("res", 4096, 1024, [(1400, 36.0, 41.7), (2048, 41.9, 43.8)]),
    ("dyt", 2048, 2048, [(64, 20.7, 17.1), (256, 24.2, 26.3), (512, 26.2, 27.6), (2048, 32.2, 30.6)]),
    ("dyt", 1024, 2816, [(128, 22.8, 19.5), (256, 23.6, 25.1), (1024, 24.4, 26.2)]),
    ("dyt", 2048, 5632, [(64, 39.5, 27.9), (256, 43.7, 38.3), (2048, 51.6, 45.2)]),
    ("dyt", 1024, 1024, [(256, 17.5, 21.2), (1024, 18.2, 22.0)]),
    ("glu", 11264, 2048, [(64, 23.5, 20.1), (256, 29.5, 26.9), (2048, 130.5, 84.3)]),
]


# rows, K, [(tokens, us more on pairs)] a product in whole steps
ADDED = [
    (2048, 2048, [(200, 3.5), (256, 2.4), (512, 4.0), (1024, 4.1)]),
    (2048, 5632, [(64, -11.4), (128, -9.1), (200, -4.4), (1024, -4.0), (2048, -2.3)]),
    (1024, 2816, [(64, -8.3), (128, -3.5), (256, 5.4), (512, 3.9)]),
    (4096, 4096, [(64, -6.1), (128, -2.6), (200, -2.5), (2048, -20.5)]),
    (4096, 2048, [(256, 3.5), (1024, 2.4), (2048, -5.8)]),
    (8192, 2048, [(200, 8.2), (256, 11.5), (1024, -8.5), (2048, -26.5)]),
    (1024, 1024, [(128, 3.6), (256, 4.2), (2048, 4.9)]),
]


@pytest.mark.parametrize("epi,rows,k,points", MEASURED, ids=[f"{e}-{r}x{k}" for e, r, k, _ in MEASURED])
def test_the_faster_one_is_taken(epi, rows, k, points):
    pay = seqlib.load().calm_b200_seq_pairs_pay
    for n, small, large in points:
        if large < small or large - small > 1.3:
            assert bool(pay(rows, n, k, EPI[epi], PAIRS)) == (large < small), (n, small, large)


@pytest.mark.parametrize("rows,k,points", ADDED, ids=[f"{r}x{k}" for r, k, _ in ADDED])
def test_the_faster_one_is_taken_in_steps(rows, k, points):
    pay = seqlib.load().calm_b200_seq_pairs_pay
    for n, more in points:
        assert bool(pay(rows, n, k, EPI["res"], PAIRS)) == (more < 0), (n, more)
