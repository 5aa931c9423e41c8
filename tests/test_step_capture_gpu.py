"""Captured decode steps outlive steps whose batch description is a few numbers longer than any before (one more wanted row at a time)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_bovinex_gpu as tb  # noqa: E402

from calm_b200 import bovinex  # noqa: E402

pytestmark = pytest.mark.gpu

CAPTURE = 0


def test_one_more_wanted_row_at_a_time():
    cfg = tb.config([tb.attn(), tb.gla()])
    t, toks = tb.weights(cfg, 4), tb.tokens(cfg, 64)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=900, max_seqs=2, page=8) as m:
        captures = lambda: m.lib.calm_b200_seq_route_count(CAPTURE)  # noqa: E731
        a, b = m.open(), m.open()
        m.step([a], [toks], list(range(9)))  # rows for 9 wanted tokens, then for 18
        m.step([a], [toks], list(range(10)))
        want = m.step([b], [toks[:1]], [0])
        at = captures()
        for n in range(11, 18):  # no buffer has to move for these
            m.step([a], [toks], list(range(n)))
            m.step([b], [toks[n:n + 1]], [0])
        assert captures() == at
        m.close_seq(b)
        b = m.open()
        again = m.step([b], [toks[:1]], [0])
    assert captures() == at and np.array_equal(want, again)
