"""The delta rule over longer portions, in blocks of tokens (k_seq_delta_system, k_seq_delta_blocks), against the plain float64 statement: value columns around a
CTA's 32, portions that end inside a block, of one token beside a long one, key heads shared by several heads, keys that repeat (a token of a portion fed again and
again, where the corrections inside a block matter most), and a state that is carried on into a second portion and a decoded token."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_vimulorn_gpu as tv  # noqa: E402
import vimulorn_plain  # noqa: E402

from calm_b200 import seqlib, vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu


def in_blocks():  # layers that ran in blocks so far (SEQ_ROUTE_DELTA_BLOCKS)
    return seqlib.load().calm_b200_seq_route_count(2)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,kv,vdim,counts", [(2, 1, 4, (32,)), (4, 2, 36, (33, 1)), (2, 2, 128, (47, 5, 64)), (3, 3, 32, (16, 113)), (1, 1, 100, (300,))])
def test_blocks(dtype, heads, kv, vdim, counts):
    cfg = tv.config([tv.delta(heads=heads, kv_heads=kv, dim=128, vdim=vdim, conv=2)])
    t, toks = tv.weights(cfg, 8), tv.tokens(cfg, max(counts) + 60)
    toks[5:25] = [toks[5]] * 20
    ref = vimulorn_plain.forward(cfg, tv.as_f64(t), toks)
    with vimulorn.from_tensors(cfg, t, dtype, max_tokens=900, max_seqs=3, page=8) as m:
        slots, ran = [m.open() for _ in counts], in_blocks()
        at = np.cumsum((0,) + counts)
        out = m.step(slots, [toks[:n] for n in counts], list(range(sum(counts))))
        for i, n in enumerate(counts):
            assert tv.rel_err(out[at[i]:at[i + 1]], ref[:n]) < tv.TOL[dtype], n
        out = m.step(slots, [toks[n:n + 59] for n in counts], list(range(59 * len(counts))))
        for i, n in enumerate(counts):
            assert tv.rel_err(out[59 * i:59 * (i + 1)], ref[n:n + 59]) < tv.TOL[dtype], n
        assert in_blocks() == ran + 2
        out = m.step(slots, [toks[n + 59:n + 60] for n in counts], list(range(len(counts))))
        assert in_blocks() == ran + 2
        for i, n in enumerate(counts):
            assert tv.rel_err(out[i:i + 1], ref[n + 59:n + 60]) < tv.TOL[dtype], n


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("bad", [16, 17, 22, 35, 43])  # first, second, third and last of a block's four tokens that a thread takes together, and in the last block
def test_no_later_value_reaches_an_earlier_token(dtype, bad):
    cfg = tv.config([tv.delta(heads=2, kv_heads=1, dim=128, vdim=36, conv=2)])
    t, toks = tv.weights(cfg, 8), [x % 90 for x in tv.tokens(cfg, 44)]
    ref = vimulorn_plain.forward(cfg, tv.as_f64(t), toks)
    t["embed"][95] = float("nan")
    toks[bad] = 95
    with vimulorn.from_tensors(cfg, t, dtype, max_tokens=64, max_seqs=1, page=8) as m:
        ran = in_blocks()
        out = m.step([m.open()], [toks], list(range(44)))
        assert in_blocks() == ran + 1
    assert tv.rel_err(out[:bad], ref[:bad]) < tv.TOL[dtype] and np.isnan(out[bad:]).all()
