"""Gated linear attention over long portions, cut into chunks of tokens (k_seq_gla_local, k_seq_gla_starts, k_seq_gla_apply), against the plain float64
statement: key channels of both instances, value columns around a CTA's share, chunks that end inside a block of tokens, portions of several lengths (one token
among them, and fewer than a chunk), two chunks of a sequence where sequences x heads x columns leave no more, a normaliser's column beside 128 (mLSTM), and a state
that is carried into a second portion.  Whether the chunks ran is asserted: their 16-byte copies need a projection of whole float4s."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_bovinex_gpu as tb  # noqa: E402
import test_zazilix_gpu as tz  # noqa: E402
import bovinex_plain  # noqa: E402
import zazilix_plain  # noqa: E402

from calm_b200 import bovinex, seqlib, zazilix  # noqa: E402

pytestmark = pytest.mark.gpu


def chunked():  # layers that ran as chunks so far (SEQ_ROUTE_GLA_CHUNKS)
    return seqlib.load().calm_b200_seq_route_count(1)


# chunks of 8 tokens for few heads; of 48 and 56 where sequences x heads x columns fill more of the device
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,dim,vdim,counts", [(2, 64, 20, (165, 1)), (3, 128, 36, (161, 7, 170)), (1, 128, 132, (200,)), (2, 64, 68, (163, 300)), (16, 128, 128, (330,)),
                                                   (12, 64, 64, (600, 160, 55, 1)), (16, 128, 128, (170, 161, 33, 1))])
def test_chunks(dtype, heads, dim, vdim, counts):
    cfg = tb.config([tb.gla(heads=heads, dim=dim, vdim=vdim, a_rank=8)])
    t, toks = tb.weights(cfg, 5), tb.tokens(cfg, max(counts) + 170)
    ref = bovinex_plain.forward(cfg, tb.as_f64(t), toks)
    with bovinex.from_tensors(cfg, t, dtype, max_tokens=3200, max_seqs=4, page=16) as m:
        slots, ran = [m.open() for _ in counts], chunked()
        out = m.step(slots, [toks[:n] for n in counts], list(range(sum(counts))))
        at = np.cumsum((0,) + counts)
        for i, n in enumerate(counts):
            assert tb.rel_err(out[at[i]:at[i + 1]], ref[:n]) < tb.TOL[dtype], n
        out = m.step(slots, [toks[n:n + 170] for n in counts], list(range(170 * len(counts))))  # from the states left behind
        for i, n in enumerate(counts):
            assert tb.rel_err(out[170 * i:170 * (i + 1)], ref[n:n + 170]) < tb.TOL[dtype], n
        assert chunked() == ran + 2
        one = m.step(slots[:1], [toks[:1]], [0])  # and a decoded token from the last one
        assert chunked() == ran + 2
        again = bovinex_plain.forward(cfg, tb.as_f64(t), toks[:counts[0] + 170] + toks[:1])[-1:]
        assert tb.rel_err(one, again) < tb.TOL[dtype]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("layer", [tz.mlstm(heads=2, dim=128, vdim=128, mlp=None), tz.mamba(heads=4, vdim=64, state=64, norm_groups=2, mlp=None), tz.pair(rheads=2, rdim=64, rvdim=68, mlp=None)],
                         ids=["mlstm", "mamba2", "hgrn2"])
def test_linear_recurrences(dtype, layer):
    cfg = tz.config([layer])
    t, toks = tz.weights(cfg, 5), tz.tokens(cfg, 200)
    ref = zazilix_plain.forward(cfg, tz.as_f64(t), toks)
    with zazilix.from_tensors(cfg, t, dtype, max_tokens=300, max_seqs=2, page=16) as m:
        ran, a, b = chunked(), m.open(), m.open()
        out = m.step([a, b], [toks[:165], toks[:7]], list(range(172)))
        assert chunked() == ran + 1
        assert tz.rel_err(out[:165], ref[:165]) < tz.TOL[dtype] and tz.rel_err(out[165:], ref[:7]) < tz.TOL[dtype]
        out = m.step([a], [toks[165:]], list(range(35)))  # the scan goes on from the state left behind
        assert chunked() == ran + 1 and tz.rel_err(out, ref[165:]) < tz.TOL[dtype]
