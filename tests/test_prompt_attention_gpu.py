"""The one-kernel prompt attention of the layer-list runtime (k_seq_attn_flash) at the widths it is built for, against the plain float64 statements: head groups
that divide over its warps in different ways, portions around multiples of its 16-row and 64-key tiles that continue a cached prefix, a window with and
without kept first positions, a gate per channel, a sink, several sequences of unequal length in one step."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_bovinex_gpu as tb  # noqa: E402
import test_vimulorn_gpu as tv  # noqa: E402
import bovinex_plain  # noqa: E402
import vimulorn_plain  # noqa: E402

from calm_b200 import bovinex, vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu


# groups of 1, 2, 3, 6 and 8 heads; the kept positions before, inside and beyond the first query's window
@pytest.mark.parametrize("heads,kv,dim,size,keep", [(2, 2, 64, 0, 0), (4, 2, 128, 23, 5), (3, 1, 64, 70, 70), (6, 1, 64, 33, 130), (8, 1, 128, 64, 1)])
def test_windows_groups_and_tiles(heads, kv, dim, size, keep):
    cfg = tb.config([tb.attn(size=size, keep=keep, heads=heads, kv_heads=kv, dim=dim, vdim=dim, rot=16, scale=dim ** -0.5)])
    t, toks = tb.weights(cfg, 21), tb.tokens(cfg, 150)
    ref = bovinex_plain.forward(cfg, tb.as_f64(t), toks)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=600, max_seqs=3, page=8) as m:
        s1, s2, s3 = m.open(), m.open(), m.open()
        a = m.step([s1], [toks[:65]], list(range(65)))
        b = m.step([s1, s2, s3], [toks[65:], toks[:16], toks[:3]], list(range(104)))  # 85 and 16 tokens in this kernel, 3 in the decode kernel
    err = tb.rel_err(np.concatenate([a, b[:85]]), ref)
    assert err < tb.TOL["bfloat16"], err
    assert tb.rel_err(b[85:101], ref[:16]) < tb.TOL["bfloat16"] and tb.rel_err(b[101:], ref[:3]) < tb.TOL["bfloat16"]


@pytest.mark.parametrize("heads,kv,dim,size", [(4, 2, 64, 40), (5, 1, 128, 200)])
def test_sink_and_short_convolutions(heads, kv, dim, size):
    cfg = tv.config([tv.window(heads=heads, kv_heads=kv, dim=dim, vdim=dim, size=size, scale=dim ** -0.5)])
    t, toks = tv.weights(cfg, 4), tv.tokens(cfg, 130)
    ref = vimulorn_plain.forward(cfg, tv.as_f64(t), toks)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=2, page=16) as m:
        s1, s2 = m.open(), m.open()
        a = m.step([s1], [toks[:63]], list(range(63)))
        b = m.step([s1, s2], [toks[63:], toks[:130]], list(range(197)))
    assert tv.rel_err(np.concatenate([a, b[:67]]), ref) < tv.TOL["bfloat16"]
    assert tv.rel_err(b[67:], ref) < tv.TOL["bfloat16"]
