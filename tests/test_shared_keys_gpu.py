"""Prompt attention of the layer-list runtime where a few new tokens stand behind a long prefix, so that its CTAs share the keys out (k_seq_attn_flash with partial
results and their merge), against the plain float64 statements: shares that are empty for a sequence without a prefix, a share whose keys all lie outside a row's
window, kept positions, a sink that counts once, a gate behind the merge, and a decoded token in the same step."""
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


def _three(m, toks, prefix, n):
    """n tokens behind `prefix`, 16 behind nothing, one behind 300."""
    s1, s2, s3 = m.open(), m.open(), m.open()
    m.step([s1, s3], [toks[:prefix], toks[:300]], [], fetch=False)
    out = m.step([s1, s2, s3], [toks[prefix:prefix + n], toks[:16], toks[300:301]], list(range(n + 17)))
    return np.concatenate([out[:n], out[n:n + 16], out[n + 16:]])


# prefixes of 8 to 18 tiles of 64 keys, in shares of two tiles or more
@pytest.mark.parametrize("heads,kv,dim,size,keep,prefix,n", [(4, 2, 64, 0, 0, 1100, 33), (8, 1, 128, 0, 0, 1024, 16), (3, 1, 64, 700, 70, 1090, 50), (6, 1, 128, 600, 0, 1150, 17),
                                                             (2, 2, 64, 0, 0, 495, 17)])
def test_shares(heads, kv, dim, size, keep, prefix, n):
    cfg = tb.config([tb.attn(size=size, keep=keep, heads=heads, kv_heads=kv, dim=dim, vdim=dim, rot=16, scale=dim ** -0.5)])
    t, toks = tb.weights(cfg, 23), tb.tokens(cfg, prefix + n)
    ref = bovinex_plain.forward(cfg, tb.as_f64(t), toks)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=2400, max_seqs=3, page=16) as m:
        got = _three(m, toks, prefix, n)
    want = np.concatenate([ref[prefix:], ref[:16], ref[300:301]])
    assert tb.rel_err(got, want) < tb.TOL["bfloat16"]
    assert tb.rel_err(got[n:n + 16], ref[:16]) < tb.TOL["bfloat16"] and tb.rel_err(got[n + 16:], ref[300:301]) < tb.TOL["bfloat16"]


@pytest.mark.parametrize("heads,kv,dim,size", [(4, 2, 64, 900), (5, 1, 128, 2000)])
def test_sink_counts_once(heads, kv, dim, size):
    cfg = tv.config([tv.window(heads=heads, kv_heads=kv, dim=dim, vdim=dim, size=size, scale=dim ** -0.5)])
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, 1050)
    ref = vimulorn_plain.forward(cfg, tv.as_f64(t), toks)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=2400, max_seqs=3, page=16) as m:
        got = _three(m, toks, 1024, 26)
    assert tv.rel_err(got, np.concatenate([ref[1024:], ref[:16], ref[300:301]])) < tv.TOL["bfloat16"]
