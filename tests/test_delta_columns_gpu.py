"""The delta-rule scan with its state in registers (k_seq_delta_scan_reg): value widths around the 32 columns of a CTA and step lengths around its blocks of four
tokens, against the plain float64 statement."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_vimulorn_gpu as tv  # noqa: E402
import vimulorn_plain  # noqa: E402

from calm_b200 import vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("dim,vdim", [(32, 4), (64, 36), (128, 32), (128, 128), (32, 100)])
def test_columns_and_blocks(dtype, dim, vdim):
    cfg = tv.config([tv.delta(heads=4, kv_heads=2, dim=dim, vdim=vdim, conv=2)])
    t, toks = tv.weights(cfg, 8), tv.tokens(cfg, 31)
    ref = vimulorn_plain.forward(cfg, tv.as_f64(t), toks)
    with vimulorn.from_tensors(cfg, t, dtype, max_tokens=96, max_seqs=2, page=8) as m:
        s1, s2 = m.open(), m.open()
        got, at = [], 0
        for n in (1, 3, 4, 5, 9, 8, 1):  # 31 tokens; the other sequence restarts nothing in between
            out = m.step([s1, s2], [toks[at:at + n], toks[at:at + n]], list(range(2 * n)))
            assert tv.rel_err(out[n:], ref[at:at + n]) < tv.TOL[dtype]
            got.append(out[:n])
            at += n
    assert tv.rel_err(np.concatenate(got), ref) < tv.TOL[dtype]
