"""Products of many tokens whose results are added to the residual stream (with and without a parked second addend, through Dynamic Tanh), leave as a decay or
leave in part as a squared rectifier: row counts around the 32 tokens that an epilogue reads at a time and the 128 of a tile, on a width that ends inside one."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_bovinex_gpu as tb  # noqa: E402
import test_vimulorn_gpu as tv  # noqa: E402
import bovinex_plain  # noqa: E402
import vimulorn_plain  # noqa: E402

from calm_b200 import bovinex, vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 65, 95, 127, 129, 161])
def test_parallel_blocks(n):
    cfg = tb.config([tb.attn(), tb.gla(), tb.gla(mlp=None)], width=72)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, n)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=200, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]


@pytest.mark.parametrize("n", [64, 79, 128, 144])
def test_dynamic_tanh(n):
    cfg = tv.config([tv.delta(), tv.window()], width=72)
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, n)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=200, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tv.rel_err(got, vimulorn_plain.forward(cfg, tv.as_f64(t), toks)) < tv.TOL["bfloat16"]
