"""Products on pairs of CTAs (k_seq_gemm_pair; K of about 1900 and more): token counts around the 32 that an epilogue reads at a time, the halves of a tile that
the two CTAs bring and its 256, row counts that end inside a CTA's half, a K that ends inside a 64-deep step, every epilogue that large products have, and
more tiles than pairs."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_bovinex_gpu as tb  # noqa: E402
import test_tabisun_gpu as tt  # noqa: E402
import test_vimulorn_gpu as tv  # noqa: E402
import bovinex_plain  # noqa: E402
import tabisun_plain  # noqa: E402
import vimulorn_plain  # noqa: E402

from calm_b200 import bovinex, tabisun, vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu

FF = {"ff": 2000, "kind": "dense"}


@pytest.mark.parametrize("n", [64, 127, 161, 256, 257, 300])
def test_parallel_blocks(n):  # fp32 columns, squared rectifiers and a decay's input from one product; the sum with a parked addend
    cfg = tb.config([tb.attn(mlp=FF), tb.gla(mlp=FF)], width=2048)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, n)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]


@pytest.mark.parametrize("n", [65, 160, 287])
def test_dynamic_tanh(n):
    cfg = tv.config([tv.window(mlp={"ff": 2000, "kind": "dense", "limit": 4.0}), tv.window(mlp=None)], width=2040)
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, n)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tv.rel_err(got, vimulorn_plain.forward(cfg, tv.as_f64(t), toks)) < tv.TOL["bfloat16"]


@pytest.mark.parametrize("n", [66, 255])
def test_gated_units(n):  # gate and up rows in turn, capped logits
    cfg = tt.config([tt.capped(mlp=FF)], width=2048)
    t, toks = tt.weights(cfg, 6), tt.tokens(cfg, n)
    with tabisun.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tt.rel_err(got, tabisun_plain.forward(cfg, tt.as_f64(t), toks), "bfloat16") < tt.TOL["bfloat16"]


def test_more_tiles_than_pairs():  # 74 x 2 tiles of logits, two to a pair
    cfg = tb.config([tb.gla(mlp=None)], width=2048, vocab=18900)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, 500)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=600, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(500)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]


# residual epilogues: deep products of one wave, with tiles that are full of tokens and that are not
@pytest.mark.parametrize("n", [64, 127, 200, 257, 300])
def test_two_addends(n):
    cfg = tb.config([tb.attn(mlp={"ff": 6000, "kind": "dense"}), tb.gla(mlp={"ff": 6000, "kind": "dense"})], width=2040)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, n)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]


def test_two_addends_over_two_waves():  # 20 x 4 tiles
    cfg = tb.config([tb.gla(mlp={"ff": 2048, "kind": "dense"})], width=5112)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, 1000)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=1100, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(1000)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]


@pytest.mark.parametrize("n", [65, 160, 287])
def test_dynamic_tanh_of_deep_products(n):
    cfg = tv.config([tv.window(mlp={"ff": 3500, "kind": "dense", "limit": 4.0}), tv.window(mlp={"ff": 3500, "kind": "dense", "limit": 4.0})], width=2040)
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, n)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tv.rel_err(got, vimulorn_plain.forward(cfg, tv.as_f64(t), toks)) < tv.TOL["bfloat16"]
