"""Products on pairs of CTAs (k_seq_gemm_pair; K of about 1900 and more, deeper ones where results are added to the stream): token counts around the 32 that an
epilogue reads at a time, the halves of a tile that the two CTAs bring and its 256, row counts that end inside a CTA's half, a K that ends inside a 64-deep step,
every epilogue that large products have, more tiles than pairs, and a captured decode step.  Each test asserts that its products did run there."""
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

from calm_b200 import bovinex, seqlib, tabisun, vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu

FF = {"ff": 2000, "kind": "dense"}
CAPTURE, PAIRS = 0, 16  # SEQ_ROUTE_*
F32, ACT, DYT, RES, GLU = 0, 1, 2, 3, 7  # EPI_*


@pytest.fixture
def on_pairs():
    """Launches on pairs of CTAs since the test began, by epilogue."""
    lib = seqlib.load()
    before = [lib.calm_b200_seq_route_count(PAIRS + e) for e in range(8)]
    return lambda epi: lib.calm_b200_seq_route_count(PAIRS + epi) - before[epi]


@pytest.mark.parametrize("n", [64, 127, 161, 256, 257, 300])
def test_parallel_blocks(n, on_pairs):  # fp32 columns, squared rectifiers and a decay's input from one product
    cfg = tb.config([tb.attn(mlp=FF), tb.gla(mlp=FF)], width=2048)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, n)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]
    assert on_pairs(F32) >= 2


@pytest.mark.parametrize("n", [65, 160, 287])
def test_dynamic_tanh(n, on_pairs):
    cfg = tv.config([tv.window(mlp={"ff": 2000, "kind": "dense", "limit": 4.0}), tv.window(mlp=None)], width=2040)
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, n)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tv.rel_err(got, vimulorn_plain.forward(cfg, tv.as_f64(t), toks)) < tv.TOL["bfloat16"]
    assert on_pairs(GLU) >= 1 and (on_pairs(DYT) >= 1) == (n <= 224)


@pytest.mark.parametrize("n", [66, 255])
def test_gated_units(n, on_pairs):  # gate and up rows in turn, capped logits
    cfg = tt.config([tt.capped(mlp=FF)], width=2048)
    t, toks = tt.weights(cfg, 6), tt.tokens(cfg, n)
    with tabisun.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tt.rel_err(got, tabisun_plain.forward(cfg, tt.as_f64(t), toks), "bfloat16") < tt.TOL["bfloat16"]
    assert on_pairs(GLU) >= 1


def test_more_tiles_than_pairs(on_pairs):  # 74 x 2 tiles of logits, two to a pair
    cfg = tb.config([tb.gla(mlp=None)], width=2048, vocab=18900)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, 500)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=600, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(500)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]
    assert on_pairs(F32) >= 2


# residual epilogues: deep products of one wave, with tiles that are full of tokens and that are not
@pytest.mark.parametrize("n", [64, 127, 200, 257, 300])
def test_two_addends(n, on_pairs):
    cfg = tb.config([tb.attn(mlp={"ff": 6000, "kind": "dense"}), tb.gla(mlp={"ff": 6000, "kind": "dense"})], width=2040)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, n)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]
    assert on_pairs(RES) == 2


def test_two_addends_over_two_waves(on_pairs):  # 20 x 4 tiles
    cfg = tb.config([tb.gla(mlp={"ff": 2048, "kind": "dense"})], width=5112)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, 1000)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=1100, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(1000)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]
    assert on_pairs(RES) == 1


@pytest.mark.parametrize("n", [65, 160, 287])
def test_dynamic_tanh_of_deep_products(n, on_pairs):
    cfg = tv.config([tv.window(mlp={"ff": 3504, "kind": "dense", "limit": 4.0}), tv.window(mlp={"ff": 3504, "kind": "dense", "limit": 4.0})], width=2040)
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, n)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(n)))
    assert tv.rel_err(got, vimulorn_plain.forward(cfg, tv.as_f64(t), toks)) < tv.TOL["bfloat16"]
    assert on_pairs(DYT) >= 2


def test_queries_from_a_deep_latent(on_pairs):
    cfg = tv.config([tv.latent(heads=3, dim=24, q_rank=2048, mlp=None)], width=64)
    t, toks = tv.weights(cfg, 6), tv.tokens(cfg, 100)
    with vimulorn.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(100)))
    assert tv.rel_err(got, vimulorn_plain.forward(cfg, tv.as_f64(t), toks)) < tv.TOL["bfloat16"]
    assert on_pairs(ACT) >= 1


def test_shallow_products_stay_on_one_cta(on_pairs):
    cfg = tb.config([tb.attn(mlp=FF), tb.gla(mlp=FF)], width=512)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, 300)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(300)))
    assert tb.rel_err(got, bovinex_plain.forward(cfg, tb.as_f64(t), toks)) < tb.TOL["bfloat16"]
    assert on_pairs(F32) == 0 and on_pairs(RES) == 0  # K = 512; K = 2000 is not deep enough for what is added to the stream


def test_captured_decode_step(on_pairs):  # 70 sequences of one token: launches in clusters inside a graph that is replayed
    cfg = tb.config([tb.attn(size=0, mlp=FF), tb.gla(mlp=FF)], width=2048)
    t, toks = tb.weights(cfg, 6), tb.tokens(cfg, 210)
    with bovinex.from_tensors(cfg, t, "bfloat16", max_tokens=70 * 8, max_seqs=70, page=8) as m:
        slots, captures = [m.open() for _ in range(70)], m.lib.calm_b200_seq_route_count(CAPTURE)
        got = [m.step(slots, [[toks[3 * s + i]] for s in slots], list(range(70))) for i in range(3)]
        assert m.lib.calm_b200_seq_route_count(CAPTURE) == captures + 1 and on_pairs(F32) >= 2
    for s in (0, 1, 31, 32, 63, 64, 69):
        ref = bovinex_plain.forward(cfg, tb.as_f64(t), toks[3 * s:3 * s + 3])
        for i in range(3):
            assert tb.rel_err(got[i][s:s + 1], ref[i:i + 1]) < tb.TOL["bfloat16"], (s, i)
