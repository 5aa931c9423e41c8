"""Steps of one token per sequence: gated linear attention as a stream over the states (k_seq_gla_step: key channels that fill part of a lane's four, one and two
groups of 128, value columns that end inside a warp's share) and the convolution with its state in one kernel (k_seq_conv_step: two to four taps, head vectors of each
instance and with a rest), against the plain float64 statement, from states that a prompt left behind; which of them ran is asserted, and what keeps the other kernels."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import bovinex_plain  # noqa: E402
import test_bovinex_gpu as tb  # noqa: E402
import test_vimulorn_gpu as tv  # noqa: E402
import vimulorn_plain  # noqa: E402

from calm_b200 import bovinex, seqlib, vimulorn  # noqa: E402

pytestmark = pytest.mark.gpu


def ran(route):
    return seqlib.load().calm_b200_seq_route_count(route)


def decode(mod, plain, t, cfg, dtype, route, steps=11):
    """Prompts of three lengths, decoded tokens of all, then of the two outer ones: (largest relative error, layers that ran as steps)."""
    weights, counts = t.weights(cfg, 5), [5, 2, 9]
    toks = [t.tokens(cfg, n + steps + 3, 3 + i) for i, n in enumerate(counts)]
    refs, worst, before = [plain.forward(cfg, t.as_f64(weights), x) for x in toks], 0.0, ran(route)
    with mod.from_tensors(cfg, weights, dtype, max_tokens=256, max_seqs=4, page=16) as m:
        slots = [m.open() for _ in counts]
        m.step(slots, [x[:n] for x, n in zip(toks, counts)], [0])
        assert ran(route) == before
        for k in range(steps + 3):
            who = [0, 1, 2] if k < steps else [2, 0]
            out = m.step([slots[i] for i in who], [[toks[i][counts[i] + k]] for i in who], list(range(len(who))))
            worst = max(worst, *(t.rel_err(out[j:j + 1], refs[i][counts[i] + k:counts[i] + k + 1]) for j, i in enumerate(who)))
    return worst, ran(route) - before


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,dim,vdim,steps", [(3, 16, 24, True), (2, 64, 20, True), (1, 128, 132, True), (4, 96, 68, True), (2, 132, 36, True), (1, 256, 64, True), (2, 64, 21, False)])
def test_gated_linear_attention(dtype, heads, dim, vdim, steps):
    cfg = tb.config([tb.gla(heads=heads, dim=dim, vdim=vdim, a_rank=8), tb.gla(heads=heads, dim=dim, vdim=vdim, a_rank=8)])
    err, layers = decode(bovinex, bovinex_plain, tb, cfg, dtype, 3)
    assert err < tb.TOL[dtype]
    assert layers >= 2 and layers % 2 == 0 if steps else layers == 0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("layer,steps", [(tv.delta(dim=64, vdim=64, conv=4), True), (tv.delta(dim=16, vdim=200, conv=3), True), (tv.window(dim=128, vdim=120, conv=2), True),
                                         (tv.window(dim=48, vdim=20, conv=4), True), (tv.delta(conv=5), False)], ids=["delta64", "delta16-200", "window128", "window48", "five taps"])
def test_convolution(dtype, layer, steps):
    cfg = tv.config([layer, layer])
    err, layers = decode(vimulorn, vimulorn_plain, tv, cfg, dtype, 4)
    assert err < tv.TOL[dtype]
    assert layers >= 2 and layers % 2 == 0 if steps else layers == 0


# keys of a decoded token: 32 a share up to eight shares, twelve shares as eight, more as before
@pytest.mark.parametrize("n,clusters", [(40, True), (95, True), (161, True), (255, True), (300, True), (383, True), (420, False)])
@pytest.mark.parametrize("layer", [tv.latent(), tv.latent(heads=16, dim=64, vdim=128, kv_rank=96), tv.window(size=1000), tb.attn(size=0), tb.attn(heads=8, kv_heads=1, dim=64, vdim=128, size=600, keep=5)],
                         ids=["latent", "latent16", "sinks", "groups", "eight heads"])
def test_shares_in_clusters(layer, n, clusters):
    t, mod, plain = (tb, bovinex, bovinex_plain) if layer["mixer"].get("rot") else (tv, vimulorn, vimulorn_plain)
    cfg = t.config([layer])
    weights, toks = t.weights(cfg, 5), t.tokens(cfg, n + 3)
    ref, before = plain.forward(cfg, t.as_f64(weights), toks), ran(5)
    with mod.from_tensors(cfg, weights, "bfloat16", max_tokens=512, max_seqs=2, page=16) as m:
        slot = m.open()
        m.step([slot], [toks[:n]], [0])
        at = ran(5)
        for k in range(3):
            out = m.step([slot], [[toks[n + k]]], [0])
            assert t.rel_err(out, ref[n + k:n + k + 1]) < t.TOL["bfloat16"], k
    assert at == before and (ran(5) > at) == clusters


# what keeps the merge: 32 clusters of eight where 33 fit, 4096 sums to read, wide latents; and next to them what does not
@pytest.mark.parametrize("layer,batch,n,clusters", [(tb.attn(heads=8, kv_heads=2, dim=128, vdim=128, size=0), 16, 250, False), (tb.attn(heads=8, kv_heads=2, dim=128, vdim=128, size=0), 8, 250, True),
                                                    (tb.attn(heads=8, kv_heads=2, dim=128, vdim=128, size=0), 16, 70, True), (tb.attn(heads=16, kv_heads=4, dim=64, vdim=64, size=0), 10, 300, False),
                                                    (tv.latent(heads=16, dim=16, vdim=16, kv_rank=256), 2, 70, False), (tv.latent(heads=8, dim=16, vdim=16, kv_rank=256), 2, 70, True)])
def test_clusters_where_they_pay(layer, batch, n, clusters):
    t, mod, plain = (tb, bovinex, bovinex_plain) if layer["mixer"].get("rot") else (tv, vimulorn, vimulorn_plain)
    cfg = t.config([layer])
    weights, toks = t.weights(cfg, 5), t.tokens(cfg, n + 2)
    ref = plain.forward(cfg, t.as_f64(weights), toks)
    with mod.from_tensors(cfg, weights, "bfloat16", max_tokens=batch * (n + 64), max_seqs=batch, page=16) as m:
        slots = [m.open() for _ in range(batch)]
        for s in slots:
            m.step([s], [toks[:n]], [0])
        before = ran(5)
        for k in range(2):
            out = m.step(slots, [[toks[n + k]]] * batch, list(range(batch)))
            for row in out:
                assert t.rel_err(row[None], ref[n + k:n + k + 1]) < t.TOL["bfloat16"], k
    assert (ran(5) > before) == clusters
