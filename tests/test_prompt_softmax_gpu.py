"""Prompt attention of the engine where one key holds nearly all of the softmax, on hand-made two-layer models whose second layer caches what the first layer's
attention gave, against the serial calls (fp32 weights)."""
import math
from dataclasses import replace

import numpy as np
import pytest
import torch

from calm_b200 import lib
from calm_b200 import modelgen as mg
from calm_b200.cstructs import FF_UPDATE_KV_ONLY

pytestmark = pytest.mark.gpu


def _model(hd, value, gain, delta):
    """Tokens 1, 2, 3 are basis vectors.  Every query scores a key of token 1 `delta` above one of any other; token t's value is value[t] in all dimensions.  The
    first layer's attention comes out in channel 4, times `gain`, and channel 4 is what the second layer's values hold."""
    spec = replace(mg.SPECS["pf-tiny"], name="softmax", dtype="fp16", dim=256, n_heads=256 // hd, n_kv_heads=256 // hd, head_dim=hd, hidden_dim=256, rotary_dim=2, max_seq_len=1200)
    t = {k: torch.zeros_like(v) for k, v in mg.generate(spec, seed=1).items()}
    root = 16.0  # a normed basis vector
    for tok in (1, 2, 3):
        t["model.embed.weight"][tok, tok] = 1.0
    for l in range(2):
        p = f"model.layers.{l}."
        t[p + "attn.norm.weight"].fill_(1.0), t[p + "mlp.norm.weight"].fill_(1.0)
    t["model.norm.weight"].fill_(1.0)
    a = "model.layers.0.attn.w%s.weight"
    for h in range(spec.n_heads):
        t[a % "q"][h * hd + 8, 1:4] = 1 / root  # a query is one in channel 8, which does not turn
        t[a % "k"][h * hd + 8, 1] = delta * math.sqrt(hd) / root
    for tok, v in value.items():
        t[a % "v"][:, tok] = v / root
    t[a % "o"][4, 5] = gain
    t["model.layers.1.attn.wv.weight"][:, 4] = 1.0
    return spec, t


def _both(spec, tensors, toks):
    out = []
    for batched in (False, True):
        with lib.DeviceModel(spec, tensors, seq_len=1200) as dm:
            if batched:
                assert dm.prefill(toks, 0) == 1
            else:
                for i, x in enumerate(toks):
                    dm.forward(int(x), i, FF_UPDATE_KV_ONLY)
            out.append(np.stack([dm.read_kv(1, i)[1] for i in range(len(toks))]))
    return out


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("bits", [10, 18, 24, 28])
def test_long_tail_of_small_weights(hd, bits):
    """A first key without a value, and a thousand keys of 2^-bits of its weight that hold all there is."""
    value = 2.0 ** min(15, bits - 8)  # large enough that what is left of it is an ordinary activation
    spec, t = _model(hd, {1: 0.0, 2: value}, 2.0 ** (bits - 9) / value, bits * math.log(2.0))
    serial, batched = _both(spec, t, [1] + [2] * 1030)
    assert np.abs(serial[40:]).min() > 1e-3
    # a weight keeps 22 bits or, where that is coarser, steps of 2^-39 of the largest (half a step: 2^-40); two roundings to fp16
    np.testing.assert_allclose(batched[40:], serial[40:], rtol=2.0 ** -10 + 2.0 ** -22 + 2.0 ** (bits - 40))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("at", [5, 15, 16, 70, 97])  # inside a 16-key block, at its ends, in later tiles
def test_an_infinite_value_reaches_no_earlier_token(hd, at):
    spec, t = _model(hd, {1: 3.0, 2: 1.0}, 0.5, 1.0)
    t["model.layers.0.attn.wv.weight"][:, 3] = 60000.0  # token 3: beyond what an fp16 cache holds (an e5m2 one saturates)
    toks = [1] + [2] * 99
    toks[at] = 3
    serial, batched = _both(spec, t, toks)
    assert np.isfinite(serial[:at]).all() and np.abs(serial[:at]).min() > 1e-3 and not np.isfinite(serial[at:]).any()
    np.testing.assert_allclose(batched[:at], serial[:at], rtol=2.0 ** -10)  # two roundings to fp16
    assert not np.isfinite(batched[at:]).any()
