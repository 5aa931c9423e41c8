"""What the tensor-core matvecs of a token (cols.cuh) keep of their operands and sums, against float64: rows so long that sums left in the tensor core, which truncates,
would show; activations many orders of magnitude below the largest one beside them; weights that are not finite."""
from dataclasses import replace

import numpy as np
import pytest
import torch

from calm_b200 import lib
from calm_b200 import modelgen as mg

pytestmark = pytest.mark.gpu

L0 = "model.layers.0."


def _values(t, dtype):
    return t.view(torch.float16 if dtype == "fp16" else torch.float8_e5m2).double()


def _store(t, name, values, dtype):
    t[name] = values.float().to(torch.float16 if dtype == "fp16" else torch.float8_e5m2).view(t[name].dtype)


def _first_token(spec, t, token):
    """Its logits and cache entries on the device, all four tensor-core stages."""
    with lib.DeviceModel(spec, t) as dm:
        plan = [lib.load().calm_b200_token_plan(s) for s in range(4)]
        logits = dm.forward(token, 0)
        k, v = dm.read_kv(0, 0)
    assert all(plan), plan
    return np.asarray(logits, np.float64), np.asarray(k, np.float64), np.asarray(v, np.float64)


def _reference(spec, t, token, cached_v):
    """The first token of a one-layer model in float64; attention sees one position, whose values are read from the cache (they are rounded there)."""
    W = {n[len(L0):] if n.startswith(L0) else n: (x.double() if x.dtype == torch.float32 else _values(x, spec.dtype)) for n, x in t.items()}
    norm = lambda x, w: x / torch.sqrt((x * x).mean() + spec.norm_eps) * w
    x = W["model.embed.weight"][token]
    xn = norm(x, W["attn.norm.weight"])
    k, v = W["attn.wk.weight"] @ xn, W["attn.wv.weight"] @ xn
    att = torch.from_numpy(cached_v).reshape(spec.n_kv_heads, -1).repeat_interleave(spec.n_heads // spec.n_kv_heads, 0).reshape(-1)
    x = x + W["attn.wo.weight"] @ att
    xn = norm(x, W["mlp.norm.weight"])
    x = x + W["mlp.w2.weight"] @ (torch.nn.functional.silu(W["mlp.w1.weight"] @ xn) * (W["mlp.w3.weight"] @ xn))
    return (W["model.output.weight"] @ norm(x, W["model.norm.weight"])).numpy(), k.numpy(), v.numpy()


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("dtype,hidden", [("fp8", 14336), ("fp8", 28672), ("fp16", 14336)])
def test_sums_of_long_rows(dtype, hidden):
    """w2's rows.  FP32 sums of them are 1.6e-7 from float64 (ring.cuh), those of FFN up 2e-7 and the classifier's 1e-7: 2.8e-7 together; left in the tensor core the
    rows of 28672 are 1.8e-6 off, those of 14336 0.9e-6."""
    spec = replace(mg.SPECS["pf-tiny-hd128"], name="long", dtype=dtype, dim=512, hidden_dim=hidden, n_layers=1, qkv_bias=False)
    err = []
    for seed in range(4):
        t = mg.generate(spec, seed=seed)
        t[L0 + "attn.wo.weight"].zero_()
        t[L0 + "mlp.norm.weight"] *= 8  # the units' output outweighs what it is added to
        got, _, v = _first_token(spec, t, 5)
        err.append(_rel(got, _reference(spec, t, 5, v)[0]))
    assert np.median(err) < 4.5e-7, err
