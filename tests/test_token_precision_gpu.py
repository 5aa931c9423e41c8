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


@pytest.mark.parametrize("dtype", ["fp8", "fp16"])
@pytest.mark.parametrize("dim,hidden", [(512, 1024), (2176, 4864)])  # one piece of a row, several
def test_small_activations_beside_large_ones(dtype, dim, hidden):
    """Every stage's input has entries of some 2^26 times the others (2^12 in front of wo, whose input is held in f16), first, in the middle and last, met by weights of zero: the
    result is made of the small ones.  FP32 products are exact to 2^-24 whatever lies beside them; 2e-6 leaves the four stages' and the classifier's sums 3e-7 each.
    Fixed point with 32 bits below the largest entry was 2e-3 to 1e-2 off."""
    spec = replace(mg.SPECS["pf-tiny-hd128"], name="outliers", dtype=dtype, dim=dim, hidden_dim=hidden, n_heads=dim // 128, n_kv_heads=dim // 128, n_layers=1, qkv_bias=False)
    t, g = mg.generate(spec, seed=4), torch.Generator().manual_seed(1)
    get = lambda n: _values(t[n], dtype)
    at, up = [0, dim // 2 + 1, dim - 1], [0, hidden // 2 + 1, hidden - 1]
    x = torch.randn(spec.vocab_size, dim, generator=g).double() * 2.0**-11
    x[:, at] = 2.0**15
    _store(t, "model.embed.weight", x, dtype)
    for n in ("attn.norm.weight", "mlp.norm.weight"):
        t[L0 + n] *= 2.0**22  # the small ones leave the norm as values of about 0.1
    for n in (L0 + "attn.wq.weight", L0 + "attn.wk.weight", L0 + "attn.wv.weight", L0 + "mlp.w1.weight", L0 + "mlp.w3.weight", "model.output.weight"):
        w = get(n)
        w[:, at] = 0
        if ".w1." in n or ".w3." in n:
            w[up] *= 2.0**13
        if ".wv." in n:
            w[at] *= 2.0**12
        _store(t, n, w, dtype)
    for n, zero in (("attn.wo.weight", at), ("mlp.w2.weight", up)):
        w = get(L0 + n)
        w[:, zero] = 0
        w[at] = 0  # (the large entries of the residual stay as they are)
        _store(t, L0 + n, w, dtype)
    got, k, v = _first_token(spec, t, 5)
    ref, rk, rv = _reference(spec, t, 5, v)
    for a, b in ((k, rk), (v, rv)):
        assert (np.abs(a - b) <= 2.0**-10 * np.abs(b) + 2.0**-24).all()  # the next f16 value at most
    assert _rel(got, ref) < 2e-6


@pytest.mark.parametrize("dtype", ["fp8", "fp16"])
def test_infinite_weights(dtype):
    """A row with an infinite weight gives that infinity with the activation's sign, not a NaN of its pieces; rows beside it are untouched.  Seen in the cache, where a value row's
    result goes by itself (a NaN would end at the lower limit of the clip, as one infinity)."""
    spec = replace(mg.SPECS["pf-tiny-hd128"], name="infinite", dtype=dtype, n_layers=1, qkv_bias=False)
    t = mg.generate(spec, seed=6)
    xn = _values(t["model.embed.weight"], dtype)[5] * t[L0 + "attn.norm.weight"].double()
    wv = _values(t[L0 + "attn.wv.weight"], dtype)
    rows = range(3, spec.kv_dim, 5)
    for i, r in enumerate(rows):
        c = (i * 37) % spec.dim
        wv[r, c] = float("inf") if i % 2 else float("-inf")
        if i % 3 == 0:  # another one of the same effect
            o = (c + 200) % spec.dim
            wv[r, o] = wv[r, c] * torch.sign(xn[c] * xn[o])
    _store(t, L0 + "attn.wv.weight", wv, dtype)
    _, _, v = _first_token(spec, t, 5)
    ref = _reference(spec, t, 5, np.zeros(spec.kv_dim))[2]
    assert np.isinf(ref[rows]).all() and (ref[rows] > 0).any() and (ref[rows] < 0).any()
    assert (v[rows] == ref[rows]).all()
    rest = np.setdiff1d(np.arange(spec.kv_dim), rows)
    assert (np.abs(v[rest] - ref[rest]) <= 2.0**-10 * np.abs(ref[rest]) + 2.0**-24).all()
