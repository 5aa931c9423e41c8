"""The tensor-core matvecs of a token (cols.cuh) against the CPU oracle: rows that fill part of the warps, of one piece and of several with a shorter last one, tiles
of rows that end early, one row a CTA, hidden vectors whose values outgrow the scale of the first piece, and what keeps the general kernels."""
from dataclasses import replace

import numpy as np
import pytest
import torch
from conftest import TOL_SIGMA

from calm_b200 import lib
from calm_b200 import modelgen as mg

pytestmark = pytest.mark.gpu

BASE = mg.SPECS["pf-tiny-hd128"]
# dim, hidden, heads, kv heads, head_dim -> (pieces of a dim row in fp8, in fp16; tiles of wo and w2)
SHAPES = {
    "part of the warps": (896, 1152, 14, 2, 64, (1, 1, 1)),
    "two pieces, the last one short": (1152, 4864, 9, 3, 128, (1, 2, 1)),
    "odd rows": (2176, 2432, 17, 1, 128, (2, 3, 2)),
    "one row a CTA": (128, 128, 2, 1, 64, (1, 1, 1)),
    "three tiles": (3072, 1536, 24, 8, 128, (2, 3, 3)),
}


def _plan():
    return [lib.load().calm_b200_token_plan(s) for s in range(4)]


def _compare(oracle_pkg, spec, host, plan, n=12):
    toks = mg.teacher_tokens(spec.vocab_size, n)
    ck = oracle_pkg.Checker("port")
    ref = oracle_pkg.teacher_forced(ck, host, toks)
    with lib.DeviceModel(spec, host.tensors) as dm:
        got_plan = _plan()
        got = np.stack([dm.forward(t, i) for i, t in enumerate(toks)])
    ck.release(host)
    assert got_plan == plan
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= TOL_SIGMA * ref.std()


@pytest.mark.parametrize("dtype", ["fp8", "fp16"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_token_products_vs_oracle(oracle_pkg, shape, dtype):
    dim, hidden, heads, kv, hd, (c8, c16, tiles) = SHAPES[shape]
    spec = replace(BASE, name=shape, dtype=dtype, dim=dim, hidden_dim=hidden, n_heads=heads, n_kv_heads=kv, head_dim=hd, n_layers=2, qkv_bias=shape == "part of the warps")
    c = c8 if dtype == "fp8" else c16
    _compare(oracle_pkg, spec, mg.HostModel(spec, seed=5), [c, tiles, c, tiles])


@pytest.mark.parametrize("dtype", ["fp8", "fp16"])
def test_hidden_vector_outgrows_its_first_pieces_scale(oracle_pkg, dtype):
    """w3's rows grow by 2^16 along the hidden vector: every piece of w2's input is about four times the one before."""
    spec = replace(BASE, name="grow", dtype=dtype, dim=512, hidden_dim=8192 if dtype == "fp16" else 16384, n_heads=4, n_kv_heads=2, n_layers=2)
    t = mg.generate(spec, 9)
    by = torch.exp2(torch.linspace(0, 16, spec.hidden_dim).floor())[:, None]
    for l in range(spec.n_layers):
        name = f"model.layers.{l}.mlp.w3.weight"
        kind = torch.float16 if dtype == "fp16" else torch.float8_e5m2
        t[name] = (t[name].view(kind).float() * by).to(kind).view(t[name].dtype)
    _compare(oracle_pkg, spec, mg.HostModel(spec, tensors=t), [1, 1, 1, 1])


@pytest.mark.parametrize("change, plan", [({"norm_type": "layernorm"}, [0, 1, 0, 1]), ({"norm_type": "layernorm_par"}, [0, 1, 1, 1]), ({"dtype": "gf4"}, [0, 0, 0, 0]), ({"hidden_dim": 1056}, [1, 1, 1, 0])])
def test_stages_that_keep_the_general_kernels(oracle_pkg, change, plan):
    spec = replace(BASE, name="general", dim=512, hidden_dim=1024, n_heads=4, n_kv_heads=2, n_layers=2, **{"dtype": "fp8", **{k: v for k, v in change.items() if k != "hidden_dim"}})
    spec = replace(spec, **{k: v for k, v in change.items() if k == "hidden_dim"})
    _compare(oracle_pkg, spec, mg.HostModel(spec, seed=5), plan)
