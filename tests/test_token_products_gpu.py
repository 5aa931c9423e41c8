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


def _compare(oracle_pkg, spec, host, plan, n=12, rings=None):
    toks = mg.teacher_tokens(spec.vocab_size, n)
    ck = oracle_pkg.Checker("port")
    ref = oracle_pkg.teacher_forced(ck, host, toks)
    with lib.DeviceModel(spec, host.tensors) as dm:
        got_plan, got_rings = _plan(), [lib.load().calm_b200_token_plan(s) > 0 for s in (5, 6, 7)]
        got = np.stack([dm.forward(t, i) for i, t in enumerate(toks)])
    ck.release(host)
    assert got_plan == plan and rings in (None, got_rings)
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= TOL_SIGMA * ref.std()


@pytest.mark.parametrize("dtype", ["fp8", "fp16"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_token_products_vs_oracle(oracle_pkg, shape, dtype):
    dim, hidden, heads, kv, hd, (c8, c16, tiles) = SHAPES[shape]
    spec = replace(BASE, name=shape, dtype=dtype, dim=dim, hidden_dim=hidden, n_heads=heads, n_kv_heads=kv, head_dim=hd, n_layers=2, qkv_bias=shape == "part of the warps")
    c = c8 if dtype == "fp8" else c16
    _compare(oracle_pkg, spec, mg.HostModel(spec, seed=5), [c, tiles, c, tiles])


# The widest rows and most tiles, each with a last piece or tile that is partly filled, and what lies behind them (stages 5 and 6: rings of rows that are whole kilobytes, where there are any)
WIDE = [("fp16", 4096, 1152, [4, 4, 4, 4]), ("fp8", 4096, 1152, [2, 4, 2, 4]), ("fp8", 6272, 2304, [4, 6, 4, 6]), ("fp16", 6272, 2304, [7, 6, 7, 6]), ("fp8", 5248, 1152, [3, 5, 3, 5]),
        ("fp16", 5248, 1152, [6, 5, 6, 5]), ("fp16", 4608, 1152, [5, 4, 5, 4]), ("fp8", 8192, 1152, [4, 7, 4, 7]), ("fp16", 8192, 1152, [8, 7, 8, 7]), ("fp8", 8320, 1152, [0, 8, 0, 8]),
        ("fp16", 9344, 1152, [0, 8, 0, 8]), ("fp8", 10240, 2048, [0, 0, 0, 0]), ("fp16", 10240, 2048, [0, 0, 0, 0])]


@pytest.mark.parametrize("dtype,dim,hidden,plan", WIDE)
def test_wide_rows(oracle_pkg, dtype, dim, hidden, plan):
    spec = replace(BASE, name="wide", dtype=dtype, dim=dim, hidden_dim=hidden, n_heads=8, n_kv_heads=1, n_layers=1, vocab_size=256, qkv_bias=False)
    _compare(oracle_pkg, spec, mg.HostModel(spec, seed=5), plan, n=4, rings=[1, 1, 1] if dim == 10240 else None)


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


@pytest.mark.parametrize("change, plan", [({"norm_type": "layernorm"}, [0, 1, 0, 1]), ({"norm_type": "layernorm_par"}, [0, 1, 1, 1]), ({"norm_type": "rmsnorm_par"}, [1, 1, 1, 1]), ({"dtype": "gf4"}, [0, 0, 0, 0]), ({"hidden_dim": 1056}, [1, 1, 1, 0])])
def test_stages_that_keep_the_general_kernels(oracle_pkg, change, plan):
    spec = replace(BASE, name="general", dim=512, hidden_dim=1024, n_heads=4, n_kv_heads=2, n_layers=2, **{"dtype": "fp8", **{k: v for k, v in change.items() if k != "hidden_dim"}})
    spec = replace(spec, **{k: v for k, v in change.items() if k == "hidden_dim"})
    _compare(oracle_pkg, spec, mg.HostModel(spec, seed=5), plan)
