"""Prompt products with more tiles than SMs whose last tiles are cut into K-slices: every product, with accumulators of hi and lo side by side (64 tokens of two
row tiles) and in one (128), from two to seven slices, the last token tile ragged; the cut that a shape is here for is asserted.  Same contract as test_prefill_gpu.py:
cache and next-token logits equal those of the serial calls."""
import ctypes as C
import os
import sys
from dataclasses import replace

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_prefill_gpu import _both, _check  # noqa: E402

from calm_b200 import lib  # noqa: E402
from calm_b200 import modelgen as mg  # noqa: E402

pytestmark = pytest.mark.gpu

SMS = 148
# dim, hidden, tokens, {product: (row tiles, tokens per item, tiles of the tail, slices)}
TAILS = [
    (2048, 2048, 804, {"qkv": (2, 64, 16, 3)}),
    (2048, 2048, 1544, {"qkv": (2, 128, 16, 2)}),
    (2048, 7168, 656, {"up": (2, 128, 40, 2)}),
    (3072, 3072, 1544, {"qkv": (2, 128, 24, 3), "wo": (2, 64, 4, 4), "up": (2, 128, 16, 3), "w2": (2, 64, 4, 4)}),
    (2048, 2048, 1174, {"up": (2, 64, 8, 3)}),
    (3072, 16512, 1589, {"wo": (2, 64, 4, 4), "up": (2, 128, 49, 3), "w2": (2, 128, 8, 7)}),
    (5120, 13824, 1990, {"qkv": (2, 128, 72, 2), "wo": (2, 128, 24, 4), "w2": (2, 128, 24, 6)}),
]


@pytest.mark.parametrize("dtype", ["fp8", "gf4", "fp16"])
@pytest.mark.parametrize("dim,hidden,n,cuts", TAILS, ids=["-".join(map(str, t[:3])) for t in TAILS])
def test_tails(dtype, dim, hidden, n, cuts):
    assert torch.cuda.get_device_properties(0).multi_processor_count == SMS
    out = (C.c_int * 5)()
    for name, product, rows, k in (("qkv", 0, 3 * dim, dim), ("wo", 1, dim, dim), ("up", 2, hidden, dim), ("w2", 1, dim, hidden)):
        lib.load().calm_b200_prefill_cut(product, rows, n, k, SMS, out)
        assert name not in cuts or tuple(out)[1:] == cuts[name], (name, tuple(out))
    spec = replace(mg.SPECS["pf-tiny"], name="tails", dtype=dtype, dim=dim, n_heads=dim // 128, n_kv_heads=dim // 128, head_dim=128, hidden_dim=hidden, max_seq_len=2048)
    tensors = mg.generate(spec, seed=6, device="cuda")
    torch.cuda.synchronize()
    toks = mg.teacher_tokens(spec.vocab_size, n + 1)
    serial, batched = _both(spec, tensors, toks, 0, 2048, 16)
    _check(spec, serial, batched, 16, f"{dtype} dim {dim} hidden {hidden}, {n} tokens")
