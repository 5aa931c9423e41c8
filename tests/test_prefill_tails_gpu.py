"""Prompt products with more tiles than SMs whose last tiles are cut into K-slices: every product, with accumulators of hi and lo side by side (64 tokens of two
row tiles) and in one (128), the last token tile ragged.  Same contract as test_prefill_gpu.py: cache and next-token logits equal those of the serial calls."""
import os
import sys
from dataclasses import replace

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_prefill_gpu import _both, _check  # noqa: E402

from calm_b200 import modelgen as mg  # noqa: E402

pytestmark = pytest.mark.gpu


# tails of 148 SMs: q/k/v 16 tiles of 64 tokens in 3 slices; q/k/v 16 of 128 in 2; FFN up 40 of 128 in 2; wo and w2 4 of 64 in 4, FFN up at 64 in the last two
@pytest.mark.parametrize("dtype", ["fp8", "gf4", "fp16"])
@pytest.mark.parametrize("dim,hidden,n", [(2048, 2048, 804), (2048, 2048, 1544), (2048, 7168, 656), (3072, 3072, 1544), (2048, 2048, 1174)])
def test_tails(dtype, dim, hidden, n):
    spec = replace(mg.SPECS["pf-tiny"], name="tails", dtype=dtype, dim=dim, n_heads=dim // 128, n_kv_heads=dim // 128, head_dim=128, hidden_dim=hidden, max_seq_len=2048)
    toks = mg.teacher_tokens(spec.vocab_size, n + 1)
    serial, batched = _both(spec, mg.generate(spec, seed=6), toks, 0, 2048, 16)
    _check(spec, serial, batched, 16, f"{dtype} dim {dim} hidden {hidden}, {n} tokens")
