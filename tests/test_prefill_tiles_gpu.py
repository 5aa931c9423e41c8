"""The prompt pass at the edges of its tiles: head groups that divide over the warps of an attention CTA in different ways, prompts around
multiples of the 16-row and 64-key tiles, a block behind a cached prefix.  Same contract as test_prefill_gpu.py: cache and next-token logits
equal those of the serial calls."""
import os
import sys
from dataclasses import replace

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_prefill_gpu import _both, _check  # noqa: E402

from calm_b200 import modelgen as mg  # noqa: E402

pytestmark = pytest.mark.gpu


# (query heads, kv heads, head_dim): groups of 1, 2, 4, 7, 8, 12 (6 heads per CTA) and 16 (8 per CTA)
@pytest.mark.parametrize("heads,kv,hd", [(2, 2, 128), (4, 2, 64), (8, 2, 128), (14, 2, 64), (8, 1, 128), (12, 1, 128), (16, 1, 128)])
@pytest.mark.parametrize("n,pos0,kvbits", [(2, 0, 16), (65, 0, 8), (144, 63, 16)])
def test_attention_groups_and_edges(heads, kv, hd, n, pos0, kvbits):
    spec = replace(mg.SPECS["pf-tiny"], name="edge", dim=256, n_heads=heads, n_kv_heads=kv, head_dim=hd, hidden_dim=512, max_seq_len=256)
    toks = mg.teacher_tokens(spec.vocab_size, n + 1)
    serial, batched = _both(spec, mg.generate(spec, seed=4), toks, pos0, 256, kvbits, warm=mg.teacher_tokens(spec.vocab_size, pos0, start=500))
    _check(spec, serial, batched, kvbits, f"heads {heads}/{kv}x{hd}, {n} at {pos0}, kv{kvbits}")


# Products: one and two row tiles per item (an odd number of row tiles leaves a single one), 64 tokens per tile and in FFN up 128, with ragged last tiles, K cut
# into slices (small models) and not, many items per CTA, all three weight formats; the other cuts are in test_prefill_choice.py.  The cache after two layers sees
# every product.
@pytest.mark.parametrize("dtype", ["fp8", "gf4", "fp16"])
@pytest.mark.parametrize("dim,heads,kv,hidden,n", [(384, 3, 1, 1152, 1), (896, 7, 1, 2432, 61), (1024, 8, 2, 3456, 65), (2048, 16, 4, 5504, 257), (4096, 32, 8, 14336, 130)])
def test_product_tiles(dtype, dim, heads, kv, hidden, n):
    spec = replace(mg.SPECS["pf-tiny"], name="tiles", dtype=dtype, dim=dim, n_heads=heads, n_kv_heads=kv, head_dim=128, hidden_dim=hidden, max_seq_len=512)
    toks = mg.teacher_tokens(spec.vocab_size, n + 1)
    serial, batched = _both(spec, mg.generate(spec, seed=6), toks, 0, 512, 16)
    _check(spec, serial, batched, 16, f"{dtype} dim {dim} hidden {hidden}, {n} tokens")
