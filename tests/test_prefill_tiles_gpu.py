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
