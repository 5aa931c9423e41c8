"""Prompt products whose slices are folded inside a thread-block cluster: every product and weight format, two to eight slices, fewer tokens than slices (CTAs without
a share), shares that are no multiple of the four tokens a thread takes, two token tiles with a ragged last one; the cut that a shape is here for is asserted.  Same contract
as test_prefill_gpu.py: cache and next-token logits equal those of the serial calls."""
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
MOST = {2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 7: 15, 8: 15}  # clusters of a size at a time
# dim, q heads, kv heads, head_dim, hidden, tokens, {product: slices}
CLUSTERS = [
    (896, 14, 2, 64, 4864, 61, {"qkv": 7, "wo": 7, "up": 3, "w2": 8}),
    (896, 14, 2, 64, 4864, 3, {"qkv": 7, "wo": 7, "up": 3, "w2": 8}),
    (896, 14, 2, 64, 4864, 130, {"qkv": 4, "wo": 6, "w2": 6}),
    (1024, 8, 2, 128, 2688, 65, {"qkv": 5, "wo": 6, "up": 3, "w2": 6}),
    (1152, 9, 3, 128, 2816, 40, {"qkv": 8, "wo": 8, "up": 6, "w2": 8}),
    (2560, 20, 4, 128, 2560, 100, {"qkv": 2, "wo": 3, "up": 3, "w2": 3}),
    (640, 5, 1, 128, 1664, 64, {"qkv": 5, "wo": 5, "up": 5, "w2": 8}),
]


@pytest.mark.parametrize("dtype", ["fp8", "gf4", "fp16"])
@pytest.mark.parametrize("dim,heads,kv,hd,hidden,n,cuts", CLUSTERS, ids=["-".join(map(str, t[:6])) for t in CLUSTERS])
def test_slices_in_clusters(dtype, dim, heads, kv, hd, hidden, n, cuts):
    assert torch.cuda.get_device_properties(0).multi_processor_count == SMS
    out = (C.c_int * 5)()
    for name, product, rows, k in (("qkv", 0, (heads + 2 * kv) * hd, dim), ("wo", 1, dim, heads * hd), ("up", 2, hidden, dim), ("w2", 1, dim, hidden)):
        lib.load().calm_b200_prefill_cut(product, rows, n, k, SMS, out)
        tiles, _, _, tail, splits = out
        if name in cuts:
            assert tail == tiles <= MOST[splits] and splits == cuts[name], (name, tuple(out))
    spec = replace(mg.SPECS["pf-tiny"], name="clusters", dtype=dtype, dim=dim, n_heads=heads, n_kv_heads=kv, head_dim=hd, hidden_dim=hidden, max_seq_len=512)
    tensors = mg.generate(spec, seed=6, device="cuda")
    torch.cuda.synchronize()
    serial, batched = _both(spec, tensors, mg.teacher_tokens(spec.vocab_size, n + 1), 0, 512, 16)
    _check(spec, serial, batched, 16, f"{dtype} dim {dim} hidden {hidden}, {n} tokens")
