"""How the products of a prompt are cut (calm_b200_prefill_cut) and that every cut it makes computes the same: each combination of row tiles and tokens per item
and tiles that are whole, in K-slices folded through memory, in K-slices folded inside clusters, or whole with a tail in slices that the rules pick anywhere in the range is run by one of the shapes here, in
test_prefill_tiles_gpu.py, test_prefill_tails_gpu.py or test_prefill_clusters_gpu.py."""
import ctypes as C
import os
import sys
from dataclasses import replace

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_prefill_gpu import _both, _check  # noqa: E402
from test_prefill_clusters_gpu import CLUSTERS  # noqa: E402
from test_prefill_tails_gpu import TAILS  # noqa: E402

from calm_b200 import build as cbuild  # noqa: E402
from calm_b200 import lib  # noqa: E402
from calm_b200 import modelgen as mg  # noqa: E402

SMS = 148
# dim, heads, kv heads, head_dim, hidden, tokens, and the cuts that only this shape reaches
SHAPES = [(896, 14, 2, 64, 4864, 449, {("res", 1, 128, "clusters")}), (896, 14, 2, 64, 4864, 1537, {("qkv", 2, 64, "whole"), ("res", 1, 256, "memory"), ("res", 2, 64, "whole")}),
          (768, 6, 2, 128, 2688, 1550, {("res", 2, 128, "clusters")}), (384, 3, 3, 128, 384, 1900, {("qkv", 1, 128, "whole")}), (896, 7, 7, 128, 896, 1717, {("qkv", 1, 256, "whole")}),
          (1536, 12, 12, 128, 1536, 1595, {("qkv", 2, 128, "whole"), ("res", 2, 128, "whole")}), (3072, 24, 8, 128, 6144, 67, {("up", 2, 128, "memory")}),
          (4096, 32, 32, 128, 1024, 70, {("qkv", 2, 128, "memory")}), (2048, 16, 4, 128, 2048, 73, {("qkv", 1, 64, "memory")}), (3072, 24, 12, 128, 3072, 73, {("qkv", 2, 64, "memory"), ("up", 2, 64, "memory")}),
          (3072, 24, 3, 128, 3072, 313, {("qkv", 2, 128, "clusters")}), (896, 7, 1, 128, 2304, 801, {("res", 1, 128, "memory")}), (4096, 32, 4, 128, 4096, 130, {("up", 2, 128, "clusters")})]
ELSEWHERE = [(dim, heads * hd, kv * hd, hidden, n) for dim, heads, kv, hd, hidden, n, _ in CLUSTERS] + [(dim, dim, dim, hidden, n) for dim, hidden, n, _ in TAILS] + [(384, 384, 128, 1152, 1), (896, 896, 128, 2432, 61), (1024, 1024, 256, 3456, 65), (2048, 2048, 512, 5504, 257), (4096, 4096, 1024, 14336, 130)]


@pytest.fixture(scope="module")
def cuts():
    cbuild.build()
    L, out = lib.load(), (C.c_int * 5)()

    def of(dim, q_dim, kv_dim, hidden, n):
        got = set()
        for name, product, rows, k in (("qkv", 0, q_dim + 2 * kv_dim, dim), ("res", 1, dim, q_dim), ("up", 2, hidden, dim), ("res", 1, dim, hidden)):
            L.calm_b200_prefill_cut(product, rows, n, k, SMS, out)
            tiles, na, bn, tail, sp = out
            # the accumulators fit half of TMEM; a slice is not empty; partial sums and counters of sliced products have one place per SM
            assert na in (1, 2) and bn in (64, 128, 256) and na * bn <= 256 and (name != "up" or na == 2) and 1 <= sp <= k // 64
            assert tiles == (rows // 128 if name == "up" else -(-rows // 128 // na)) * -(-n // bn) and tail * sp <= SMS and (tail == 0) == (sp == 1) and tail in (0, tiles, tiles % SMS)
            got.add((name, na, bn, "whole" if tail == 0 else "tail" if tail != tiles else "clusters" if L.calm_b200_prefill_clusters(product, rows, n, k, SMS) else "memory"))
        return got

    return of


def test_every_cut_is_run_by_a_test(cuts):
    run = set()
    for s in ELSEWHERE:
        run |= cuts(*s)
    for dim, heads, kv, hd, hidden, n, only in SHAPES:
        here = cuts(dim, heads * hd, kv * hd, hidden, n)
        assert only <= here
        run |= here
    picked = set()
    for dim in (384, 512, 768, 896, 1024, 1536, 2048, 3072, 4096, 5120, 8192):
        for kv in {max(128, dim // f // 128 * 128) for f in (1, 2, 4, 8)}:
            for hidden in {max(128, int(dim * f) // 128 * 128) for f in (1, 1.5, 2, 2.7, 3.5, 5.4)}:
                for n in list(range(1, 130, 9)) + list(range(130, 2049, 61)):
                    picked |= cuts(dim, dim, kv, hidden, n)
    assert picked <= run, sorted(picked - run)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["fp8", "gf4", "fp16"])
@pytest.mark.parametrize("dim,heads,kv,hd,hidden,n", [s[:6] for s in SHAPES])
def test_cuts(dtype, dim, heads, kv, hd, hidden, n):
    assert torch.cuda.get_device_properties(0).multi_processor_count == SMS
    spec = replace(mg.SPECS["pf-tiny"], name="cuts", dtype=dtype, dim=dim, n_heads=heads, n_kv_heads=kv, head_dim=hd, hidden_dim=hidden, max_seq_len=2048)
    tensors = mg.generate(spec, seed=6, device="cuda")
    torch.cuda.synchronize()
    serial, batched = _both(spec, tensors, mg.teacher_tokens(spec.vocab_size, n + 1), 0, 2048, 16)
    _check(spec, serial, batched, 16, f"{dtype} dim {dim} hidden {hidden}, {n} tokens")
