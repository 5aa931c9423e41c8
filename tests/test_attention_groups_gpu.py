"""Decode attention (k_attn2) for query-head groups it runs with zero queries in the spare heads, and for contexts that fill one, some or none of a
slice's steps, against the kernel it replaces (k_attn) on the same model and cache."""
import numpy as np
import pytest

from calm_b200 import lib
from calm_b200 import modelgen as mg
from dataclasses import replace

pytestmark = pytest.mark.gpu


# groups of 3, 5, 6, 7 and 12 (two units of 6), and the whole groups 2, 4 and 8
@pytest.mark.parametrize("heads,kv,hd", [(6, 2, 128), (10, 2, 64), (12, 2, 128), (14, 2, 64), (12, 1, 64), (4, 2, 64), (8, 2, 128), (8, 1, 128)])
@pytest.mark.parametrize("kvbits", [16, 8])
def test_padded_groups_and_short_contexts(heads, kv, hd, kvbits, monkeypatch):
    spec = replace(mg.SPECS["attn-l8"], name="groups", n_heads=heads, n_kv_heads=kv, head_dim=hd, dim=256)
    tensors = mg.generate(spec, seed=8)
    out = []
    for a2 in ("0", "1"):
        monkeypatch.setenv("CALM_B200_ATTN2", a2)
        with lib.DeviceModel(spec, tensors, kvbits=kvbits) as dm:
            rows = []
            for pos in (0, 15, 16, 131, 777, 1151, 2049, 4095):
                dm.fill_kv(pos, 5)
                rows.append(dm.forward(7, pos))
            out.append(np.stack(rows))
    # the same sums in another order, a few 1e-6; and where that moves an entry of layer 1 over a rounding boundary of the fp16 cache, 2^-11 of a value
    # that at position 0 is the whole output of its head
    assert np.abs(out[0] - out[1]).max() <= 1e-3 * out[0].std()
