"""The prompt pass clears its buffers in its own stream: another stream's work (here: the default stream's, still running) decides neither when they are cleared nor
what a first or a longer prompt reads."""
from dataclasses import replace

import numpy as np
import pytest
import torch

from calm_b200 import lib
from calm_b200 import modelgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(61,), (40, 200)])  # a first prompt; one that outgrows the buffers
def test_default_stream_busy(lengths):
    spec = replace(mg.SPECS["pf-tiny"], name="buffers", dim=512, n_heads=4, n_kv_heads=2, head_dim=128, hidden_dim=1024, max_seq_len=512)  # small: K is cut into slices
    tensors = mg.generate(spec, seed=5)
    got = []
    for busy in (False, True):
        with lib.DeviceModel(spec, tensors, seq_len=512) as dm:
            pos = 0
            for n in lengths:
                if busy:
                    torch.cuda._sleep(100_000_000)  # some 50 ms
                assert dm.prefill(mg.teacher_tokens(spec.vocab_size, n, start=pos), pos) == 1
                pos += n
            torch.cuda.synchronize()
            got.append((dm.forward(7, pos), *[x for p in (0, 17, pos - 1) for x in dm.read_kv(spec.n_layers - 1, p)]))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
