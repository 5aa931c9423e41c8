"""Waits of the layer-list products on pairs of CTAs (k_seq_gemm_pair) that run out: the kernel ends with a code that the host reports, with no warp split and
nothing left on its way into the shared memory of a CTA that has ended."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path.insert(0, "tests")
import test_bovinex_gpu as tb
from calm_b200 import bovinex
cfg = tb.config([tb.attn(mlp={"ff": 2000, "kind": "dense"})], width=2048)
with bovinex.from_tensors(cfg, tb.weights(cfg, 6), "bfloat16", max_tokens=400, max_seqs=1, page=8) as m:
    m.step([m.open()], [tb.tokens(cfg, 200)], [199])
print("done")
"""


def test_both_ctas_wait_for_what_arrives_in_them():
    """A release or a hand-over of the MMAs arrives on a barrier of either CTA: an arrival at a CTA that has ended would be an access to memory that is gone."""
    src = open(os.path.join(ROOT, "calm_b200", "csrc", "seqgemm_tc.cuh")).read()
    kernel = src[src.index("k_seq_gemm_pair(const __grid_constant__"):]
    roles, end = kernel[:kernel.index("__syncthreads_or(!ok)")], kernel[kernel.index("__syncthreads_or(!ok)"):kernel.index("pair_tmem_dealloc")]
    assert "mbar_wait_bounded(" not in roles  # whole warps give up
    assert len(re.findall(r"mbar_wait_warp\(&\w+\[", roles)) == len(re.findall(r"mbar_wait_warp\(&\w+\[.*?, tries\)", roles)) == 5
    assert not re.search(r"if \([^\n]*rank == 0 &&", end)  # both CTAs wait, whichever of them gave up
    for bar in ("full", "empty", "acc_full"):
        assert f"mbar_wait_bounded(&{bar}[" in end
    assert "gave_up_s[0]" in end and "gave_up_s[1]" in end
    copies = roles[roles.index("pair_tma_load_2d"):roles.index("} else if (warp == 1)")]
    assert copies.index("mbar_wait_warp(&empty") < copies.index("atomicExch(err")  # a release that never came is reported too


@pytest.mark.gpu
@pytest.mark.parametrize("tries", [0, 1])  # none: no role starts; one: the ring is filled, what waits for a copy that has not landed gives up
def test_reported(tries):
    env = dict(os.environ, CALM_B200_SEQ_WAIT=str(tries), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    gave_up = re.search(r"product pipeline stalled \(code [1-4]\)", r.stdout + r.stderr)
    assert r.returncode != 0 and gave_up if tries == 0 else bool(gave_up) != ("done" in r.stdout), r.stdout + r.stderr
