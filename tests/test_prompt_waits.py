"""Waits of the prompt products that run out: the kernel ends with a code that the host reports, with no warp split and nothing left on its way."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
from dataclasses import replace
from calm_b200 import lib, modelgen as mg
spec = replace(mg.SPECS["pf-tiny"], name="waits", dtype="%s", max_seq_len=256)
with lib.DeviceModel(spec, mg.generate(spec, seed=3), seq_len=256) as dm:
    dm.prefill(mg.teacher_tokens(spec.vocab_size, 130), 0)
print("done")
"""


def test_warps_give_up_together():
    """A lane that left a loop alone would be missing at its warp's next barrier for good."""
    src = open(os.path.join(ROOT, "calm_b200", "csrc", "prefill.cuh")).read()
    roles = src[src.index("k_pf_gemm(const __grid_constant__"):src.index("__syncthreads_or(!ok)")]
    assert "mbar_wait_warp(" in roles
    assert not re.findall(r"(?<!bar_and\(1, 128, )mbar_wait_bounded\(", roles)
    src = open(os.path.join(ROOT, "calm_b200", "csrc", "seqgemm_tc.cuh")).read()
    epilogue = src[src.index("} else {\n\t\tok = "):src.index("__syncthreads_or(!ok)")]  # the roles before it are one lane each
    assert "mbar_wait_warp(" in epilogue and "mbar_wait_bounded(" not in epilogue


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["fp16", "fp8", "gf4"])
@pytest.mark.parametrize("tries", [0, 1])  # none: no role starts; one: the rings are filled, what waits for a copy that has not landed gives up
def test_reported(dtype, tries):
    env = dict(os.environ, CALM_B200_PREFILL_WAIT=str(tries), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD % dtype], env=env, capture_output=True, text=True, timeout=300)
    gave_up = re.search(r"a wait inside a product gave up \(code 93\d\d\)", r.stdout + r.stderr)
    assert r.returncode != 0 and gave_up if tries == 0 else bool(gave_up) != ("done" in r.stdout), r.stdout + r.stderr
