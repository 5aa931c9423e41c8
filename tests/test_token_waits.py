"""Waits of a token's tensor-core matvecs (cols.cuh) that run out: whichever role gives up, the kernel ends with a code that the host reports, with no warp split and
nothing left on its way into the shared memory of a CTA that has ended."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# 512 x 1024: a CTA's copying warps have requested all of their stages before the first is used
CHILD = """
from dataclasses import replace
from calm_b200 import lib, modelgen as mg
spec = replace(mg.SPECS["pf-tiny-hd128"], name="waits", dtype="%s", dim=%d, hidden_dim=%d, n_layers=2)
with lib.DeviceModel(spec, mg.generate(spec, seed=3)) as dm:
    assert all(lib.load().calm_b200_token_plan(s) for s in range(4))
    dm.forward(5, 0)
print("done")
"""


def test_copies_end_before_their_cta_whichever_role_gave_up():
    """A multiplying warp can give up on a stage behind which the copying warps have nothing left to request: they wait for what they requested in any case."""
    src = open(os.path.join(ROOT, "calm_b200", "csrc", "cols.cuh")).read()
    assert "mbar_wait_bounded(" not in src  # whole warps give up
    produce = src[src.index("void cols_produce("):]
    produce = produce[:produce.index("\n}\n")]
    loop, end = produce[:produce.index("\n\t}\n")], produce[produce.index("\n\t}\n") + 4:]
    assert "return" not in produce and "break" in loop
    drain = re.search(r"for \(int k = i - 2; k >= max\(0, i - COLS_STAGES\); k -= 2\) mbar_wait_warp\(&sh->full\[k % COLS_STAGES\], \(k / COLS_STAGES\) & 1\);", end)
    assert drain and not re.search(r"\bif\b(?! \(!waited\))", end)
    for kernel in ("k_qkv_cols", "k_ffn_up_cols", "k_matres_cols"):
        body = src[src.index(kernel + "(const"):]
        body = body[:body.index("\n}\n")]
        assert body.index("cols_produce(") < body.index("cols_epilogue(") < body.index("\n\t__syncthreads();") < body.index("r.err) = sh.gave_up")
        assert not re.search(r"\n\t{1,3}return;", body)  # every thread comes to the end


def test_a_wait_gives_up_within_seconds():
    """A try of mbarrier.try_wait that does not succeed takes 3.95 us on a B200."""
    src = open(os.path.join(ROOT, "calm_b200", "csrc", "tc05.cuh")).read()
    assert 1 <= (1 << int(re.search(r"#define MBAR_SPINS \(1u << (\d+)\)", src).group(1))) * 3.95e-6 <= 10


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,dim,hidden", [("fp8", 512, 1024), ("fp16", 512, 1024), ("fp8", 2048, 8192), ("fp16", 2048, 8192)])
@pytest.mark.parametrize("tries", [0, 1])  # none: no role gets a stage; one: the ring is filled, what waits for a copy that has not landed gives up
def test_reported(dtype, dim, hidden, tries):
    env = dict(os.environ, CALM_B200_TOKEN_WAIT=str(tries), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD % (dtype, dim, hidden)], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    gave_up = re.search(r"a wait inside a matvec of a token gave up \(code 94\d\d\)", r.stdout + r.stderr)
    assert r.returncode != 0 and gave_up if tries == 0 else bool(gave_up) != ("done" in r.stdout), r.stdout + r.stderr
