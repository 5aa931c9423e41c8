"""The greedy pick (k_seq_argmax) at vocabularies that are whole float4s and that are not, below and above what a CTA reads in one round, with the largest logit
more than once; and embedding rows of widths that allow 16-byte pieces and that do not."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_bovinex_gpu as tb  # noqa: E402
import bovinex_plain  # noqa: E402

from calm_b200 import bovinex  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,width", [(8, 48), (97, 44), (4096, 40), (4101, 50), (16384, 264), (20004, 48)])
def test_first_of_the_largest(vocab, width):
    cfg = tb.config([tb.gla()], width=width, vocab=vocab)
    t, toks = tb.weights(cfg, 4), tb.tokens(cfg, 21)
    ref = bovinex_plain.forward(cfg, tb.as_f64(t), toks)
    top = int(ref[-1].argmax())
    for other in (0, 3, vocab // 2, vocab - 1):  # the last token's largest logit several times
        t["head"][other] = t["head"][top]
    with bovinex.from_tensors(cfg, t, "float32", max_tokens=64, max_seqs=1, page=8) as m:
        got = m.step([m.open()], [toks], list(range(21)))
        pick = m.argmax(21)
    assert (pick == got.argmax(-1)).all()  # numpy takes the first one too
    ref = bovinex_plain.forward(cfg, tb.as_f64(t), toks)
    assert tb.rel_err(got, ref) < tb.TOL["float32"] and np.isclose(ref[-1][pick[-1]], ref[-1].max())
