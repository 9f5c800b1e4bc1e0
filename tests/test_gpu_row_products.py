"""One token's products with bf16 matrices, at the sizes where rows are dealt to threads in another way.

Rows of up to 512 and 1024 columns are shared by 64 and 128 threads, longer ones by 256; a thread holds one chunk of
eight columns of up to 2048 and three of longer rows, and fetches again beyond 6144; a CTA takes one to
eight rows at a time and, in a vocabulary, several times.
"""
import numpy as np
import pytest

from mongoose_b200 import registry
from tests import layered_util as U

pytestmark = pytest.mark.gpu


def one(width, ff, vocab, heads=2, dim=16):
    return U.config(width, vocab, 1e-5, [U.layer(heads, 1, dim, 0.25, 0.3, 9, 1, 16, 16, 5.0, ff)])


CASES = {
    "512": one(512, 520, 300), "576": one(576, 1024, 75), "1088": one(1088, 2048, 149), "2112": one(2112, 2176, 40),
    "6144": one(64, 6144, 40), "6208": one(64, 6208, 40), "16448": one(48, 16448, 40), "33000": one(48, 33000, 40),
    "vocab": one(40, 64, 148 * 256 + 300), "vocab2": one(64, 64, 148 * 512 + 5),
}


@pytest.mark.parametrize("name", list(CASES))
def test_tokens_one_by_one(cuda, mglib, tmp_path, name):
    cfg = CASES[name]
    w = U.weights(cfg, 3)
    toks = U.tokens(cfg, 5)
    U.write_folder(str(tmp_path), cfg, w)
    e = registry.load_model(str(tmp_path), dtype="float32", max_seq=16)
    try:
        got = np.stack([e.Forward(toks[i:i + 1], i, (0,))[0] for i in range(len(toks))])
        ref = U.want(cfg, w, toks)
        assert U.rel(got, ref).max() < 3e-5
        e.StepToken(int(toks[0]), 0)
        assert e.GetCursor() == (int(np.argmax(ref[0])), 1)
    finally:
        e.close()
