"""Both kernels of the bf16 gate attention: heads and key heads on either side of the rule between them, every
width of the kernel that mixes pairs, and blocks of queries that its workspace cuts.

The memory beside the attention is scaled to nothing: where its denominators pass near zero, the rounding of
its bf16 inputs grows tenfold, whichever kernel attends.  What is left are three products of operands rounded to
bf16 (2^-9 of an operand, at random) one behind the other: 4e-3 of the logits at most over these shapes."""
import numpy as np
import pytest

from tests import layered_util as U

pytestmark = pytest.mark.gpu

TOL = 1e-2
# heads, key heads, dim: one head at a time with one and two groups of columns, pairs of up to 4, 8, 16 and 32 heads
SHAPES = [(8, 2, 64), (8, 8, 64), (20, 20, 12), (32, 32, 16), (3, 3, 128), (6, 6, 128), (7, 7, 120), (12, 12, 64), (20, 20, 40), (32, 16, 96), (17, 17, 33)]


@pytest.fixture
def load(cuda, mglib, tmp_path):
    from mongoose_b200 import registry
    made = []

    def make(cfg, w, dtype, max_seq):
        path = str(tmp_path / str(len(made)))
        U.write_folder(path, cfg, w)
        made.append(registry.load_model(path, dtype=dtype, max_seq=max_seq))
        return made[-1]

    yield make
    for e in made:
        e.close()


def attention_only(w):
    w["l0.mix.right.out"][:] = 0
    return w


@pytest.mark.parametrize("heads,kv,dim", SHAPES)
def test_routes_agree_with_the_oracle(load, heads, kv, dim):
    cfg = U.config(72, 60, 1e-5, [U.layer(heads, kv, dim, 0.8 / dim, 0.4, 50, 1, 16, 16, 6.0, 48)])
    w = attention_only(U.weights(cfg, seed=heads + dim))
    toks = U.tokens(cfg, 290)
    ref = U.want(cfg, w, toks)
    e = load(cfg, w, "bfloat16", 290)
    for cuts in ([290], [3, 130, 157], [128, 162], [97, 31, 162]):
        got, at = [], 0
        for n in cuts:
            got.append(e.Forward(toks[at:at + n], at, range(n)))
            at += n
        err = U.rel(np.concatenate(got), ref)
        assert err.max() < TOL, (cuts, int(err.argmax()), float(err.max()))


# a portion of 2048 rows in blocks of 1920 and 1792 queries, and few heads far back
@pytest.mark.parametrize("heads,kv,dim,max_seq,edges", [(32, 32, 24, 2176, (1919, 1920, 1921)), (32, 32, 136, 2304, (1791, 1792, 1793)), (3, 1, 64, 2176, ())])
def test_blocks_of_queries_and_long_contexts(load, heads, kv, dim, max_seq, edges):
    cfg = U.config(64, 90, 1e-5, [U.layer(heads, kv, dim, 0.8 / dim, 0.3, 300, 1, 16, 16, 8.0, 0)])
    w = attention_only(U.weights(cfg, seed=41))
    n = 2175
    toks = U.tokens(cfg, n)
    places = sorted({0, 700, *edges, 2046, 2047, 2048, 2049, n - 1})
    a, b = load(cfg, w, "float32", max_seq), load(cfg, w, "bfloat16", max_seq)
    ref = a.Forward(toks, 0, places)
    assert U.rel(b.Forward(toks, 0, places), ref).max() < TOL
    got, at = [], 0
    for k in (1500, 100, 575):                  # portions behind a long context
        got.append(b.Forward(toks[at:at + k], at, [p - at for p in places if at <= p < at + k]))
        at += k
    assert U.rel(np.concatenate(got), ref).max() < TOL
