"""One token's gate attention where the ranges of keys change: part of a run of four keys, one run, a whole tile, several tiles, and
the new key at the start and the end of each; heads and widths that no lane count divides.  The prompt path in 32 bits is the
reference: both compute in fp32, in another order."""
import numpy as np
import pytest

from tests import layered_util as U
from tests.test_gpu_gate_routes import attention_only, load  # noqa: F401

pytestmark = pytest.mark.gpu


def steps_against_a_prompt(load, layer, seed, edges, dtype, tol):  # noqa: F811
    cfg = U.config(64, 60, 1e-5, [layer])
    w = attention_only(U.weights(cfg, seed=seed))
    n = edges[-1] + 1
    toks = U.tokens(cfg, n)
    ref = load(cfg, w, "float32", n).Forward(toks, 0, edges)
    e = load(cfg, w, dtype, n)
    got, at = [], 0
    for p in edges:
        if p > at:
            e.Forward(toks[at:p], at, ())
        got.append(e.Forward(toks[p:p + 1], p, (0,)))
        at = p + 1
    err = U.rel(np.concatenate(got), ref)
    assert err.max() < tol, (edges[int(err.argmax())], float(err.max()))


# 147 CTAs attend: ranges of 4 keys up to 588, of 8 up to 1176, of 12 (three quarters of a tile) up to 1764
EDGES = (0, 1, 2, 3, 4, 5, 7, 8, 586, 587, 588, 589, 592, 1175, 1176, 1177, 1180, 1184, 1764)


@pytest.mark.parametrize("heads,kv,dim", [(1, 1, 8), (3, 1, 15), (14, 2, 64), (32, 4, 64), (7, 7, 136), (40, 8, 24), (33, 33, 200)])
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-4), ("bfloat16", 1e-2)])
def test_steps_where_ranges_change(load, heads, kv, dim, dtype, tol):  # noqa: F811
    steps_against_a_prompt(load, U.layer(heads, kv, dim, 0.8 / dim, 0.4, 50, 1, 16, 16, 6.0, 48), heads + dim, EDGES, dtype, tol)


# With 120 memory heads 32 CTAs attend: ranges of 4 keys up to 128, ..., of 16 (a whole tile) up to 512, of 20 (a tile and a part) beyond, of 32 up to 1024, of
# 36 (three tiles) up to 1152, of 64 up to 2048, of 68 beyond; four lanes share a score up to 192 of a tile, a lane has one beyond
LONG_EDGES = (0, 1, 4, 127, 128, 129, 255, 256, 257, 383, 384, 511, 512, 513, 1023, 1024, 1025, 1055, 1056, 1151, 1152, 1153, 2047, 2048, 2049)


@pytest.mark.parametrize("heads,kv,dim", [(1, 1, 8), (3, 1, 15), (8, 2, 64), (9, 3, 40), (32, 4, 64), (33, 33, 48)])
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-4), ("bfloat16", 1e-2)])
def test_steps_with_many_keys_per_cta(load, heads, kv, dim, dtype, tol):  # noqa: F811
    steps_against_a_prompt(load, U.layer(heads, kv, dim, 0.8 / dim, 0.4, 50, 120, 8, 8, 6.0, 48), heads + dim, LONG_EDGES, dtype, tol)
