"""One token's gate attention where the ranges of keys change: part of a run of four keys, one run, a whole tile, several tiles, and
the new key at the start and the end of each; heads and widths that no lane count divides.  The prompt path in 32 bits is the
reference: both compute in fp32, in another order."""
import numpy as np
import pytest

from tests import layered_util as U
from tests.test_gpu_gate_routes import attention_only, load  # noqa: F401

pytestmark = pytest.mark.gpu

# 147 CTAs attend: ranges of 4 keys up to 588, of 8 up to 1176, of 12 (a tile and a half) up to 1764
EDGES = (0, 1, 2, 3, 4, 5, 7, 8, 586, 587, 588, 589, 592, 1175, 1176, 1177, 1180, 1184, 1764)


@pytest.mark.parametrize("heads,kv,dim", [(1, 1, 8), (3, 1, 15), (14, 2, 64), (32, 4, 64), (7, 7, 136), (40, 8, 24), (33, 33, 200)])
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-4), ("bfloat16", 1e-2)])
def test_steps_where_ranges_change(load, heads, kv, dim, dtype, tol):  # noqa: F811
    cfg = U.config(64, 60, 1e-5, [U.layer(heads, kv, dim, 0.8 / dim, 0.4, 50, 1, 16, 16, 6.0, 48)])
    w = attention_only(U.weights(cfg, seed=heads + dim))
    n = EDGES[-1] + 1
    toks = U.tokens(cfg, n)
    ref = load(cfg, w, "float32", n).Forward(toks, 0, EDGES)
    e = load(cfg, w, dtype, n)
    got, at = [], 0
    for p in EDGES:
        if p > at:
            e.Forward(toks[at:p], at, ())
        got.append(e.Forward(toks[p:p + 1], p, (0,)))
        at = p + 1
    err = U.rel(np.concatenate(got), ref)
    assert err.max() < tol, (EDGES[int(err.argmax())], float(err.max()))
