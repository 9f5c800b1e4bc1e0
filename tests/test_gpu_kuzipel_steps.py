"""One token of Kuzipel models where its kernels change their split: chosen experts' rows two, four and five at a time, over
one and two turns of columns, runs that cross from expert to expert; ranges of cached latents of part of a run, a run, a tile
and more.  The prompt path in 32 bits is the reference: both compute in fp32, in another order."""
import numpy as np
import pytest

from tests import kuzipel_util as U
from tests.test_gpu_kuzipel import load  # noqa: F401

pytestmark = pytest.mark.gpu


def steps_against_a_prompt(load, cfg, seed, edges, dtype, tol):  # noqa: F811
    w = U.weights(cfg, seed=seed, steady=True)
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


# width, experts, top, ff: on 148 SMs two rows at a time, five (ten on a CTA), four, three turns over wide rows, many short experts
@pytest.mark.parametrize("width,experts,top,ff", [(64, 5, 2, 33), (1088, 5, 4, 704), (1088, 4, 2, 592), (2112, 4, 3, 470), (528, 6, 4, 301), (320, 24, 17, 3)])
def test_chosen_rows(load, width, experts, top, ff):  # noqa: F811
    cfg = U.config(width, 41, 1e-5, [U.layer(U.wkv(2, 16, 8), U.moe(experts, top, ff, 48))])
    steps_against_a_prompt(load, cfg, ff, (0, 1, 2, 5), "float32", 1e-4)


# 148 CTAs of a range each (74 for 40 heads): ranges of 4 rows up to 592, of 8 up to 1184, of 12 beyond
@pytest.mark.parametrize("mixer", [U.latent(5, 24, 12, 40, 36, 52), U.latent(16, 32, 16, 32, 48, 128), U.latent(40, 16, 8, 16, 24, 72)])
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-4), ("bfloat16", 3e-2)])
def test_ranges_of_latents(load, mixer, dtype, tol):  # noqa: F811
    cfg = U.config(64, 53, 1e-5, [U.layer(mixer, U.moe(3, 1, 16, 16))])
    steps_against_a_prompt(load, cfg, 5, (0, 1, 3, 4, 5, 8, 15, 16, 17, 295, 296, 297, 591, 592, 593, 1183, 1184, 1185), dtype, tol)
