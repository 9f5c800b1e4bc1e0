"""bf16 prompts of layers wide enough that a CTA of the tensor-core product walks several tiles, at every width of
tile, and that a row takes every width of the row kernels, against the 32-bit engine (held to the oracle elsewhere).

Tiles a CTA walks at most, over 148 SMs: `up` of 2048 rows by 4100 columns two of 256 columns, 6700 three, 8500 four; products of 2400
columns three of 128; 1700 rows by 1340 columns two of 64.  The gated products of 1800 rows: experts three of 128 columns, one expert
without a token among them; the shared expert three of 256.  The memory beside the attention is scaled to nothing: where
its denominators pass near zero, bf16 rounding grows tenfold.  Bounds as in the other tests of these models in bf16.
"""
import numpy as np
import pytest

from tests import kuzipel_util as KU
from tests import layered_util as U

pytestmark = pytest.mark.gpu


def compare(util, tmp_path, cfg, w, n, bound):
    from mongoose_b200 import registry
    util.write_folder(str(tmp_path), cfg, w)
    toks = util.tokens(cfg, n)
    places = sorted({0, 63, 127, 128, n // 2, n - 129, n - 65, n - 2, n - 1})
    got = []
    for dtype in ("float32", "bfloat16"):
        e = registry.load_model(str(tmp_path), dtype=dtype, max_seq=n)
        got.append(e.Forward(toks, 0, places))
        e.close()
    err = util.rel(got[1], got[0])
    assert err.max() < bound, (int(err.argmax()), err)


@pytest.mark.parametrize("n,width,ffn", [(2048, 2400, 4100), (1999, 1100, 6700), (1930, 900, 8500), (1700, 1340, 1340)])
def test_products_of_several_tiles(cuda, mglib, tmp_path, n, width, ffn):
    cfg = U.config(width, 300, 1e-5, [U.layer(4, 2, 24, 0.05, 0.3, 300, 2, 16, 24, 6.0, ffn)])
    w = U.weights(cfg, seed=n)
    w["l0.mix.right.out"][:] = 0
    compare(U, tmp_path, cfg, w, n, 3e-2)


def test_gated_products_of_several_tiles(cuda, mglib, tmp_path):
    n, width = 1800, 1030
    cfg = KU.config(width, 300, 1e-5, [KU.layer(KU.latent(4, 24, 12, 40, 36, 52), KU.moe(8, 2, 700, 3000))])
    w = KU.weights(cfg, seed=4, steady=True)
    w["l0.mlp.router.b"][3] = -100              # nobody's choice
    compare(KU, tmp_path, cfg, w, n, 3e-2)
