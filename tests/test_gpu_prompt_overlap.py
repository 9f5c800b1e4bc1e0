"""Prompts whose launches overlap (programmatic dependent launch) against the same launches one after the other."""
import numpy as np
import pytest

from tests import kuzipel_util, layered_util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("util", [layered_util, kuzipel_util], ids=["mitotar", "kuzipel"])
def test_overlapped_prompts_equal_serial_ones(cuda, mglib, tmp_path, monkeypatch, util, dtype):
    from mongoose_b200 import registry
    cfg = util.CONFIGS["mixed"]
    util.write_folder(str(tmp_path), cfg, util.weights(cfg, seed=3))
    toks = util.tokens(cfg, 300)
    got = []
    for off in ("0", "1"):
        monkeypatch.setenv("MG_NO_PDL", off)
        e = registry.load_model(str(tmp_path), dtype=dtype, max_seq=300)
        got.append(np.concatenate([e.Forward(toks[:230], 0, range(230)), e.Forward(toks[230:], 230, range(70))]))
        e.close()
    assert np.array_equal(*got)
