"""Persistent kernel: cached rows that reach attention through the weight ring.

Contexts at the edges of blocks (8 rows), copies (40 rows) and ring entries (480, 240 and 120 rows for head sizes 32, 64 and
128), where heads start to be shared, and one layer, whose rows are read back soonest.  The graph of per-phase kernels fetches
its rows without a ring; both engines fill their caches by the same code.
"""
import numpy as np
import pytest

from mongoose_b200 import configs as mc
from oracle import gen
from tests.test_gpu_attention_splits import engines
from tests.util import assert_close

pytestmark = pytest.mark.gpu


def config(hd, max_seq, layers=2):
    heads = {32: 8, 64: 4, 128: 4}[hd]
    return mc.TINY.with_(name=f"rows-hd{hd}", dim=heads * hd, n_heads=heads, n_kv_heads=2, head_dim=hd, ffn_dim=2400, vocab=130, n_layers=layers,
                         max_seq=max_seq)


@pytest.mark.parametrize("hd, positions", [
    (32, (0, 1, 7, 8, 9, 39, 40, 41, 120, 479, 480, 481, 488, 719, 720, 721)),
    (64, (0, 1, 7, 8, 9, 39, 40, 41, 120, 239, 240, 241, 248, 480, 719, 720, 721, 959, 960)),
    (128, (0, 1, 7, 8, 9, 39, 40, 41, 119, 120, 121, 128, 240, 1439, 1440, 1441)),
])
def test_steps_at_the_edges(cuda, mglib, monkeypatch, hd, positions):
    cfg = config(hd, positions[-1] + 1)
    a, b = engines(cfg, monkeypatch)
    try:
        tokens = gen.prompt_ids(21, cfg.max_seq, cfg.vocab)
        at = 0
        x, y = np.empty(cfg.vocab, np.float32), np.empty(cfg.vocab, np.float32)
        for pos in positions:
            for e in (a, b):
                if pos > at:
                    e.Forward(tokens[at:pos], at)
                e.StepToken(int(tokens[pos]), pos, logitsOut=x if e is a else y)
            at = pos + 1
            # the caches may differ by one rounding to fp16 of the rows that steps appended
            assert_close(x, y, 5e-4, f"{cfg.name} position {pos}")
    finally:
        a.close(); b.close()


@pytest.mark.parametrize("hd, first, n, layers", [(32, 1, 60, 1), (64, 3, 300, 1), (64, 700, 60, 1), (64, 700, 60, 3), (128, 100, 60, 1), (128, 1425, 40, 2)])
def test_rows_appended_by_the_same_launch(cuda, mglib, monkeypatch, hd, first, n, layers):
    cfg = config(hd, first + n, layers)
    a, b = engines(cfg, monkeypatch)
    try:
        prompt = gen.prompt_ids(22, first, cfg.vocab)
        toks = a.Generate(prompt, n)
        b.Forward(np.concatenate((prompt, toks[:-1])), 0)
        x, y = np.empty(cfg.vocab, np.float32), np.empty(cfg.vocab, np.float32)
        for e, out in ((a, x), (b, y)):
            e.StepToken(int(toks[-1]), first + n - 1, logitsOut=out)
        assert_close(x, y, 5e-4, f"{cfg.name} behind {n} tokens")
    finally:
        a.close(); b.close()
