"""Persistent kernel: CTAs that share a query head, at the positions where another one joins.

The graph of per-phase kernels attends with one CTA per head; both engines fill their caches by the same code.
"""
import numpy as np
import pytest

from mongoose_b200 import configs as mc
from mongoose_b200.fused_infer import CUDAFusedInference
from oracle import gen
from tests.util import assert_close, fill_models

pytestmark = pytest.mark.gpu

# every CTA owns gate/up rows, so that heads may be shared
CASES = [
    mc.TINY.with_(name="hd64", dim=256, n_heads=4, n_kv_heads=2, head_dim=64, ffn_dim=2400, vocab=777, max_seq=1300),
    mc.TINY.with_(name="hd128", dim=512, n_heads=4, n_kv_heads=1, head_dim=128, ffn_dim=2400, vocab=130, max_seq=1300),
    mc.TINY.with_(name="hd32", dim=1376, n_heads=43, n_kv_heads=43, head_dim=32, ffn_dim=2400, vocab=130, max_seq=1300),    # three CTAs a head
]


def engines(cfg, monkeypatch):
    a = CUDAFusedInference(cfg)
    monkeypatch.setenv("MG_NO_MEGA", "1")
    b = CUDAFusedInference(cfg)
    monkeypatch.delenv("MG_NO_MEGA")
    for e in (a, b):
        fill_models(cfg, seed=11, jitter=0.1, engine=e)
        e.BuildFusedDispatch()
    assert a.DecodePath() != b.DecodePath()
    return a, b


@pytest.mark.parametrize("cfg", CASES, ids=lambda c: c.name)
def test_steps_where_a_cta_joins(cuda, mglib, monkeypatch, cfg):
    a, b = engines(cfg, monkeypatch)
    try:
        tokens = gen.prompt_ids(12, 1300, cfg.vocab)
        at = 0
        x, y = np.empty(cfg.vocab, np.float32), np.empty(cfg.vocab, np.float32)
        for pos in (240, 318, 319, 320, 321, 479, 480, 481, 719, 720, 961, 1199, 1200, 1299):
            for e in (a, b):
                if pos > at:
                    e.Forward(tokens[at:pos], at)
                e.StepToken(int(tokens[pos]), pos, logitsOut=x if e is a else y)
            at = pos + 1
            # the caches may differ by one rounding to fp16 of the rows that steps appended
            assert_close(x, y, 5e-4, f"{cfg.name} position {pos}")
    finally:
        a.close(); b.close()


@pytest.mark.parametrize("cfg", CASES, ids=lambda c: c.name)
def test_one_call_across_the_joins(cuda, mglib, monkeypatch, cfg):
    a, b = engines(cfg, monkeypatch)
    try:
        prompt = gen.prompt_ids(13, 230, cfg.vocab)
        n = 270                                 # from one CTA a head to three
        toks = a.Generate(prompt, n)
        b.Forward(np.concatenate((prompt, toks[:-1])), 0)
        x, y = np.empty(cfg.vocab, np.float32), np.empty(cfg.vocab, np.float32)
        for e, out in ((a, x), (b, y)):
            e.StepToken(int(toks[-1]), 230 + n - 1, logitsOut=out)
        assert_close(x, y, 5e-4, f"{cfg.name} behind {n} tokens")
        k, v = a.ReadKV(cfg.n_layers - 1, 0, 230 + n)
        kb, vb = b.ReadKV(cfg.n_layers - 1, 0, 230 + n)
        for p, q in ((k, kb), (v, vb)):
            p, q = p.view(np.float16).astype(np.float32), q.view(np.float16).astype(np.float32)
            assert np.all(np.abs(p - q) <= 2.0 ** -10 * np.abs(q) + 2e-4 * np.abs(q).max(1, keepdims=True))
    finally:
        a.close(); b.close()
