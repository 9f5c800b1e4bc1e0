"""Persistent kernel: CTAs that share a query head, at the positions where another one joins.

The graph of per-phase kernels attends with one CTA per head; both engines fill their caches by the same code.
"""
import os
import re

import numpy as np
import pytest

from mongoose_b200 import build, configs as mc
from mongoose_b200.fused_infer import CUDAFusedInference
from oracle import gen
from tests.util import assert_close, fill_models

pytestmark = pytest.mark.gpu

# every CTA owns gate/up rows, so that heads may be shared
CASES = [
    mc.TINY.with_(name="hd64", dim=256, n_heads=4, n_kv_heads=2, head_dim=64, ffn_dim=2400, vocab=777),
    mc.TINY.with_(name="hd128", dim=512, n_heads=4, n_kv_heads=1, head_dim=128, ffn_dim=2400, vocab=130),
    mc.TINY.with_(name="hd32", dim=1376, n_heads=43, n_kv_heads=43, head_dim=32, ffn_dim=2400, vocab=130),    # three CTAs a head
]


def joins(cfg, sms=148):
    """Positions from which one more CTA (or several at once) shares a head, by the constants of the kernel."""
    with open(os.path.join(build.CSRC, "mega_kernel.cuh")) as f:
        src = f.read()
    run, most = (int(re.search(rf"constexpr int {n} = (\d+);", src)[1]) for n in ("MK_SPLIT_POSITIONS", "MK_MAX_SPLITS"))
    wide, narrow = map(int, re.search(r"mk_split_from\(int head_dim\) { return head_dim > 64 \? (\d+) : (\d+); }", src).groups())
    first, most = wide if cfg.head_dim > 64 else narrow, min(most, sms // cfg.n_heads)

    def count(pos):
        return 1 if pos < first else min((pos + run) // run, most)

    at = [p for p in range(1, run * most + 1) if count(p) != count(p - 1)]
    assert at and at[0] == first and count(at[-1]) == most
    return at


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
    edges = sorted({240, 479, 480, 481} | {p + d for p in joins(cfg) for d in (-1, 0, 1)})
    cfg = cfg.with_(max_seq=edges[-1] + 1)
    a, b = engines(cfg, monkeypatch)
    try:
        tokens = gen.prompt_ids(12, cfg.max_seq, cfg.vocab)
        at = 0
        x, y = np.empty(cfg.vocab, np.float32), np.empty(cfg.vocab, np.float32)
        for pos in edges:
            for e in (a, b):
                if pos > at:
                    e.Forward(tokens[at:pos], at)
                e.StepToken(int(tokens[pos]), pos, logitsOut=x if e is a else y)
            at = pos + 1
            # the caches may differ by one rounding to fp16 of the rows that steps appended
            assert_close(x, y, 5e-4, f"{cfg.name} position {pos}")
    finally:
        a.close(); b.close()


# One launch decodes tokens before and behind a join: CTAs that join have appended the launch's rows without attending.  (The first
# join ends a launch: behind it the other instance of the kernel runs.)
@pytest.mark.parametrize("cfg", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("which", ["each", "all"])
def test_one_call_across_the_joins(cuda, mglib, monkeypatch, cfg, which):
    at = joins(cfg)
    ranges = [(p - 30, 60) for p in at] if which == "each" else [(at[0] - 20, at[-1] - at[0] + 40)]
    cfg = cfg.with_(max_seq=at[-1] + 40)
    a, b = engines(cfg, monkeypatch)
    try:
        for first, n in ranges:
            prompt = gen.prompt_ids(13, first, cfg.vocab)
            toks = a.Generate(prompt, n)
            b.Forward(np.concatenate((prompt, toks[:-1])), 0)
            x, y = np.empty(cfg.vocab, np.float32), np.empty(cfg.vocab, np.float32)
            for e, out in ((a, x), (b, y)):
                e.StepToken(int(toks[-1]), first + n - 1, logitsOut=out)
            assert_close(x, y, 5e-4, f"{cfg.name} behind {first} + {n} tokens")
            k, v = a.ReadKV(cfg.n_layers - 1, 0, first + n)
            kb, vb = b.ReadKV(cfg.n_layers - 1, 0, first + n)
            for p, q in ((k, kb), (v, vb)):
                p, q = p.view(np.float16).astype(np.float32), q.view(np.float16).astype(np.float32)
                assert np.all(np.abs(p - q) <= 2.0 ** -10 * np.abs(q) + 2e-4 * np.abs(q).max(1, keepdims=True))
    finally:
        a.close(); b.close()
