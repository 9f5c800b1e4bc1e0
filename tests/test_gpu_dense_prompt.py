"""Prompts of the seven-matrix block in batches of tokens against the same tokens fed one by one.

Sizes at the edges of the kernels: 4 tokens are the fewest that are batched, products take 32 or 64 tokens
and 128 rows per tile, attention 32 queries and 64 keys, a batch 512 tokens; widths that are odd multiples of
32 leave half a step of K.  Keys and values are rounded to fp16: a sum's last bits move some of them to the
neighbouring half, which is 2^-10 of the entry, and moves logits by less than 5e-4 of their largest.
"""
import numpy as np
import pytest

from mongoose_b200 import configs as mc
from mongoose_b200.fused_infer import CUDAFusedInference
from oracle import gen
from tests.util import assert_close, fill_models

pytestmark = pytest.mark.gpu

ODD = mc.TINY.with_(name="odd", dim=224, n_heads=7, n_kv_heads=1, head_dim=32, ffn_dim=416, vocab=333, n_layers=3, max_seq=160)
HD64 = mc.TINY.with_(name="hd64", dim=256, n_heads=4, n_kv_heads=1, head_dim=64, ffn_dim=352, vocab=333, max_seq=600)
HD128 = mc.TINY.with_(name="hd128", dim=384, n_heads=3, n_kv_heads=3, head_dim=128, ffn_dim=160, vocab=333, max_seq=160)
CASES = [(ODD, n) for n in (5, 33, 66)] + [(HD64, n) for n in (65, 513, 580)] + [(HD128, n) for n in (34, 130)]


def same_cache(cfg, a, b, n):
    for l in range(cfg.n_layers):
        for x, y in zip(a.ReadKV(l, 0, n), b.ReadKV(l, 0, n)):
            x, y = (np.asarray(v).view(np.float16).astype(np.float64).reshape(n, -1) for v in (x, y))
            assert np.all(np.isfinite(x))
            # one rounding to fp16 (2^-10 of the entry) over sums that agree to 1e-4 of the row's largest
            bound = 2.0 ** -10 * np.abs(y) + 1e-4 * np.abs(y).max(1, keepdims=True)
            assert np.all(np.abs(x - y) <= bound), f"layer {l}: off by {np.abs(x - y).max():.2e}"


@pytest.mark.parametrize("cfg,n", CASES, ids=lambda v: getattr(v, "name", v))
@pytest.mark.parametrize("fmt", [mc.FMT_Q8_0, mc.FMT_Q4_0, mc.FMT_F16], ids=["q8_0", "q4_0", "f16"])
def test_batched_prompt_equals_tokens_one_by_one(cuda, oracle, mglib, cfg, n, fmt):
    cfg = cfg.with_(layer_fmt=fmt, head_fmt=fmt)
    a, b, om = CUDAFusedInference(cfg), CUDAFusedInference(cfg), oracle.OracleModel(cfg)
    try:
        fill_models(cfg, seed=5, jitter=0.1, engine=a, oracle_model=om, bias=True)
        fill_models(cfg, seed=5, jitter=0.1, engine=b, bias=True)
        tokens = gen.prompt_ids(6, n, cfg.vocab)
        got = a.Forward(tokens, 0, (n - 1,))[0]
        step = np.empty(cfg.vocab, np.float32)
        for i, t in enumerate(tokens):
            b.StepToken(int(t), i, logitsOut=step if i == n - 1 else None)
            if i < 200:                         # the oracle's steps grow with the context
                want = om.step_token(int(t), i)
        same_cache(cfg, a, b, n)
        assert_close(got, step, 5e-4, "logits behind the prompt")
        if n <= 200:
            assert_close(got, want, 5e-4, "logits against the oracle")
        assert a.GetCursor() == b.GetCursor()
        assert_close(a.ExportHidden(), b.ExportHidden(), 5e-4, "hidden state")
    finally:
        a.close(); b.close(); om.close()


def test_cuts_wanted_places_and_start_positions(cuda, mglib):
    cfg = HD64
    a, b = CUDAFusedInference(cfg), CUDAFusedInference(cfg)
    try:
        for e in (a, b):
            fill_models(cfg, seed=7, jitter=0.1, engine=e)
        tokens = gen.prompt_ids(8, 150, cfg.vocab)
        want = a.Forward(tokens, 0, (2, 70, 149))
        got = [b.Forward(tokens[:3], 0, (2,)), b.Forward(tokens[3:71], 3, (67,)), b.Forward(tokens[71:72], 71), b.Forward(tokens[72:], 72, (77,))]
        for w, g in zip(want, [got[0][0], got[1][0], got[3][0]]):
            assert_close(g, w, 5e-4, "logits at a wanted place")
        same_cache(cfg, a, b, 150)
        # a sequence that goes on from its cached prompt
        assert np.array_equal(a.Generate(tokens[:40], 6, start_pos=150), b.Generate(tokens[:40], 6, start_pos=150))
        same_cache(cfg, a, b, 195)
    finally:
        a.close(); b.close()


def test_batches_on_the_graph_of_kernels(cuda, mglib, monkeypatch):
    monkeypatch.setenv("MG_NO_MEGA", "1")
    cfg = ODD
    a, b = CUDAFusedInference(cfg), CUDAFusedInference(cfg)
    try:
        for e in (a, b):
            fill_models(cfg, seed=9, jitter=0.1, engine=e)
        tokens = gen.prompt_ids(10, 50, cfg.vocab)
        a.Forward(tokens, 0)
        for i, t in enumerate(tokens):
            b.StepToken(int(t), i)
        same_cache(cfg, a, b, 50)
    finally:
        a.close(); b.close()


@pytest.mark.parametrize("cfg", [ODD, HD64, HD128], ids=lambda c: c.name)
def test_a_value_that_overflows_leaves_earlier_tokens_alone(cuda, mglib, cfg):
    """One token's value is beyond fp16 (infinite in the cache): the tokens before it, in the same tile of keys or
    an earlier one, are as they are without it."""
    n, at = 90, 77
    tokens = [int(t) % (cfg.vocab - 1) for t in gen.prompt_ids(11, n, cfg.vocab)]
    tokens[at] = cfg.vocab - 1
    embed = gen.tensor_f32(12, 1, cfg.vocab, cfg.dim)
    embed[:, 0] = 0
    embed[-1] = 0
    embed[-1, 0] = 1                        # of the normed input nothing but column 0, which is 0 for every other token
    wv = gen.tensor_f32(12, 2, cfg.kv_dim, cfg.dim)
    wv[0, 0] = 2e4
    a, b = CUDAFusedInference(cfg), CUDAFusedInference(cfg)
    try:
        for e in (a, b):
            fill_models(cfg, seed=12, jitter=0.1, engine=e)
            e.SetWeight(12 * cfg.n_layers + 1, embed)
            e.SetWeight(mc.SLOT_WV, wv)
        a.Forward(tokens, 0)
        for i, t in enumerate(tokens[:at]):
            b.StepToken(t, i)
        assert np.isinf(a.ReadKV(0, at, 1)[1].view(np.float16)[0, 0])
        same_cache(cfg, a, b, at)
    finally:
        a.close(); b.close()
