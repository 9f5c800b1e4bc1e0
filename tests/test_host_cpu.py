"""What the engine's host code asks of the CUDA runtime, seen through a stand-in for it (fake_cuda.cpp):
the library's own objects, host memory for device memory, kernels that do nothing.  Its results mean nothing;
which launches it makes, and which a device would refuse, does."""
import glob
import os
import subprocess

import numpy as np
import pytest

from mongoose_b200 import _lib, build
from mongoose_b200 import configs as mc
from mongoose_b200.fused_infer import CUDAFusedInference
from mongoose_b200.layered import (MATH_BF16, MATH_F32, GateAttention, LatentAttention, LayeredConfig, LayeredInference, MatrixMemory,
                                   MixtureOfExperts, ParallelLayer, PrenormLayer, Wkv, slot_shapes)

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    build.build()
    out = str(tmp_path_factory.mktemp("fake") / "libmongoose_fake.so")
    objs = [os.path.join(build.HERE, "build", u.replace(".cu", ".o")) for u in build.UNITS]
    subprocess.run(["g++", "-O1", "-fPIC", "-shared", "-I", os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include"), "-Wl,-Bsymbolic",
                    *objs, os.path.join(HERE, "fake_cuda.cpp"), "-o", out, "-ldl", "-lpthread"], check=True, capture_output=True, text=True)
    return out


@pytest.fixture
def fake(fake_path, monkeypatch):
    lib = _lib._open(fake_path, True)
    lib.fake_in_use.restype = lib.fake_smem.restype = _lib.sz
    lib.fake_memory.argtypes = [_lib.sz]
    monkeypatch.setattr(_lib, "_lib", lib)
    lib.fake_memory(8 << 30)
    lib.fake_forget()
    return lib


def layered(fake, layers, math=MATH_BF16, width=96, device=0, **kw):
    cfg = LayeredConfig("t", width, 50, tuple(layers), 1e-5, max_seq=512, math=math, **kw)
    e = LayeredInference(cfg, device)
    for idx, _, _, r, c in slot_shapes(cfg):
        e.SetWeightBF16(idx, np.zeros(max(r, 1) * c, np.uint16))
    e.BuildFusedDispatch()
    return e


def parallel(dim=64, heads=4, kv=2, ffn=160):
    return ParallelLayer(GateAttention(heads, kv, dim, 0.2), MatrixMemory(2, 16, 24, 5.0), ffn)


def prenorm():
    moe = MixtureOfExperts(4, 2, 40, 72)
    return [PrenormLayer(LatentAttention(4, 32, 16, 40, 72, 64, 0.1, 1e4), moe), PrenormLayer(Wkv(3, 32, 24), moe)]


def use(e, n=300):
    e.Forward([1] * n, 0, [n - 1])
    e.Forward([1] * 7, n, [6])
    e.Forward([1], n + 7, [0])


@pytest.mark.parametrize("kind", ["dim64", "dim256", "latent"])
@pytest.mark.parametrize("math", [MATH_BF16, MATH_F32])
def test_every_device_of_a_process_takes_the_kernels(fake, kind, math):
    """How much shared memory a kernel may be launched with belongs to the device."""
    layers = prenorm() if kind == "latent" else [parallel(int(kind[3:]))]
    for device in (0, 1, 2):
        e = layered(fake, layers, math, device=device)
        use(e)
        e.close()
    assert fake.fake_refused() == 0


@pytest.mark.parametrize("math", [MATH_BF16, MATH_F32])
def test_a_smaller_engine_takes_nothing_from_a_larger_one(fake, math):
    for layers, small, w in (([parallel(128, 8, 8, 30000)], [parallel(16, 2, 1, 64)], 128),
                             ([PrenormLayer(l.mixer, MixtureOfExperts(4, 2, 12000, 16000)) for l in prenorm()], prenorm(), 2048)):
        a = layered(fake, layers, math, width=w)
        b = layered(fake, small, math, width=32)
        use(b)
        use(a)
        a.close()
        b.close()
    assert fake.fake_refused() == 0


def dense(fake, cfg):
    e = CUDAFusedInference(cfg)
    for idx in range(12 * cfg.n_layers + 2):
        s = idx % 12 if idx < 12 * cfg.n_layers else -1
        if s in mc.MATRIX_SLOTS:
            e.SetWeight(idx, np.zeros(cfg.matrix_shape(s), np.float32))
        elif s in (mc.SLOT_NORM1, mc.SLOT_NORM2) or idx == 12 * cfg.n_layers:
            e.SetWeight(idx, np.zeros(cfg.dim, np.float32))
        elif s == -1:
            e.SetWeight(idx, np.zeros((cfg.vocab, cfg.dim), np.float32))
    e.BuildFusedDispatch()
    return e


@pytest.mark.parametrize("mega", [True, False])
@pytest.mark.parametrize("sizes", [({"ffn_dim": 9600}, {}), ({"max_seq": 16000}, {}), ({"ffn_dim": 9600, "max_seq": 9000}, {"max_seq": 64})])
def test_dense_engines_take_nothing_from_each_other(fake, monkeypatch, mega, sizes):
    if not mega:
        monkeypatch.setenv("MG_NO_MEGA", "1")
    engines = [dense(fake, mc.TINY.with_(**s)) for s in (*sizes, sizes[0])]
    for e in engines:
        e.Generate([1] * 40, 3)
    assert fake.fake_refused() == 0
    for e in engines:
        e.close()


@pytest.mark.parametrize("math", [MATH_BF16, MATH_F32])
@pytest.mark.parametrize("layers", [[parallel()], prenorm()], ids=["mitotar", "kuzipel"])
def test_no_pdl_covers_prompts(fake, monkeypatch, layers, math):
    for off in ("0", "1"):
        monkeypatch.setenv("MG_NO_PDL", off)
        e = layered(fake, layers, math)
        fake.fake_forget()
        e.Forward([1] * 300, 0, [299])
        e.Forward([1], 300, [0])
        assert fake.fake_launches(b"", -1) > 20
        assert (fake.fake_launches(b"", 1) > 0) == (off == "0")
        e.close()


@pytest.mark.parametrize("fmt", ["q8_0", "q4_0"])
@pytest.mark.parametrize("rows", [20, 2400, 8192])
@pytest.mark.parametrize("cols", [896, 18944, 27872, 28672, 32768, 38784, 40960, 49152, 51200])
def test_matvecs_stage_wide_inputs_in_shared_memory(fake, fmt, rows, cols):
    getattr(fake, f"mongoose_{fmt}_matvec")(256, 4096, 8192, rows, cols, None)
    assert fake.fake_launches(b"raw_block_matvec", -1) == 1 and fake.fake_refused() == 0
    assert fake.fake_smem() >= 4 * cols


@pytest.mark.parametrize("fmt", ["q8_0", "q4_0"])
@pytest.mark.parametrize("cols", [896, 5120, 5280, 5376, 5440, 5472, 18944])
def test_matvecs_launch_no_more_ctas_than_fit(fake, fmt, cols):
    getattr(fake, f"mongoose_{fmt}_matvec")(256, 4096, 8192, 20000, cols, None)
    assert fake.fake_ctas() <= 148 * (228 * 1024 // (fake.fake_smem() + 1024))


# heads, key heads, dim, tokens behind position -> the kernel of the bf16 attention
ROUTES = [(32, 4, 64, 0, 500, "flash"), (32, 8, 64, 0, 500, "flash"), (32, 16, 64, 0, 500, "scores"), (32, 32, 64, 0, 500, "scores"), (32, 32, 64, 0, 2, "scores"),
          (28, 4, 128, 0, 500, "flash"), (32, 8, 128, 0, 128, "flash"), (32, 8, 128, 0, 129, "scores"), (16, 8, 128, 0, 500, "scores"), (20, 20, 12, 0, 500, "flash"), (6, 6, 136, 0, 300, "scores"),
          (4, 4, 64, 0, 200, "flash"), (4, 4, 64, 0, 500, "scores"), (32, 4, 64, 400, 100, "flash"), (16, 4, 64, 400, 100, "scores"), (2, 2, 64, 400, 100, "scores")]


@pytest.mark.parametrize("heads,kv,dim,pos,n,kernel", ROUTES)
def test_route_of_the_gate_attention(fake, heads, kv, dim, pos, n, kernel):
    e = layered(fake, [parallel(dim, heads, kv)])
    if pos:
        e.Forward([1] * pos, 0)
    fake.fake_forget()
    e.Forward([1] * n, pos)
    other = {"flash": "scores", "scores": "flash"}[kernel]
    assert fake.fake_launches(b"gate_%s_kernel" % kernel.encode(), -1) == 1 and fake.fake_launches(b"gate_%s_kernel" % other.encode(), -1) == 0
    assert fake.fake_refused() == 0
    e.close()


def test_prompt_workspace_is_for_engines_that_batch_prompts(fake, monkeypatch):
    """Stages of a pipeline give it back, and it is never the price of an engine that would otherwise be made."""
    monkeypatch.setenv("MG_NO_MEGA", "1")
    cfg = mc.TINY.with_(ffn_dim=9600, max_seq=512)
    least = 3 * 512 * cfg.ffn_dim * 2                       # of one of its buffers
    e = dense(fake, cfg)
    whole = e.ArenaStats()
    assert whole["in_use"] > least and whole["outside"] == 0
    e.Generate([1] * 40, 3)
    assert fake.fake_launches(b"prompt_gemm", -1) > 0
    e.SetLayerRange(0, 1)
    e.BuildFusedDispatch()
    assert e.ArenaStats()["in_use"] < whole["in_use"] - least
    e.SetLayerRange(0, cfg.n_layers)
    e.BuildFusedDispatch()
    assert e.ArenaStats() == {**whole, "peak": e.ArenaStats()["peak"]}
    e.close()
    assert fake.fake_in_use() == 0
    # no room: token by token
    monkeypatch.setenv("MG_ARENA_MB", "1")
    fake.fake_memory(2 * least)
    e = dense(fake, cfg)
    fake.fake_forget()
    e.Generate([1] * 40, 3)
    assert fake.fake_launches(b"prompt_gemm", -1) == 0 and fake.fake_launches(b"", -1) > 0
    e.close()
    assert fake.fake_in_use() == 0
