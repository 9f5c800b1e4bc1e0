"""Raw blocks on the integer tensor path: runs of rows around a tile and a pass, part segments, rows off 16 bytes, activations off
every alignment, and numbers that are not finite, against the kernel that a matrix off 16 bytes takes."""
import numpy as np
import pytest

from mongoose_b200 import kernels as K

pytestmark = pytest.mark.gpu


def quantized(oracle, fmt, n, k, seed):
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    x = (rng.standard_normal(k) * np.exp(2 * rng.standard_normal(k))).astype(np.float32)
    return np.ascontiguousarray(oracle.quantize(fmt, w)).reshape(-1).view(np.uint8), x


def product(t, fmt, blocks, x, n, k, shift=0, off=0):
    buf = t.zeros(blocks.size + shift, dtype=t.uint8, device="cuda")
    buf[shift:] = t.from_numpy(blocks).cuda()
    xb = t.zeros(k + off, device="cuda")
    xb[off:] = t.from_numpy(x).cuda()
    out = t.full((n + 2,), 5.0, device="cuda")
    (K.KQ8_0Matvec if fmt == 0 else K.KQ4_0Matvec)(xb[off:], buf[shift:], out, n, k)
    t.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.all(got[n:] == 5.0)
    return got[:n]


@pytest.mark.parametrize("N,K_", [(592, 1088), (593, 1152), (1200, 8192), (2369, 8256), (2384, 1984), (4736, 2048), (4737, 4096), (9475, 1088), (1184, 20544),
                                  (2400, 26624)])
@pytest.mark.parametrize("off", [0, 1, 2])
@pytest.mark.parametrize("fmt", [0, 1])
def test_rows_and_segments(cuda, oracle, mglib, N, K_, off, fmt):
    blocks, x = quantized(oracle, fmt, N, K_, N + K_)
    got = product(cuda, fmt, blocks, x, N, K_, off=off)
    values, x64 = oracle.dequant(fmt, blocks, N, K_).astype(np.float64), x.astype(np.float64)
    # a block's sum is exact but for the inputs, 2^-31 of the block's largest each; then at most K / 1024 + 2 roundings of sums over
    # blocks per digit, two over the digits and five over warps, each 2^-24 of a sum that the sizes of the terms bound
    size = np.abs(values) @ np.abs(x64)
    top = np.repeat(np.abs(x64).reshape(-1, 32).max(1), 32)
    assert np.all(np.abs(got - values @ x64) <= (9 + K_ / 1024) * 2.0 ** -24 * 2 * size + 2.0 ** -31 * (np.abs(values) @ top))


# matrices that end 4, 12 and 8 bytes behind a multiple of 16: those bytes of the last row do not come with its copy
@pytest.mark.parametrize("N,K_", [(593, 1088), (595, 1088), (593, 1152)])
@pytest.mark.parametrize("fmt", [0, 1])
def test_bytes_behind_the_last_whole_piece(cuda, oracle, mglib, N, K_, fmt):
    blocks, x = quantized(oracle, fmt, N, K_, N)
    other = quantized(oracle, fmt, N, K_, N + 1)[0]
    x[:-32] = 0                                             # the last row's sum hangs on them
    for b in (other, blocks, other, blocks):                # (shared memory holds the other matrix's)
        got = product(cuda, fmt, b, x, N, K_)
        values = oracle.dequant(fmt, b, N, K_).astype(np.float64)
        size = np.abs(values) @ np.abs(x.astype(np.float64))
        assert np.all(np.abs(got - values @ x.astype(np.float64)) <= 50 * 2.0 ** -24 * size + 2.0 ** -30 * np.abs(x).max() * np.abs(values[:, -32:]).sum(1))


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("kind", ["inf", "two infs", "nan", "scale inf", "huge", "tiny", "zeros"])
def test_numbers_off_the_range(cuda, oracle, mglib, fmt, kind):
    n, k = 640, 2048
    blocks, x = quantized(oracle, fmt, n, k, 7)
    values = oracle.dequant(fmt, blocks, n, k).astype(np.float64)
    if kind == "inf":
        x[100] = np.inf
    elif kind == "two infs":
        x[100], x[1500] = np.inf, -np.inf
    elif kind == "nan":
        x[64] = np.nan
    elif kind == "scale inf":
        size = 34 if fmt == 0 else 18
        blocks[(3 * k // 32 + 5) * size:][:2] = (0x00, 0x7C)
    elif kind == "huge":
        x[:] = np.where(np.arange(k) % 2, 1e34, -1e34)      # (beyond 1e36 the plain kernel's products overflow on the way to finite sums)
    elif kind == "tiny":
        x *= np.float32(1e-36)
    else:
        x[:1024] = 0
    got, want = product(cuda, fmt, blocks, x, n, k), product(cuda, fmt, blocks, x, n, k, shift=2)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.array_equal(got[~ok & ~np.isnan(want)], want[~ok & ~np.isnan(want)])
    # of the rows that stay finite: both are off by at most 40 + K / 1024 roundings of sums that the sizes of the terms bound
    size = np.abs(values[ok]) @ np.abs(np.where(np.isfinite(x), x, 0).astype(np.float64))
    assert np.all(np.abs(got[ok].astype(np.float64) - want[ok]) <= 2 * (40 + k / 1024) * 2.0 ** -24 * size + 1e-44)
