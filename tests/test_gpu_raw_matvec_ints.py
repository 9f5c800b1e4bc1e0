"""Raw blocks on the integer tensor path: runs of rows around a tile and a turn, part segments, rows off 16 bytes, activations off
every alignment, activations that span more than digits hold, and numbers that are not finite, against 64 bits and the kernel that a
matrix off 16 bytes takes."""
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
    # a block's inputs are exact; each part's sum is rounded once per block, at most K / 1024 + 2 times over blocks, twice over the parts
    # and five times over warps, each 2^-24 of a sum that the sizes of the parts bound: twice an element's own where it is 2^-13 of its
    # block's largest or more (three times below, which weighs nothing here)
    size = np.abs(values) @ np.abs(x64)
    assert np.all(np.abs(got - values @ x64) <= (9 + K_ / 1024) * 2.0 ** -24 * 2 * size)


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
        assert np.all(np.abs(got - values @ x.astype(np.float64)) <= 50 * 2.0 ** -24 * size)


def one_weight_a_row(rng, fmt, n, k, col, scale):
    """Blocks whose only weight other than zero is q * scale in column col[row] of a row."""
    q = rng.choice((-7, -3, -1, 1, 2, 5, 7), n)
    size = 34 if fmt == 0 else 18
    blocks = np.zeros((n, k // 32, size), np.uint8)
    blocks[:, :, :2] = np.full(1, scale, np.float16).view(np.uint8)
    if fmt == 0:
        blocks[np.arange(n), col // 32, 2 + col % 32] = q.astype(np.int8).view(np.uint8)
    else:
        blocks[:, :, 2:] = 0x88
        at, high = 2 + col % 16, col % 32 >= 16
        blocks[np.arange(n), col // 32, at] = np.where(high, (q + 8) << 4 | 8, 0x80 | (q + 8)).astype(np.uint8)
    return blocks.reshape(-1)


def assert_terms(cuda, oracle, fmt, blocks, x, col):
    n, k = len(col), len(x)
    values = oracle.dequant(fmt, blocks, n, k).astype(np.float64)
    want = values @ x.astype(np.float64)
    assert np.array_equal(want, values[np.arange(n), col] * x.astype(np.float64)[col])
    got = product(cuda, fmt, blocks, x, n, k)
    # digits: one rounding of each part's product and two of their sum, parts of up to three times the term in all; a rest and a term in fp32 one
    # of q x and one of its product with the scale
    assert np.all(np.abs(got - want) <= 9 * 2.0 ** -24 * np.abs(want))


# Every row has one weight that is not zero, so that its sum has one term; the first activation of a block is 2^top, the others around 2^power, and
# `scale` is the blocks': whatever shares a block with an activation, and however small the scales' product is, a term has fp32's bits.  The last lines
# are products near the ends of fp32's range.
@pytest.mark.parametrize("top,power,scale", [(0, 0, 1e-2), (10, 0, 1e-2), (12, 0, 1e-2), (16, 0, 1e-2), (20, 0, 1e-2), (24, 0, 1e-2), (34, 0, 1e-2), (100, 0, 1e-2), (126, -60, 1e-2),
                                             (-78, -82, 2.0 ** -20), (-82, -86, 2.0 ** -20), (-96, -98, 2.0 ** -14), (126, 122, 2.0 ** -10)])
@pytest.mark.parametrize("fmt", [0, 1])
def test_one_term_a_row(cuda, oracle, mglib, fmt, top, power, scale):
    n, k = 640, 2048
    rng = np.random.default_rng(top + 200)
    x = (rng.standard_normal(k) * 2.0 ** power).astype(np.float32)
    x[::32] = 2.0 ** top
    col = rng.integers(0, k // 32, n) * 32 + rng.integers(1, 32, n)
    assert_terms(cuda, oracle, fmt, one_weight_a_row(rng, fmt, n, k, col, scale), x, col)


# the same where a share of the activations is 2^-10 to 2^-40 of the others: no, few and most blocks go without digits
@pytest.mark.parametrize("share", [0.003, 0.02, 0.3])
@pytest.mark.parametrize("n,k", [(640, 2048), (5000, 3584), (2400, 20544)])
@pytest.mark.parametrize("fmt", [0, 1])
def test_few_small_activations(cuda, oracle, mglib, fmt, n, k, share):
    rng = np.random.default_rng(k)
    x = rng.standard_normal(k).astype(np.float32)
    small = np.flatnonzero(rng.random(k) < share)
    x[small] *= (2.0 ** -rng.integers(10, 40, small.size)).astype(np.float32)
    col = rng.choice(small, n)
    col[::3] = rng.integers(0, k, col[::3].size)
    assert_terms(cuda, oracle, fmt, one_weight_a_row(rng, fmt, n, k, col, 1e-2), x, col)


# the same with all weights: fp32 sums of 32 terms in blocks without digits, of K / 32 blocks in some order
@pytest.mark.parametrize("top", [6, 11, 12, 13, 16, 20, 24, 34, 60])
@pytest.mark.parametrize("N,K_", [(640, 2048), (2369, 1088), (1190, 20544)])
@pytest.mark.parametrize("fmt", [0, 1])
def test_largest_of_a_block_under_no_weight(cuda, oracle, mglib, fmt, N, K_, top):
    rng = np.random.default_rng(top)
    w = (rng.standard_normal((N, K_)) * 0.02).astype(np.float32)
    w[:, ::32] = 0
    x = rng.standard_normal(K_).astype(np.float32)
    x[rng.integers(0, K_, K_ // 8)] = 0
    x[::32] = np.where(rng.random(K_ // 32) < 0.7, 2.0 ** top, x[::32])
    blocks = np.ascontiguousarray(oracle.quantize(fmt, w)).reshape(-1).view(np.uint8)
    values, x64 = oracle.dequant(fmt, blocks, N, K_).astype(np.float64), x.astype(np.float64)
    assert not values[:, ::32].any()
    got = product(cuda, fmt, blocks, x, N, K_)
    size = np.abs(values) @ np.abs(x64)
    assert np.all(np.abs(got - values @ x64) <= 3 * (40 + K_ / 1024) * 2.0 ** -24 * size)
    # without a term in the block's largest, and close: the errors of all rows together are those of a few roundings each
    assert np.linalg.norm(got - values @ x64) <= 3 * 2.0 ** -24 * np.linalg.norm(size)


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
