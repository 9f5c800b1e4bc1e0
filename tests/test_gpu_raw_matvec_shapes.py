"""Matvec on raw blocks at the edges of its split: shared rows, pairs with an odd row, part chunks, matrices and
activations off every alignment a caller may use, inputs too wide for shared memory."""
import numpy as np
import pytest

from mongoose_b200 import kernels as K

pytestmark = pytest.mark.gpu
# activations without gaps: pairs, single rows on 16 and on 8 warps; the narrowest that stay in global memory
WIDE = [(2369, 28672), (2369, 32800), (40, 39648), (70, 44640), (33, 50752), (9, 51232), (9, 54304)]


@pytest.mark.parametrize("N,K_", [(1, 32), (3, 1056), (100, 8192), (65, 19200), (2369, 2080), (3553, 64), (7105, 1024), (20, 51200), *WIDE])
@pytest.mark.parametrize("shift", [0, 2, 4, 8])
@pytest.mark.parametrize("fmt", [0, 1])
def test_raw_matvec_shapes(cuda, oracle, mglib, N, K_, shift, fmt):
    t = cuda
    rng = np.random.default_rng(N + K_)
    w = (rng.standard_normal((N, K_)) * 0.02).astype(np.float32)
    x = rng.standard_normal(K_).astype(np.float32)
    blocks = np.ascontiguousarray(oracle.quantize(fmt, w)).reshape(-1).view(np.uint8)
    buf = t.zeros(blocks.size + shift, dtype=t.uint8, device="cuda")
    buf[shift:] = t.from_numpy(blocks).cuda()
    xb = t.zeros(K_ + 1, device="cuda")
    xv = xb[shift == 2:][:K_]                       # off 16 bytes as well
    xv.copy_(t.from_numpy(x))
    out = t.full((N + 2,), 5.0, device="cuda")
    (K.KQ8_0Matvec if fmt == 0 else K.KQ4_0Matvec)(xv, buf[shift:], out, N, K_)
    t.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.all(got[N:] == 5.0)
    values = oracle.dequant(fmt, blocks, N, K_).astype(np.float64)
    # fp32 sums of up to K terms in pieces of 32 and their tree: each rounding is 2^-24 of a partial sum, which the sum of
    # the terms' sizes bounds; at most 32 + K / 1024 + 8 of them follow one another
    bound = (40 + K_ / 1024) * 2.0 ** -24 * (np.abs(values) @ np.abs(x.astype(np.float64)))
    assert np.all(np.abs(got[:N] - values @ x.astype(np.float64)) <= bound)
