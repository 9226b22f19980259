"""Many-row bf16 products on pairs of SMs: ragged rows, columns and lengths, fewer k-steps than ring stages and more, up to five tiles per
pair (an accumulator is used again from the third on), every part of the epilogue, against the product of the rounded rows in float64.  That the
rows go to the pairs is asserted, so that a case keeps testing what it names (148 SMs)."""
import ctypes

import numpy as np
import pytest

from deepj_b200 import _lib
from deepj_b200.compute_graph import OP_BF16_LINEAR_SUM, float_bits
from test_bf16_ops_gpu import bf16, dev  # noqa: F401

pytestmark = pytest.mark.gpu


def route(dev, M, K, N):  # noqa: F811
    out = (ctypes.c_int32 * 2)()
    _lib.check(dev.lib.deepj_cuda_bf16_route(M, K, N, out))
    return tuple(out)


@pytest.mark.parametrize("M,K,N,glu", [(2048, 64, 4096, 4096), (1900, 200, 4600, 4600), (2047, 1032, 4608, 2304), (1290, 520, 8680, 4344), (1500, 264, 7848, 0),
                                       (2040, 72, 11400, 11400), (640, 3592, 4096, 2048)])
def test_pairs(dev, M, K, N, glu):  # noqa: F811
    assert route(dev, M, K, N) == (1, 256)
    rng = np.random.default_rng(M + K + N)
    w, x = bf16(rng.standard_normal((N, K)) * 0.05), bf16(rng.standard_normal((M, K)))
    bias, res = rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, max(glu, 1))).astype(np.float32)
    pairs = (N - glu) // 2
    xi, bi, ri, W = dev.buf(x.size, x), dev.buf(bias.size, bias), dev.buf(res.size, res), dev.weight(K, N, [(w, 0, 1, 0)])
    out, gl = dev.buf(M * max(glu, 1)), dev.buf(M * max(pairs, 1))
    dev.flush([OP_BF16_LINEAR_SUM, xi, 0, K, -1, 0, float_bits(0.0), -1, 0, 0, K, -1, 0, 0, W, ri if glu else -1, 0, glu, out if glu else -1, 0, glu, M, glu,
               float_bits(0.0), gl if pairs else -1, 0, pairs, float_bits(0.0), 0, bi if glu else -1, 1, -1, 0, 0, float_bits(0.0), -1, 0, 0])
    want = x.astype(np.float64) @ w.astype(np.float64).T
    # exact products; fp32 sums that the tensor core cuts instead of rounding, one per 16 of the length
    bound = 2.0 ** -22 * (K / 16 + 8) * (np.abs(x).max() * 0.2 * np.sqrt(K) + 4)
    if glu:
        got = dev.get(out, M * glu).reshape(M, glu)
        assert np.abs(got - (want[:, :glu] + bias[:glu] + res)).max() <= bound
    if pairs:
        g, u = want[:, glu::2], want[:, glu + 1::2]
        got = dev.get(gl, M * pairs).reshape(M, pairs)
        assert np.abs(got - g / (1 + np.exp(-g)) * u).max() <= 4 * bound * (np.abs(want).max() + 1)


def test_rows_stay_on_single_sms(dev):  # noqa: F811
    """Short lengths whose rounds are no cheaper on pairs, and the length from which they are."""
    assert [route(dev, 640, K, 4096) for K in (64, 2048, 3576, 3584)] == [(0, 64), (0, 64), (0, 64), (1, 256)]
    assert [route(dev, M, 2048, 40000) for M in (256, 640, 768, 2048)] == [(0, 128), (0, 128), (1, 256), (1, 256)]
