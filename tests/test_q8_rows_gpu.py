"""The many-row Q8 projection (tensor cores, one accumulation per scale block) in small sizes: rows and columns that fill no
tile, K of odd block counts and of no whole block, strided windows, and the fused LayerNorm and GELU, on tiles of 16 to 64 rows; a
few shapes lie just outside its dispatch.  test_q8_routes_gpu.py takes every tile width and split by name."""
import numpy as np
import pytest

import oracle
from deepj_b200.compute_graph import OP_Q8_LINEAR, OP_Q8_LINEAR_LN, OP_Q8_SWIGLU, float_bits
from test_q8_gpu import dev  # noqa: F401

pytestmark = pytest.mark.gpu


def bound(K):
    """2-norm error over the result's: activations as two fp16 values (2^-22), fp32 sums of 32 products and of K/32 blocks
    (2^-24 each in the worst case); weights are exact."""
    return 2.0 ** -22 + (32 + (K + 31) // 32) * 2.0 ** -24


def weights(dev, rng, K, N):  # noqa: F811
    W = (rng.standard_normal((K, N)) * 0.02).astype(np.float32)
    return dev.q8(W), oracle.q8_dequantize(*oracle.q8_quantize(W)).astype(np.float64)


def check(got, want, K):
    assert np.linalg.norm(got - want) <= bound(K) * np.linalg.norm(want)


@pytest.mark.parametrize("M,K,N", [(17, 36, 50), (33, 160, 130), (48, 100, 257), (65, 1600, 96), (129, 352, 333), (300, 2048, 128), (97, 4128, 640),
                                   (5, 1600, 1600), (16, 96, 4096), (513, 64, 2050), (260, 32, 17)])
def test_rows(dev, M, K, N):  # noqa: F811
    rng = np.random.default_rng(M + K + N)
    q, W = weights(dev, rng, K, N)
    x, g, b, r = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), K, N, (M, N)))
    xb, gb, bb, rb, ob = dev.buf(M * K, x), dev.buf(K, g), dev.buf(N, b), dev.buf(M * N, r), dev.buf(M * (N + 3), np.full(M * (N + 3), 7.0))
    dev.flush([OP_Q8_LINEAR, xb, 0, K, gb, float_bits(1e-6), q, bb, rb, 0, N, ob, 3, N + 3, M - 1])        # a strided window; the last row stays
    xd = x.astype(np.float64)
    want = (xd / np.sqrt((xd * xd).mean(1, keepdims=True) + 1e-6) * g) @ W + b + r
    got = dev.get(ob, M * (N + 3)).reshape(-1)[3:]
    got = np.concatenate([got, np.zeros(3)]).reshape(M, N + 3)
    check(got[:M - 1, :N], want[:M - 1], K)
    assert np.all(got[:M - 1, N:] == 7.0) and np.all(got[M - 1, :N] == 7.0)


@pytest.mark.parametrize("M,K,F", [(18, 64, 33), (70, 1600, 200), (130, 416, 64), (260, 2048, 130), (9, 1056, 2200)])
def test_pairs(dev, M, K, F):  # noqa: F811
    rng = np.random.default_rng(M + K + F)
    (q1, W1), (q2, W2) = weights(dev, rng, K, F), weights(dev, rng, K, F)
    x, b1, b2 = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), F, F))
    ob = dev.buf(M * F)
    dev.flush([OP_Q8_SWIGLU, dev.buf(M * K, x), 0, K, -1, float_bits(1e-6), q1, dev.buf(F, b1), q2, dev.buf(F, b2), ob, 0, F, M])
    a = x.astype(np.float64) @ W1 + b1
    check(dev.get(ob, M * F).reshape(M, F), a / (1.0 + np.exp(-a)) * (x.astype(np.float64) @ W2 + b2), K)


@pytest.mark.parametrize("M,K,N,act", [(20, 1600, 200, 1), (130, 96, 130, 0), (200, 1600, 64, 1), (6, 1600, 1600, 1)])
def test_layernorm_and_gelu(dev, M, K, N, act):  # noqa: F811
    rng = np.random.default_rng(M + K + N)
    q, W = weights(dev, rng, K, N)
    x, g, b, c = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), K, K, N))
    ob = dev.buf(M * N)
    dev.flush([OP_Q8_LINEAR_LN, dev.buf(M * K, x), 0, K, dev.buf(K, g), dev.buf(K, b), float_bits(1e-5), q, dev.buf(N, c), -1, 0, 0, ob, 0, N, M, act])
    xd = x.astype(np.float64)
    v = ((xd - xd.mean(1, keepdims=True)) / np.sqrt(xd.var(1, keepdims=True) + 1e-5) * g + b) @ W + c
    if act:
        v = 0.5 * v * (1.0 + np.tanh(np.sqrt(2.0 / np.pi) * (v + 0.044715 * v ** 3)))
    check(dev.get(ob, M * N).reshape(M, N), v, K)
