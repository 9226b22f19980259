"""The few-row Q8 kernel at the edges of its groups (128), its warps (8 groups), its register rounds (4 groups a warp), its tiles (16 rows,
half tiles) and its chunks (16 tiles × rows), with RMSNorm, LayerNorm, GELU and the gated pair, against float64."""
import os
import subprocess
import sys

import numpy as np
import pytest

from deepj_b200.compute_graph import OP_Q8_LINEAR, OP_Q8_LINEAR_LN, OP_Q8_SWIGLU, float_bits
from test_q8_gpu import Dev

pytestmark = pytest.mark.gpu

SHAPES = [(32, 8), (96, 40), (128, 17), (160, 2400), (992, 24), (1024, 33), (1056, 1200), (1600, 4800), (4096, 72), (4128, 40), (8352, 16), (128, 40000)]


def dequantized(dev, q, K, N):
    codes, scales = dev.q8_download(q, K, N)
    return codes.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, axis=1)[:, :K]      # [N × K]


@pytest.mark.parametrize("K,N", SHAPES)
@pytest.mark.parametrize("M", [1, 2, 4])
def test_few_rows(K, N, M, off=0, pad=0):            # rows that start `off` values into their buffer and lie K + pad apart
    dev = Dev(9 << 20)
    try:
        rng = np.random.default_rng(K + N + M)
        x = rng.standard_normal((M, K)).astype(np.float32) + 0.3
        gamma, beta = rng.uniform(0.5, 1.5, K).astype(np.float32), rng.standard_normal(K).astype(np.float32)
        bias, res = rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
        q, q2 = (dev.q8((rng.standard_normal((K, N)) * 0.05).astype(np.float32)) for _ in range(2))
        w, w2 = dequantized(dev, q, K, N), dequantized(dev, q2, K, N)
        spaced = np.full(off + M * (K + pad), np.nan, np.float32)
        for m in range(M):
            spaced[off + m * (K + pad):][:K] = x[m]
        xb, gb, tb, bb, rb = (dev.buf(a.size, a) for a in (spaced, gamma, beta, bias, res))
        ob, ld = dev.buf(M * N), K + pad
        x64 = x.astype(np.float64)
        rms = x64 / np.sqrt((x64 ** 2).mean(1, keepdims=True) + 1e-5) * gamma
        mean = x64.mean(1, keepdims=True)
        ln = (x64 - mean) / np.sqrt(((x64 - mean) ** 2).mean(1, keepdims=True) + 1e-5) * gamma + beta

        def check(row, want, weights, what):
            # a digit is within 2^-22 of its block's largest value; 32-bit sums of K / 32 / 8 blocks per warp; activations are 1-Lipschitz or nearly so
            got = dev.get(ob, M * N).reshape(M, N)
            size = (np.abs(row).max(1, keepdims=True) * np.abs(weights).sum(1)[None]) * (2.0 ** -22 + K / 256 * 2.0 ** -24) + 1e-6 * (np.abs(want) + 4)
            assert (np.abs(got - want) <= 2 * size).all(), (what, np.abs(got - want).max())

        dev.flush([OP_Q8_LINEAR, xb, off, ld, -1, 0, q, -1, -1, 0, 0, ob, 0, N, M])
        check(x64, x64 @ w.T, w, "plain")
        dev.flush([OP_Q8_LINEAR, xb, off, ld, gb, float_bits(1e-5), q, bb, rb, 0, N, ob, 0, N, M])
        check(rms, rms @ w.T + bias + res, w, "rms")
        dev.flush([OP_Q8_LINEAR_LN, xb, off, ld, gb, tb, float_bits(1e-5), q, bb, -1, 0, 0, ob, 0, N, M, 1])
        z = ln @ w.T + bias
        check(ln, 0.5 * z * (1 + np.tanh(np.sqrt(2 / np.float64(np.float32(np.pi))) * (z + 0.044715 * z ** 3))), w, "layer norm and gelu")
        dev.flush([OP_Q8_SWIGLU, xb, off, ld, gb, float_bits(1e-5), q, bb, q2, -1, ob, 0, N, M])
        g, u = rms @ w.T + bias, rms @ w2.T
        check(rms * np.abs(u).max(), g / (1 + np.exp(-g)) * u, np.maximum(np.abs(w), np.abs(w2)) + np.abs(g).max() * np.abs(w2) / np.abs(u).max(), "gated pair")
    finally:
        dev.close()


# rows whose digits leave room for: a barrier every two tiles; two ring items; two rows of three (a pass of two, a pass of one); two items and one tile
@pytest.mark.parametrize("K,N,M", [(4096, 9600, 4), (11008, 5000, 2), (11008, 40, 3), (5632, 4744, 4)])
def test_rings_beside_several_rows(K, N, M):
    test_few_rows(K, N, M)


# rows that do not come in 16-byte pieces, up to the reduction lengths beyond the FMA kernel's; a block with an SM to itself (from about 24000)
@pytest.mark.parametrize("K,N,M,off,pad", [(128, 17, 4, 1, 1), (1056, 600, 1, 2, 0), (1600, 72, 2, 0, 1), (4096, 4800, 3, 3, 2), (11008, 40, 4, 0, 3), (16416, 24, 1, 1, 0),
                                           (24864, 17, 2, 1, 1), (24864, 17, 1, 0, 0), (24864, 9, 4, 0, 4), (52608, 8, 1, 0, 0)])
def test_rows_anywhere(K, N, M, off, pad):
    test_few_rows(K, N, M, off, pad)


@pytest.mark.parametrize("K", [1600, 2048])
def test_rows_of_tiny_values(K):
    """Values below 2^-106, whose digit scale has no 32-bit inverse: the scale's last place is 2^-127, and with the weights' scales a subnormal
    number of 12 bits or more."""
    dev = Dev(9 << 20)
    try:
        rng = np.random.default_rng(K)
        N, x = 40, (rng.standard_normal((2, K)) * 1e-33).astype(np.float32)
        gamma, q = rng.uniform(0.5, 1.5, K).astype(np.float32), dev.q8((rng.standard_normal((K, N)) * 0.05).astype(np.float32))
        w, ob = dequantized(dev, q, K, N), dev.buf(2 * N)
        for g, row in ((-1, x.astype(np.float64)), (dev.buf(K, gamma), x.astype(np.float64) / np.sqrt(1e-5) * gamma)):
            dev.flush([OP_Q8_LINEAR, dev.buf(x.size, x), 0, K, g, float_bits(1e-5), q, -1, -1, 0, 0, ob, 0, N, 2])
            assert (np.abs(dev.get(ob, 2 * N).reshape(2, N) - row @ w.T) <= 2.0 ** -11 * (np.abs(row) @ np.abs(w).T)).all()
    finally:
        dev.close()


def test_without_tensor_copies():
    """The setting that leaves the kernels on tensor copies out: the same rows, lengths beyond the FMA kernel's among them."""
    env = dict(os.environ, DEEPJ_CUDA_GEMV="cpasync")
    here = os.path.abspath(__file__)
    res = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-p", "no:cacheprovider", "-m", "gpu", here, "-k", "few_rows or rows_anywhere"], env=env,
                         capture_output=True, text=True, timeout=600, cwd=os.path.dirname(os.path.dirname(here)))
    assert res.returncode == 0 and f"{3 * len(SHAPES) + 10} passed" in res.stdout, res.stdout + res.stderr
