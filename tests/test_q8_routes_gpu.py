"""Which kernel rows of a Q8 projection go to, and the many-row kernel at every tile width and split that its plan takes: rows and
columns that fill no tile, reductions with and without totals, of odd block counts and of no whole block, pairs, and LayerNorm with
GELU.  The plan's choice is asserted, so that a case keeps testing what it names (148 SMs)."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from deepj_b200 import _lib
from deepj_b200.compute_graph import OP_Q8_LINEAR, OP_Q8_LINEAR_LN, OP_Q8_SWIGLU, float_bits
from test_q8_gpu import dev  # noqa: F401
from test_q8_rows_gpu import check, weights

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def route(dev, M, K, N, pair=False):  # noqa: F811
    out = (ctypes.c_int32 * 3)()
    _lib.check(dev.lib.deepj_cuda_q8_route(M, K, N, int(pair), out))
    return tuple(out)


# rows, K, N, tile rows, splits
@pytest.mark.parametrize("M,K,N,nt,splits", [
    (6, 1600, 1600, 16, 4), (17, 688, 4800, 32, 2), (700, 1392, 33, 32, 4), (257, 4096, 33, 32, 8), (97, 100, 4800, 64, 1), (129, 2080, 2050, 64, 2),
    (200, 288, 4800, 96, 1), (200, 100, 4800, 96, 1), (257, 1392, 2050, 96, 2), (300, 288, 4800, 128, 1), (300, 100, 4800, 128, 1), (300, 64, 4800, 128, 1)])
def test_plain(dev, M, K, N, nt, splits):  # noqa: F811
    assert route(dev, M, K, N) == (1, nt, splits)
    rng = np.random.default_rng(M + K + N)
    q, W = weights(dev, rng, K, N)
    x, b, r = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), N, (M, N)))
    ob = dev.buf(M * N)
    dev.flush([OP_Q8_LINEAR, dev.buf(M * K, x), 0, K, -1, 0, q, dev.buf(N, b), dev.buf(M * N, r), 0, N, ob, 0, N, M])
    check(dev.get(ob, M * N).reshape(M, N), x.astype(np.float64) @ W + b + r, K)


@pytest.mark.parametrize("M,K,N,nt,splits", [(33, 288, 4800, 64, 1), (65, 2048, 1000, 64, 4), (65, 288, 4800, 96, 1), (385, 4096, 333, 96, 4),
                                             (97, 288, 4800, 128, 1), (97, 100, 4800, 128, 1)])
def test_pairs(dev, M, K, N, nt, splits):  # noqa: F811
    assert route(dev, M, K, N, True) == (1, nt, splits)
    rng = np.random.default_rng(M + K + N)
    (q1, W1), (q2, W2) = weights(dev, rng, K, N), weights(dev, rng, K, N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    ob = dev.buf(M * N)
    dev.flush([OP_Q8_SWIGLU, dev.buf(M * K, x), 0, K, -1, float_bits(1e-6), q1, -1, q2, -1, ob, 0, N, M])
    a = x.astype(np.float64) @ W1
    check(dev.get(ob, M * N).reshape(M, N), a / (1.0 + np.exp(-a)) * (x.astype(np.float64) @ W2), K)


@pytest.mark.parametrize("M,K,N,nt", [(97, 288, 4800, 64), (200, 288, 4800, 96), (300, 288, 4800, 128)])
def test_layernorm_and_gelu(dev, M, K, N, nt):  # noqa: F811
    assert route(dev, M, K, N) == (1, nt, 1)
    rng = np.random.default_rng(M + K)
    q, W = weights(dev, rng, K, N)
    x, g, b, c = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), K, K, N))
    ob = dev.buf(M * N)
    dev.flush([OP_Q8_LINEAR_LN, dev.buf(M * K, x), 0, K, dev.buf(K, g), dev.buf(K, b), float_bits(1e-5), q, dev.buf(N, c), -1, 0, 0, ob, 0, N, M, 1])
    xd = x.astype(np.float64)
    v = ((xd - xd.mean(1, keepdims=True)) / np.sqrt(xd.var(1, keepdims=True) + 1e-5) * g + b) @ W + c
    check(dev.get(ob, M * N).reshape(M, N), 0.5 * v * (1.0 + np.tanh(np.sqrt(2.0 / np.pi) * (v + 0.044715 * v ** 3))), K)


def test_rows_stay_with_the_faster_kernel(dev):  # noqa: F811
    """Both sides of each line: the head of sixteen sequences, short reductions of no whole block, and what lies beyond."""
    assert [route(dev, M, 4096, 32000)[0] for M in (8, 12, 16, 24, 300)] == [0, 0, 0, 1, 1]
    assert [route(dev, M, 688, 256)[0] for M in (4, 8, 32, 128)] == [0, 0, 0, 1]
    assert [route(dev, M, 5648, 2048)[0] for M in (4, 6, 64)] == [0, 1, 1]
    assert route(dev, 64, 690, 256)[0] == 0                       # rows of this kernel are multiples of 16 bytes


def test_normalised_rows_without_the_many_row_kernel():
    """The passes of the 16-row kernels behind a normalising pass, and the FMA kernel: where the many-row kernel is faster it takes
    their rows, so they are tested with it switched off."""
    env = dict(os.environ, DEEPJ_CUDA_NO_TC="1")
    res = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-p", "no:cacheprovider", "-m", "gpu", os.path.join(HERE, "test_gpt_decoder_gpu.py"), "-k",
                          "test_layernorm_q8_linear_gelu"], env=env, capture_output=True, text=True, timeout=600, cwd=os.path.dirname(HERE))
    assert res.returncode == 0 and "20 passed" in res.stdout, res.stdout + res.stderr
