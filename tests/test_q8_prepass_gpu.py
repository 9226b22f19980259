"""The pass that leaves normalised, scaled and split activation rows for the many-row Q8 product: rows of one to six chunks of eight values per
thread (2048 values each), not all of them filled, and longer ones, plain, with RMSNorm and with LayerNorm, against float64."""
import ctypes

import numpy as np
import pytest

from deepj_b200 import _lib
from deepj_b200.compute_graph import OP_Q8_LINEAR, OP_Q8_LINEAR_LN, float_bits
from test_q8_gpu import dev  # noqa: F401
from test_q8_rows_gpu import check, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [480, 512, 2048, 2080, 4128, 6400, 8192, 8224, 12288, 12320, 14336])
def test_rows_of_every_length(dev, K):  # noqa: F811
    rng = np.random.default_rng(K)
    M, N = 300, 72
    out = (ctypes.c_int32 * 3)()
    _lib.check(dev.lib.deepj_cuda_q8_route(M, K, N, 0, out))
    assert out[0] == 1
    q, W = weights(dev, rng, K, N)
    x = rng.standard_normal((M, K)).astype(np.float32) + 0.3
    g, t = rng.uniform(0.5, 1.5, K).astype(np.float32), rng.standard_normal(K).astype(np.float32)
    xb, gb, tb, ob = dev.buf(M * K, x), dev.buf(K, g), dev.buf(K, t), dev.buf(M * N)
    xd = x.astype(np.float64)
    rms = xd / np.sqrt((xd ** 2).mean(1, keepdims=True) + 1e-5) * g
    ln = (xd - xd.mean(1, keepdims=True)) / np.sqrt(xd.var(1, keepdims=True) + 1e-5) * g + t
    for cmd, row in (([OP_Q8_LINEAR, xb, 0, K, -1, 0], xd), ([OP_Q8_LINEAR, xb, 0, K, gb, float_bits(1e-5)], rms),
                     ([OP_Q8_LINEAR_LN, xb, 0, K, gb, tb, float_bits(1e-5)], ln)):
        dev.flush(cmd + [q, -1, -1, 0, 0, ob, 0, N, M] + ([0] if cmd[0] == OP_Q8_LINEAR_LN else []))
        check(dev.get(ob, M * N).reshape(M, N), row @ W, K)
