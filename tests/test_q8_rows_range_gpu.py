"""The many-row Q8 projection on rows whose magnitudes lie at the ends of the fp32 range, for reduction lengths that are and are
not whole scale blocks: results are those of 32-bit arithmetic, not a question of which kernel a row count selects."""
import numpy as np
import pytest

import oracle
from deepj_b200 import _lib
from deepj_b200.compute_graph import OP_Q8_LINEAR
from test_q8_gpu import dev  # noqa: F401
from test_q8_rows_gpu import bound, weights

pytestmark = pytest.mark.gpu

MAXIMA = (1.0, 1e-36, 1e-37, 1e-40, 1e-43, 0.0, 1e30, 1e32, 2e37)      # 2e37 times a column's weights stays finite


def product(dev, x, q, N):  # noqa: F811
    M, K = x.shape
    ob = dev.buf(M * N)
    dev.flush([OP_Q8_LINEAR, dev.buf(M * K, x), 0, K, -1, 0, q, -1, -1, 0, 0, ob, 0, N, M])
    return dev.get(ob, M * N).reshape(M, N).astype(np.float64)


@pytest.mark.parametrize("M,K,N", [(40, 256, 300), (300, 688, 130), (300, 128, 96), (96, 1600, 70)])
def test_rows_of_every_magnitude(dev, M, K, N):  # noqa: F811
    rng = np.random.default_rng(M + K)
    q, W = weights(dev, rng, K, N)
    x = rng.uniform(-1.0, 1.0, (M, K))
    x[:, K // 2] = 1.0                                                     # the row's largest value
    x[:, 3:K // 2:5] = 0.0
    top = np.asarray([MAXIMA[m % len(MAXIMA)] for m in range(M)])
    x = (x * top[:, None]).astype(np.float32)
    got, want = product(dev, x, q, N), x.astype(np.float64) @ W
    # a subnormal result is rounded to a multiple of 2^-149, and so may be each of its products
    room = bound(K) * np.linalg.norm(want, axis=1) + np.sqrt(N) * (K + 1) * 2.0 ** -149
    assert np.all(np.isfinite(got))
    assert np.all(np.linalg.norm(got - want, axis=1) <= room)


@pytest.mark.parametrize("M,K,N", [(40, 256, 300), (300, 688, 130), (96, 1600, 70)])
def test_infinities_and_nan_stay_in_their_rows(dev, M, K, N):  # noqa: F811
    """One infinity times a code is an infinity of the code's sign, and NaN where the code is zero; a NaN spoils its row."""
    rng = np.random.default_rng(M * K)
    q, W = weights(dev, rng, K, N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    plain = x.astype(np.float64) @ W
    x[1, 5], x[2, K - 1], x[4, 0] = np.inf, -np.inf, np.nan
    got = product(dev, x, q, N)
    for m, k, sign in ((1, 5, 1.0), (2, K - 1, -1.0)):
        zero = W[k] == 0.0
        assert np.all(np.isnan(got[m]) == zero) and np.array_equal(got[m][~zero], np.where(W[k] > 0, np.inf, -np.inf)[~zero] * sign)
    assert np.all(np.isnan(got[4]))
    rest = [m for m in range(M) if m not in (1, 2, 4)]
    assert np.linalg.norm(got[rest] - plain[rest]) <= bound(K) * np.linalg.norm(plain[rest])


@pytest.mark.parametrize("size", [1e-6, 0.02, 1e5])
def test_the_coarse_settings_take_weights_of_any_size(dev, size):  # noqa: F811
    """deepj_cuda_tc_configure without bit 1 rounds the block scales to 11 bits, whatever their size: an error of at most 2^-11."""
    M, K, N = 300, 512, 160
    rng = np.random.default_rng(3)
    W = (rng.standard_normal((K, N)) * size).astype(np.float32)
    q, Wq = dev.q8(W), oracle.q8_dequantize(*oracle.q8_quantize(W)).astype(np.float64)
    x = rng.standard_normal((M, K)).astype(np.float32)
    try:
        _lib.check(dev.lib.deepj_cuda_tc_configure(1))
        got = product(dev, x, q, N)
    finally:
        _lib.check(dev.lib.deepj_cuda_tc_configure(3))
    want = x.astype(np.float64) @ Wq
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert 2.0 ** -15 < err <= 2.0 ** -11
