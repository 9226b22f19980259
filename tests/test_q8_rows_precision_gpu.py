"""How close the many-row Q8 projection comes to 64 bits where shorter batches run as 32-bit sums (K no multiple of 128): no
further off than those, at any length."""
import numpy as np
import pytest

import oracle
from deepj_b200.compute_graph import OP_Q8_LINEAR
from test_q8_gpu import dev  # noqa: F401
from test_q8_rows_range_gpu import product

pytestmark = pytest.mark.gpu

# Relative 2-norm of the error: the activations' two halves, the two full-size accumulations in the tensor core (cut to 24 bits)
# and the running sums of eight blocks each leave less than 2^-24; independent, together below sqrt(3) 2^-24 < 2^-23 = 1.19e-7.
LIMIT = 2.0 ** -23


def exact_weights(dev, W):  # noqa: F811
    codes, scales = oracle.q8_quantize(W)
    K = W.shape[0]
    return dev.q8(W), (codes.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, axis=1)[:, :K]).T


@pytest.mark.parametrize("M,K,N", [(130, 688, 256), (64, 1392, 200), (200, 1600, 320), (700, 1600, 200), (64, 4128, 200), (150, 5648, 320), (300, 5616, 64),
                                   (20, 10992, 512)])
def test_error_does_not_grow_with_the_length(dev, M, K, N):  # noqa: F811
    rng = np.random.default_rng(M + K + N)
    q, W = exact_weights(dev, (rng.standard_normal((K, N)) * 0.02).astype(np.float32))
    x = rng.standard_normal((M, K)).astype(np.float32)
    got, want = product(dev, x, q, N), x.astype(np.float64) @ W
    assert np.linalg.norm(got - want) <= LIMIT * np.linalg.norm(want)


@pytest.mark.parametrize("K", [688, 1600, 2048])
def test_small_values_beside_a_large_one_keep_their_bits(dev, K):  # noqa: F811
    """One value of a row 2^22 times the others', against weights that are zero there: the others' 22 bits decide the result."""
    M, N = 150, 160
    rng = np.random.default_rng(K)
    w = (rng.standard_normal((K, N)) * 0.02).astype(np.float32)
    w[K - 9] = 0.0
    q, W = exact_weights(dev, w)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[:, K - 9] = 2.0 ** 22
    got, want = product(dev, x, q, N), x.astype(np.float64) @ W
    assert np.linalg.norm(got - want) <= (LIMIT if K % 128 else 2 * LIMIT) * np.linalg.norm(want)
