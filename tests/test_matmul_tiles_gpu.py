"""The fp32 product is bit for bit the reference's loop (ascending k, one rounding for the multiply, one for the add), also
where it runs in 64 x 64 tiles: tile edges, short and ragged k."""
import numpy as np
import pytest

from deepj_b200.compute_graph import OP_MATMUL
from test_q8_gpu import dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(640, 640, 64), (641, 577, 33), (1024, 1000, 1), (63, 6400, 17), (5000, 65, 16), (700, 512, 15), (64, 64, 40), (1, 4736, 31)])
def test_bit_exact(dev, m, n, k):  # noqa: F811
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    a[0, 0] = np.float32(-0.0)
    want = np.zeros((m, n), dtype=np.float32)
    for i in range(k):
        want = want + a[:, i:i + 1] * b[i:i + 1]
    ob = dev.buf(m * n)
    dev.flush([OP_MATMUL, dev.buf(m * k, a), dev.buf(k * n, b), ob, m, n, k])
    got = dev.get(ob, m * n).reshape(m, n)
    assert np.array_equal(got, want) and np.array_equal(np.signbit(got), np.signbit(want))
