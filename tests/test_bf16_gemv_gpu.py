"""The ring kernel of 1-16 rows: sizes at the edges of its items (1024 columns), row groups (two or four rows), blocks (one per
SM), rings and staging pieces, against the product in float64."""
import os
import subprocess
import sys

import numpy as np
import pytest

from deepj_b200.compute_graph import OP_BF16_LINEAR_SUM, float_bits
from test_bf16_ops_gpu import bf16, dev  # noqa: F401

pytestmark = pytest.mark.gpu


# K: below a piece of a warp, an item less and more one unit, rows of which half an SM holds two and one ring items, a whole SM; odd tails
# N: fewer rows than warps or blocks, one row group more than the blocks, many groups per warp
@pytest.mark.parametrize("K,N", [(8, 2), (8, 8), (24, 594), (1016, 298), (1024, 296), (1032, 2368), (2048, 66), (3000, 40), (4104, 304), (9000, 26), (20001, 18),
                                 (50000, 10), (264, 20000)])
@pytest.mark.parametrize("M", [1, 2, 3, 7])
def test_ring_kernel(dev, K, N, M):  # noqa: F811
    rng = np.random.default_rng(K * 7 + N + M)
    w = bf16(rng.standard_normal((N, K)) * 0.05)
    x, base = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((M, K)).astype(np.float32)
    gamma, bias = rng.uniform(0.5, 1.5, K).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    groups = 4 if K % 32 == 0 else 1
    xi, bi, gi, bb, ri = (dev.buf(a.size, a) for a in (x, base, gamma, bias, res))
    out, total, W = dev.buf(M * N), dev.buf(M * K), dev.weight(K, N, [(w, 0, 1, 0)])
    norm = x.astype(np.float64).reshape(M, groups, -1)
    norm = (norm / np.sqrt((norm ** 2).mean(-1, keepdims=True) + 1e-5)).reshape(M, K) * gamma
    for normed in (False, True):                     # a plain row; the normed row (added to a base) with every part of the epilogue
        summed = normed and groups == 1
        row = base + 0.5 * norm if summed else norm if normed else x.astype(np.float64)
        cmd = [OP_BF16_LINEAR_SUM, xi, 0, K, gi if normed else -1, groups if normed else 0, float_bits(1e-5), -1, 0, 0, K, -1, 0, 0, W,
               ri if normed else -1, 0, N, out, 0, N, M, N, float_bits(0.0), -1, 0, 0, float_bits(0.0), 1, bb if normed else -1, 1]
        dev.flush(cmd + ([bi, 0, K, float_bits(0.5), total, 0, K] if summed else [-1, 0, 0, float_bits(0.0), -1, 0, 0]))
        want = row @ w.astype(np.float64).T + ((bias + res) if normed else 0.0)
        # fp32 products and sums: a rounding of 2^-24 per term of a chain no longer than K / 32, and of the norm and the epilogue
        size = np.abs(row) @ np.abs(w).astype(np.float64).T + 8.0
        got = dev.get(out, M * N).reshape(M, N)
        assert (np.abs(got - want) <= 2.0 ** -24 * (K / 32 + 24) * size).all(), (normed, np.abs(got - want).max())
        if summed:
            assert np.allclose(dev.get(total, M * K).reshape(M, K), row, rtol=1e-5, atol=1e-5)


def test_without_tensor_copies():
    """The setting that leaves the kernels on tensor copies out, as a driver without tensor maps would: these rows, and table-routed experts."""
    env = dict(os.environ, DEEPJ_CUDA_GEMV="cpasync")
    here = os.path.abspath(__file__)
    files = [here, os.path.join(os.path.dirname(here), "test_bf16_ops_gpu.py")]
    res = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-p", "no:cacheprovider", "-m", "gpu", *files, "-k", "ring_kernel or experts or test_linear"],
                         env=env, capture_output=True, text=True, timeout=600, cwd=os.path.dirname(os.path.dirname(here)))
    assert res.returncode == 0 and " passed" in res.stdout and "skipped" not in res.stdout, res.stdout + res.stderr
