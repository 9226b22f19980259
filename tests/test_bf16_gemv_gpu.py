"""The ring kernel of 1-16 rows: sizes at the edges of its items (1024 columns), row groups (two or four rows), blocks (one per
SM), rings and staging pieces, against the product in float64."""
import os
import subprocess
import sys

import numpy as np
import pytest

from deepj_b200 import _lib
from deepj_b200.compute_graph import OP_BF16_LINEAR_SUM, OP_TABLE_EXPERTS, float_bits
from test_bf16_ops_gpu import bf16, dev  # noqa: F401

pytestmark = pytest.mark.gpu


# K: below a piece of a warp, an item less and more one unit, rows of which half an SM holds two and one ring items, a whole SM; four
# rows beside rings of half of the warps and of fewer, which go two by two; odd tails
# N: fewer rows than warps or blocks, one row group more than the blocks, many groups per warp
@pytest.mark.parametrize("K,N", [(8, 2), (8, 8), (24, 594), (1016, 298), (1024, 296), (1032, 2368), (2048, 66), (3000, 40), (4104, 304), (9000, 26), (11840, 26), (13312, 18), (20001, 18),
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


# slots so many that two or four weight rows per item leave their padded rows no room (eight of 256 columns), up to the widest output whose sums still fit
@pytest.mark.parametrize("M,k,d,ff,top", [(2, 72, 40, 8, 110), (1, 64, 24, 16, 180), (7, 16, 49152, 8, 195)])
def test_experts_of_many_slots(dev, M, k, d, ff, top):  # noqa: F811
    rng = np.random.default_rng(top + d)
    vocab = 5
    x, tok = rng.standard_normal((M, k)).astype(np.float32), rng.integers(0, vocab, M)
    table = np.stack([rng.permutation(top) for _ in range(vocab)])
    up, down = bf16(rng.standard_normal((top * 2 * ff, k)) * 0.3), bf16(rng.standard_normal((d, ff)) * 0.3)      # one down matrix for all experts
    res = rng.standard_normal((M, d)).astype(np.float32)
    U, W = dev.weight(k, top * 2 * ff, [(up, 0, 1, 0)]), dev.new()
    _lib.check(dev.lib.deepj_cuda_bf16_alloc(W, ff, top * d))
    src = dev.buf(down.size, down)
    for e in range(top):
        _lib.check(dev.lib.deepj_cuda_bf16_store(W, e * d, 1, 0, src, 0, d, ff))
    out = dev.buf(M * d)
    dev.flush([OP_TABLE_EXPERTS, dev.buf(x.size, x), 0, k, -1, 0, float_bits(0.0), dev.buf(M, tok), dev.buf(table.size, table), vocab, top, top, U, W, ff,
               float_bits(7.0), dev.buf(res.size, res), 0, d, out, 0, d, d, M, 1])
    pairs = (x.astype(np.float64) @ up.T.astype(np.float64)).reshape(M, top, ff, 2)
    g, u = np.minimum(pairs[..., 0], 7.0), np.clip(pairs[..., 1], -7.0, 7.0)
    y = g / (1 + np.exp(-1.702 * g)) * (u + 1)                       # [M, expert, ff]; every token names every expert
    want = res + y.mean(1) @ down.T.astype(np.float64)
    # fp32 chains of top · 8 / 32 ... products per lane and the warps' sums, of terms that add up to `size`; the gated values are good to 2^-21
    size = np.abs(y).mean(1) @ np.abs(down).T.astype(np.float64) + np.abs(res)
    assert (np.abs(dev.get(out, M * d).reshape(M, d) - want) <= (2.0 ** -21 + 2.0 ** -24 * (top / 4 + 40)) * size).all()


def test_without_tensor_copies():
    """The setting that leaves the kernels on tensor copies out, as a driver without tensor maps would: these rows, and table-routed experts."""
    env = dict(os.environ, DEEPJ_CUDA_GEMV="cpasync")
    here = os.path.abspath(__file__)
    files = [here, os.path.join(os.path.dirname(here), "test_bf16_ops_gpu.py")]
    res = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-p", "no:cacheprovider", "-m", "gpu", *files, "-k", "ring_kernel or experts or test_linear"],
                         env=env, capture_output=True, text=True, timeout=600, cwd=os.path.dirname(os.path.dirname(here)))
    assert res.returncode == 0 and " passed" in res.stdout and "skipped" not in res.stdout, res.stdout + res.stderr
