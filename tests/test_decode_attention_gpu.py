"""Decode attention (op 67) step by step against the plain chain in float64: positions below, at and above every border of the
rings (4 warps × 32 / (hd / 16) positions a round) and of the splits, 1 … 8 splits (merged inside a cluster) and more (merged
behind a ticket), both cache formats, sequences at unequal positions, a position that moves right before the op."""
import ctypes

import numpy as np
import pytest

from deepj_b200 import _lib
from deepj_b200.compute_graph import OP_ADD_SCALAR_INPLACE, OP_ATTN_DECODE, OP_ATTN_PREFILL, float_bits
from deepj_b200.decoder import rope_tables
from test_attn_prefill_gpu import reference
from test_q8_gpu import Dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [0, 1])
# head dim, cache rows (one split per 64), cached positions of the first sequence
@pytest.mark.parametrize("hd,max_seq,start", [(16, 40, 1), (32, 130, 63), (64, 70, 30), (64, 500, 127), (128, 60, 15), (128, 66, 33), (128, 640, 300), (256, 200, 70),
                                              (512, 140, 8), (64, 1300, 700)])
def test_steps(hd, max_seq, start, half, B=2, H=3, steps=5):
    dev = Dev(9 << 20)
    try:
        d, n = H * hd, min(start + 7, max_seq - steps - 1)               # cached positions: `start` and n
        rng = np.random.default_rng(hd + max_seq)
        L = n + steps
        qkv = rng.standard_normal((B, L, 3, H, hd)).astype(np.float32)
        qkv[:, :, 0] *= 2.0
        cos, sin = rope_tables(hd, max_seq)
        cb, sb = dev.buf(cos.size, cos), dev.buf(sin.size, sin)
        kv = dev.next
        dev.next += 1
        dev.owned.append(kv)
        _lib.check((dev.lib.deepj_cuda_kv_alloc_f16 if half else dev.lib.deepj_cuda_kv_alloc)(kv, 1, B, H, max_seq, hd))
        xb, pb = dev.buf(B * n * 3 * d, qkv[:, :n]), dev.buf(B, np.zeros(B))
        dev.flush([OP_ATTN_PREFILL, xb, 0, d, 2 * d, 3 * d, kv, 0, pb, cb, sb, dev.buf(B * n * d), 0, d, B, H, hd, n])
        at = [start if b % 2 == 0 else n for b in range(B)]
        pb = dev.buf(B, np.array(at, dtype=np.float32))
        cmd, outs = [], []
        for s in range(steps):                                           # one stream: the position moves between the ops
            rows = np.stack([qkv[b, at[b] + s] for b in range(B)]).reshape(B, 3 * d)
            outs.append(dev.buf(B * d))
            cmd += [OP_ATTN_DECODE, dev.buf(B * 3 * d, rows), 0, d, 2 * d, 3 * d, kv, 0, pb, cb, sb, outs[-1], 0, d, B, H, hd]
            cmd += [OP_ADD_SCALAR_INPLACE, pb, float_bits(1.0), B]
        dev.flush(cmd)
        for b in range(B):
            k, v = qkv[b, :, 1], qkv[b, :, 2]
            want = reference(qkv[b, :, 0], k, v, cos, sin)
            # outputs are convex combinations of N(0,1) values; half-precision keys move a score of deviation 2 by 2^-11 of it at most
            # a few times over, values by 2^-11
            tol = 6e-3 if half else 2e-5
            for s in range(steps):
                got = dev.get(outs[s], B * d).reshape(B, d)[b]
                assert np.abs(got - want[at[b] + s]).max() <= tol, (b, s)
        st = (ctypes.c_int64 * 6)()
        _lib.check(dev.lib.deepj_cuda_stats(st, 6))
        assert st[5] == 0
    finally:
        dev.close()


# three and six splits of so many heads that their clusters do not all fit onto the chip at once (187 and 93 do), and of fewer
@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("hd,max_seq,start,B,H", [(16, 192, 100, 24, 8), (64, 400, 300, 6, 16), (128, 192, 150, 10, 6)])
def test_clusters_that_fit_and_do_not(hd, max_seq, start, B, H, half):
    test_steps(hd, max_seq, start, half, B, H, 2)
