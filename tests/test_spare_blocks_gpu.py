"""Device blocks of released float buffers that the library keeps: a block handed on reads as zeros, the kept ones are bounded in
bytes and in number, and an allocation that fails gives all of them back first."""
import ctypes

import numpy as np
import pytest

from deepj_b200 import _lib

pytestmark = pytest.mark.gpu

MIB = 1 << 20
FIRST = 7 << 20


@pytest.fixture()
def lib():
    h = _lib.load()
    _lib.check(h.deepj_cuda_init(0))
    yield h
    h.deepj_cuda_tp_destroy()


def ints(values):
    return (ctypes.c_int32 * len(values))(*values)


def alloc(lib, ids, floats):
    _lib.check(lib.deepj_cuda_alloc_buffers(ints(ids), ints([floats] * len(ids)), len(ids)))


def release(lib, ids):
    _lib.check(lib.deepj_cuda_release_buffers(ints(ids), len(ids)))


def kept(lib):
    """(bytes, blocks) held for later buffers."""
    st = (ctypes.c_int64 * 8)()
    _lib.check(lib.deepj_cuda_stats(st, 8))
    return st[6], st[7]


@pytest.mark.parametrize("floats", [1, 128, 129, 5 * MIB])
def test_a_block_handed_on_reads_as_zeros(lib, floats):
    alloc(lib, [FIRST], floats)
    data = np.full(floats, 7.0, np.float32)
    _lib.check(lib.deepj_cuda_upload_buffer(FIRST, data.ctypes.data, floats))
    release(lib, [FIRST])
    held = kept(lib)
    alloc(lib, [FIRST + 1], floats)
    now = kept(lib)
    assert held[1] - now[1] == 1 and held[0] - now[0] == (4 * floats + 511) // 512 * 512
    _lib.check(lib.deepj_cuda_download_buffer(FIRST + 1, data.ctypes.data, floats))
    release(lib, [FIRST + 1])
    assert not data.any()


def test_bounds(lib):
    ids = [FIRST + i for i in range(5000)]
    alloc(lib, ids, 3)
    release(lib, ids)
    assert kept(lib)[1] <= 4096
    big = ids[:6]
    alloc(lib, big, 15 * MIB)                     # 60 MiB each
    release(lib, big)
    held = kept(lib)
    assert 240 * MIB <= held[0] <= 256 * MIB      # four of them; what came before went first
    alloc(lib, big[:1], 16 * MIB + 1)             # more than 64 MiB: never kept
    release(lib, big[:1])
    assert kept(lib) == held


def test_an_allocation_that_fails_gives_the_blocks_back(lib):
    handle = ctypes.create_string_buffer(64)
    for refused in (lambda: lib.deepj_cuda_q8_alloc(FIRST, 1 << 30, 1 << 14), lambda: lib.deepj_cuda_tp_create(0, 2, 1 << 44, handle)):
        alloc(lib, [FIRST + 1], 1000)
        release(lib, [FIRST + 1])
        assert kept(lib)[1] > 0
        assert refused() != 0 and b"memory" in lib.deepj_cuda_last_error()
        assert kept(lib) == (0, 0)
