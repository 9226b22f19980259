"""Where a downloaded result lands: in the tensor's own array, whatever its layout, and nowhere else; an array that cannot take
the result is refused as it always was."""
import numpy as np
import pytest

from deepj_b200.tensor import Tensor
from test_stream_format import rt  # noqa: F401

WANT = np.arange(6, dtype=np.float32).reshape(2, 3)


def result(rt, data):  # noqa: F811
    rt.download_result = WANT
    t = Tensor(2, 3).neg()
    t.data = data
    return t


@pytest.mark.parametrize("make", [
    lambda: np.full((2, 3), 9.0, np.float32),
    lambda: np.full((3, 2), 9.0, np.float32).T,                              # column-major
    lambda: np.full((2, 8), 9.0, np.float32)[:, 1:7:2],                      # strided
    lambda: np.full((2, 3), 9.0, np.float64),
    lambda: np.full((2, 3), 9.0, ">f4"),
    lambda: np.full((1, 2, 3), 9.0, np.float32),
    lambda: np.frombuffer(bytearray(25), np.uint8)[1:].view(np.float32).reshape(2, 3),      # off a 4-byte boundary
])
def test_result_lands_in_the_array_at_hand(rt, make):  # noqa: F811
    data = make()
    base = data if data.base is None else data.base
    t = result(rt, data)
    t.materialize()
    assert t.data is data and np.array_equal(data.reshape(2, 3), WANT)
    if base.size > 6 and base.dtype == np.float32:
        assert np.all(base[:, 0::2] == 9.0)
    t.materialize()
    assert rt.calls.count("download") == 1


@pytest.mark.parametrize("make", [lambda: np.zeros((3, 2), np.float32), lambda: np.zeros(6, np.float32)])
def test_arrays_of_another_shape_are_refused(rt, make):  # noqa: F811
    t = result(rt, make())
    with pytest.raises(ValueError):
        t.materialize()


def test_read_only_arrays_are_refused_and_stay(rt):  # noqa: F811
    data = np.zeros((2, 3), np.float32)
    data.flags.writeable = False
    t = result(rt, data)
    with pytest.raises(ValueError):
        t.materialize()
    assert not data.any()
