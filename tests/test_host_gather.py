"""rr_host_gather (CPU): the concatenation of host arrays, at the sizes where
it starts to split over threads, with empty and one-byte parts; sizes that
do not fit are refused."""

import numpy as np
import pytest

from redrock_b200 import _lib


def _gather(parts, out, nbytes):
    src = np.array([p.ctypes.data if p.size else 0 for p in parts], dtype=np.uintp)
    size = np.array([p.nbytes for p in parts], dtype=np.int64)
    return _lib.lib().rr_host_gather(src.ctypes.data, size.ctypes.data, len(parts),
                                     out.ctypes.data, nbytes)


@pytest.mark.parametrize("sizes", [
    [1], [0, 5, 0], [(4 << 20) - 1], [4 << 20], [(4 << 20) + 1, 1], [1] * 100,
    [700001] * 60, [3, 64 << 20, 0, 5], [(2 << 20) + 63] * 17,
])
def test_gather_is_concatenation(sizes):
    rng = np.random.default_rng(len(sizes))
    parts = [rng.integers(0, 255, n, dtype=np.uint8) for n in sizes]
    total = sum(sizes)
    out = np.zeros(total + 16, dtype=np.uint8)
    assert _gather(parts, out, total) == _lib.RR_OK
    np.testing.assert_array_equal(out[:total], np.concatenate(parts))
    assert not out[total:].any()
    assert _gather(parts, out, total - 1) == _lib.RR_EINVAL


def test_gather_arguments():
    L = _lib.lib()
    assert L.rr_host_gather(None, None, 0, None, 0) == _lib.RR_OK
    assert L.rr_host_gather(None, None, 1, None, 8) == _lib.RR_EINVAL
    z = np.zeros(1, dtype=np.int64)
    neg = np.array([-1], dtype=np.int64)
    p = np.array([z.ctypes.data], dtype=np.uintp)
    assert L.rr_host_gather(p.ctypes.data, neg.ctypes.data, 1, z.ctypes.data, 8) == _lib.RR_EINVAL
