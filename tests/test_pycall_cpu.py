"""The Python extension behind Context's list calls (redzone_b200/pycall.c), with a callback in the
place of the library's functions: what it passes, what it returns, what it refuses."""
import ctypes

import pytest
import torch

from redzone_b200 import _native

rzcall = _native.load_pycall()
pytestmark = pytest.mark.skipif(rzcall is None, reason="built without Python's headers")

FN = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_uint32, ctypes.c_void_p,
                      ctypes.c_int64, ctypes.POINTER(ctypes.c_int64), ctypes.c_uint32, ctypes.c_void_p)


@pytest.mark.parametrize("shape,w", [((7,), 4), ((7, 2), 8), ((5, 2, 2), 16), ((0, 8), 32)])
@pytest.mark.parametrize("status", [0, 1, 8])
def test_list_call_passes_sizes_and_returns_length_or_status(shape, w, status):
    seen = []

    @FN
    def fn(ctx, data, n, elem, idx, k, new_len, flags, stream):
        seen.append((ctx, data, n, elem, idx, k, flags, stream))
        new_len[0] = n - k
        return status

    addr = ctypes.cast(fn, ctypes.c_void_p).value
    data, idx = torch.zeros(shape, dtype=torch.int32), torch.zeros(3, dtype=torch.int32)
    got = rzcall.call(addr, 0x1234, data, idx, 0x80000003, 0x77)
    assert got == (shape[0] - 3 if status == 0 else -status) or (status == 0 and shape[0] < 3)
    assert seen == [(0x1234, data.data_ptr() or None, shape[0], w, idx.data_ptr(), 3, 0x80000003, 0x77)]


def test_list_call_looks_the_stream_up_and_refuses_what_has_no_sizes():
    seen = []

    @FN
    def fn(ctx, data, n, elem, idx, k, new_len, flags, stream):
        seen.append((ctx, stream))
        new_len[0] = n
        return 0

    addr = ctypes.cast(fn, ctypes.c_void_p).value
    data, idx = torch.zeros(4, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    rzcall.bind(lambda: 3, lambda d: 0x50 + d)
    assert rzcall.call(addr, 0, data, idx, 0, None) == 4
    assert seen == [(None, 0x53)]  # a closed context is a null pointer, which the library refuses
    with pytest.raises(IndexError):
        rzcall.call(addr, 0, torch.zeros((), dtype=torch.int32), idx, 0, 1)
    with pytest.raises(AttributeError):
        rzcall.call(addr, 0, data, [1, 2], 0, 1)
    with pytest.raises(TypeError):
        rzcall.call(addr, 0, data, idx, 0)
    assert len(seen) == 1
