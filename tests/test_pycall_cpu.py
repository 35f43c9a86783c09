"""The Python extension behind Context's list calls (redzone_b200/pycall.c), with a callback in the
place of the library's functions: what it passes, what it returns, what it refuses."""
import ctypes
import importlib.machinery
import subprocess
import sys

import numpy as np
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


class Buffer:
    """Device memory of another owner: what Context's list calls ask of a tensor, and no more."""

    def __init__(self, shape, numel, itemsize=4, at=0x1000):
        self.shape, self._numel, self._itemsize, self._at = shape, numel, itemsize, at

    def data_ptr(self):
        return self._at

    def element_size(self):
        return self._itemsize

    def numel(self):
        return self._numel


@pytest.mark.parametrize("shape", [[7, 2], np.array([7, 2]), (np.int64(7), 2), torch.Size([7, 2])])
def test_list_call_takes_any_sequence_and_integer(shape):
    seen = []

    @FN
    def fn(ctx, data, n, elem, idx, k, new_len, flags, stream):
        seen.append((data, n, elem, idx, k))
        new_len[0] = n - k
        return 0

    addr = ctypes.cast(fn, ctypes.c_void_p).value
    got = rzcall.call(addr, 1, Buffer(shape, 14), Buffer([3], np.int64(3), at=0x2000), 0, 1)
    assert got == 4 and seen == [(0x1000, 7, 8, 0x2000, 3)]
    for bad, error in ((Buffer([], 0), IndexError), (Buffer([2.5, 2], 5), TypeError), (Buffer(7, 7), TypeError)):
        with pytest.raises(error):
            rzcall.call(addr, 1, bad, Buffer([3], 3), 0, 1)
    assert len(seen) == 1


def test_list_call_without_a_bound_stream_is_an_error():
    code = ("import torch\nfrom redzone_b200 import _native\nm = _native.load_pycall()\n"
            "t = torch.zeros(4, dtype=torch.int32)\n"
            "try:\n    m.call(1, 1, t, t, 0, None)\nexcept RuntimeError as e:\n    print('refused', e)\n")
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=_native.PKG.parent)
    assert out.returncode == 0 and "refused" in out.stdout, out


def test_extension_is_named_for_its_interpreter_and_left_out_without_a_compiler(monkeypatch, tmp_path):
    """Another Python does not find this one's extension (a name without its binary interface would load
    there), and a build without a C compiler goes on without it."""
    from redzone_b200 import build
    assert build.PYCALL == _native.PYCALL_PATH
    assert build.PYCALL.name == "_rzcall" + importlib.machinery.EXTENSION_SUFFIXES[0] != "_rzcall.so"
    monkeypatch.setattr(build, "PYCALL", tmp_path / build.PYCALL.name)
    monkeypatch.setenv("PATH", str(tmp_path))
    assert build.build_pycall(quiet=True) is None
    monkeypatch.setattr(_native, "PYCALL_PATH", tmp_path / "_rzcall.cpython-300-x86_64-linux-gnu.so")
    assert _native.load_pycall() is None
