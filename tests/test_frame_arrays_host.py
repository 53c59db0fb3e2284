"""The arrays an output frame is handed out in (_lib._frame_arrays), with the
library's calls replaced: over the buffer itself, given back once with the last
array over it, or the caller's own copies where it cannot be handed over."""
import ctypes
import gc
import os

import numpy as np
import pytest

from anuga_core_gb300 import _lib

FP = ctypes.POINTER(ctypes.c_float)


class _Library:
    def __init__(self, n, refuse):
        self.buffer = np.arange(n, dtype=np.float32)
        self.refuse, self.given = refuse, []

    def _at(self, k):
        return ctypes.cast(self.buffer.ctypes.data + 4 * k, FP)

    def take(self, handle, out):
        if self.refuse:
            return _lib.E_NOMEM
        ctypes.cast(out, ctypes.POINTER(FP))[0] = self._at(0)
        return 0

    def wait(self, P, handle, v, c):
        ctypes.cast(v, ctypes.POINTER(FP))[0] = self._at(0)
        ctypes.cast(c, ctypes.POINTER(FP))[0] = self._at(3 * P)
        return 0

    def agx_frame_give(self, p):
        self.given.append(ctypes.cast(p, ctypes.c_void_p).value)


@pytest.mark.parametrize("P,N", [(0, 1), (5, 4), (60, 100)])
@pytest.mark.parametrize("refuse", [False, True])
def test_frame_arrays(monkeypatch, P, N, refuse):
    L = _Library(3 * P + 3 * N, refuse)
    monkeypatch.setattr(_lib, "load", lambda: L)
    want = L.buffer.copy()
    v, c = _lib._frame_arrays(L.take, lambda *a: L.wait(P, *a), (None,), P, N)
    assert v.shape == (3, P) and c.shape == (3, N) and v.dtype == c.dtype == np.float32
    assert np.array_equal(np.concatenate([v.ravel(), c.ravel()]), want)
    assert np.shares_memory(c, L.buffer) != refuse
    c[:] = -1.0                                   # writable, and the caller's own
    assert np.array_equal(L.buffer, want) == refuse
    part = c[1:2]
    del v, c
    gc.collect()
    assert not L.given                            # an array over it is still there
    del part
    gc.collect()
    assert L.given == ([] if refuse else [L.buffer.ctypes.data])


def test_a_forked_process_gives_nothing_back(monkeypatch):
    L = _Library(6, False)
    monkeypatch.setattr(_lib, "load", lambda: L)
    v, c = _lib._frame_arrays(L.take, None, (None,), 1, 1)
    here = os.getpid()
    monkeypatch.setattr(os, "getpid", lambda: here + 1)      # its copy of the arrays goes
    del v, c
    gc.collect()
    assert not L.given
