"""A pending read-back keeps the device buffer that it reads."""
import ctypes as C
import gc
from types import SimpleNamespace

import numpy as np
import pytest


def test_buffer_outlives_a_pending_read_back(monkeypatch):
    vkarray = pytest.importorskip("vulkpy_gb300.vkarray")
    events = []

    class Buf:
        ptr, nbytes, h2d_job = 4096, 16, None

        def __del__(self):
            events.append("freed")

    def d2h_async(h, dst, src, nbytes, job):
        C.cast(job, C.POINTER(C.c_void_p))[0] = 7
        return 0

    monkeypatch.setattr(vkarray, "lib", SimpleNamespace(
        vkc_d2h_async=d2h_async, vkc_job_wait=lambda j, t: events.append("copied") or 0, vkc_job_destroy=lambda j: 0))
    monkeypatch.setattr(vkarray, "_PinnedBlock", lambda nbytes, shape, dtype: np.zeros(shape, dtype))
    dev = SimpleNamespace(h=None, hv=0, capture=None, streams=[None])
    a = vkarray.Array.__new__(vkarray.Array)
    a._gpu, a.shape, a._size, a._buf = SimpleNamespace(_dev=dev), (4,), 4, Buf()
    a.prefetch()
    assert events == []
    del a
    gc.collect()
    assert events == ["copied", "freed"]
