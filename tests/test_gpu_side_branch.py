"""The side branch is the calling thread's: other threads' calls go on to the
device's stream, in order with the rest of their work."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_thread(f):
    out = []
    t = threading.Thread(target=lambda: out.append(f()))
    t.start()
    t.join(60)
    assert not t.is_alive() and out
    return out[0]


def _stream(gpu):
    from vulkpy_gb300 import _lib
    s = C.c_void_p()
    assert _lib.lib.vkc_device_stream(gpu.handle, C.byref(s)) == 0
    return s.value


def test_branch_of_one_thread_only(gpu):
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib
    lib, h = _lib.lib, gpu.handle
    own = _stream(gpu)
    x = vk.Array(gpu, data=np.arange(1000, dtype=np.float32))
    assert lib.vkc_side_begin(h) == 0
    try:
        branch = _stream(gpu)
        assert branch != own
        assert _in_thread(lambda: _stream(gpu)) == own
        got = _in_thread(lambda: np.asarray(x + 1.0))
        assert _in_thread(lambda: lib.vkc_side_end(h)) == _lib.ERR_INVALID   # not that thread's branch
        assert _stream(gpu) == branch
    finally:
        assert lib.vkc_side_end(h) == 0
    assert _stream(gpu) == own
    np.testing.assert_array_equal(got, np.arange(1000, dtype=np.float32) + 1)


def test_deferral_of_one_thread_only(gpu):
    """Another thread's Dense backward is joined before it returns while this
    thread defers its joins: its gradients are in order on the device's
    stream."""
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib
    lib, h = _lib.lib, gpu.handle
    rng = np.random.default_rng(0)
    b, i, o = 512, 300, 16      # no scratch on the main stream, whose reuse could order it after the branch
    x, w, dy = (rng.standard_normal(s).astype(np.float32) for s in ((b, i), (o, i), (b, o)))
    ax, aw, ady = (vk.Array(gpu, data=v) for v in (x, w, dy))
    dx, dw, db = vk.Array(gpu, shape=(b, i)), vk.Array(gpu, shape=(o, i)), vk.Array(gpu, shape=(o,))
    pdw = dw._buf.ptr
    big = vk.zeros(gpu, shape=(8192, 8192))

    def backward_and_read():
        st = lib.vkc_dense_backward_ex(h, _lib.MM_FP32, ax._dptr(), aw._dptr(), ady._dptr(), None, _lib.ACT_NONE, None,
                                       dx._buf.ptr, pdw, db._buf.ptr, b, i, o, 0)
        out = np.empty((o, i), np.float32)
        return st, lib.vkc_d2h(h, out.ctypes.data, pdw, out.nbytes), out

    big @ big                                  # every kernel loaded (that waits for running ones)
    backward_and_read()
    dw[:] = np.zeros((o, i), np.float32)
    assert dw._dptr() == pdw
    gpu.wait()
    assert lib.vkc_side_defer(h, 1) == 0
    try:
        assert lib.vkc_side_begin(h) == 0
        big @ big                              # milliseconds on the side branch
        assert lib.vkc_side_end(h) == 0
        st, rd, got = _in_thread(backward_and_read)
    finally:
        assert lib.vkc_side_defer(h, 0) == 0
    assert st == 0 and rd == 0
    exp = dy.T.astype(np.float64) @ x
    assert np.linalg.norm(got - exp) < 1e-5 * np.linalg.norm(exp)
