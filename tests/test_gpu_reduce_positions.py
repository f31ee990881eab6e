"""Arg-reductions with the extreme at every place of a thread's group of 16, and
axis reductions with every remainder of eight rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one block (256 threads, 16 elements each) and a little more; aligned and not
@pytest.mark.parametrize("n", [1, 5, 255, 1030, 4096, 4099])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("op", ["argmax", "argmin"])
def test_extreme_at_every_place(gpu, n, offset, op):
    import ctypes as C
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib
    sign = np.float32(1 if op == "argmax" else -1)
    out = vk.U32Array(gpu, shape=(1,))
    for at in sorted({0, 1, 3, 4, n // 4, n // 2, 3 * n // 4, n - 4, n - 2, n - 1} & set(range(n))):
        for twin in (n - 1, at):
            x = np.zeros(n + 1, np.float32)
            x[offset + at] = x[offset + max(at, twin)] = 2 * sign     # equal ones: the first
            x[offset + n:] = 9 * sign                                # not part of the input
            if offset:
                x[0] = 9 * sign
            a = vk.Array(gpu, data=x)
            st = _lib.lib.vkc_arg_reduce_all(gpu.handle, _lib.ARGMAX if op == "argmax" else _lib.ARGMIN,
                                             C.c_void_p(a._dptr() + 4 * offset), n, out._buf.ptr)
            assert st == 0
            out._written()
            assert np.asarray(out)[0] == at, (at, twin)


# slices of k_cols_block with every remainder of eight rows (32 to 4 warps),
# k_cols with and without loads that stay in the L2 cache
@pytest.mark.parametrize("shape", [(32 * 8 + r, 77) for r in (0, 1, 32, 96, 128, 160, 224)]
                         + [(300, 7777), (60, 73728), (64 + 7, 30001), (2003, 4099), (1031, 31001)])
def test_remainders_of_axis_reductions(gpu, shape):
    """maximum is exact; sum within 2^-21 of the sum of magnitudes, prod (near
    1) within 2e-5."""
    import vulkpy_gb300 as vk
    rng = np.random.default_rng(shape[0] + shape[1])
    X = rng.standard_normal(shape, dtype=np.float32)
    x = vk.Array(gpu, data=X)
    np.testing.assert_array_equal(np.asarray(x.maximum(axis=0)), X.max(axis=0))
    np.testing.assert_array_equal(np.asarray(x.minimum(axis=0)), X.min(axis=0))
    s = np.asarray(x.sum(axis=0)).astype(np.float64)
    X64 = X.astype(np.float64)
    assert np.all(np.abs(s - X64.sum(axis=0)) <= 2.0 ** -21 * np.abs(X64).sum(axis=0))
    E = np.exp(X * np.float32(1e-4))
    np.testing.assert_allclose(np.asarray(vk.Array(gpu, data=E).prod(axis=0)), E.astype(np.float64).prod(axis=0), rtol=2e-5)
