"""The small fp32 product with a long K and many tiles (its rule bounds the
tiles, not K), B contiguous along either index: against float64, within FMAs'
K 2^-24 sum |a||b|, and the bits of the grouped GEMM's 128 x 128 tile."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(9900, 17, 1301), (700, 1000, 130), (33, 64, 5000)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_long_products(gpu, m, n, k, ta, tb):
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib, autotune
    lib = _lib.lib
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    B = rng.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    one, grouped = vk.Array(gpu, shape=(m, n)), vk.Array(gpu, shape=(m, n))
    n0, n1 = C.c_uint64(), C.c_uint64()
    try:
        assert lib.vkc_gemm_plan_set(_lib.MM_FP32, m, n, k, 1, 256) == 0
        assert lib.vkc_launch_count(C.byref(n0)) == 0
        st = lib.vkc_gemm(gpu.handle, _lib.MM_FP32, ta, tb, m, n, k, C.c_float(1.0), a._dptr(), A.shape[1], b._dptr(),
                          B.shape[1], C.c_float(0.0), one._buf.ptr, n)
        assert st == 0, _lib.last_error()
        assert lib.vkc_launch_count(C.byref(n1)) == 0 and n1.value - n0.value == 1
        p = _lib.GemmProblem(ta=ta, tb=tb, m=m, n=n, k=k, alpha=1.0, beta=0.0, a=a._dptr(), lda=A.shape[1], b=b._dptr(),
                             ldb=B.shape[1], c=grouped._buf.ptr, ldc=n)
        assert lib.vkc_gemm_grouped(gpu.handle, _lib.MM_FP32, C.byref(p), 1) == 0
    finally:
        lib.vkc_gemm_tune_clear()
        autotune.load_table()
    one._written()
    grouped._written()
    A64, B64 = (A.T if ta else A).astype(np.float64), (B.T if tb else B).astype(np.float64)
    assert np.all(np.abs(np.asarray(one) - A64 @ B64) <= (k + 3) * 2.0 ** -24 * (np.abs(A64) @ np.abs(B64)))
    np.testing.assert_array_equal(np.asarray(one), np.asarray(grouped))
