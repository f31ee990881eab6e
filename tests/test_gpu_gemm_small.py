"""The small fp32 product (32 x 32 tiles, 64 of K at a time) at its tile and K
edges (and the split form beside it), against float64: FMAs in order of k are
within K 2^-24 sum |a||b| of the exact product (and 2^-24 for each of alpha,
beta C and the bias)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(2, 2, 1), (31, 33, 16), (32, 32, 63), (33, 31, 64), (64, 96, 65), (65, 100, 127),
                                   (129, 40, 128), (40, 257, 200), (1000, 1200, 20), (17, 9, 1000)])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_small_products(gpu, m, n, k, splits, ta, tb):
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib, autotune
    lib = _lib.lib
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    B = rng.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    C0 = rng.standard_normal((m, n)).astype(np.float32)
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    A64, B64 = (A.T if ta else A).astype(np.float64), (B.T if tb else B).astype(np.float64)
    e, mag = A64 @ B64, np.abs(A64) @ np.abs(B64)
    u = 2.0 ** -24
    try:
        assert lib.vkc_gemm_plan_set(_lib.MM_FP32, m, n, k, splits, 256) == 0
        for alpha, beta in ((1.0, 0.0), (0.5, 2.0)):
            c = vk.Array(gpu, data=C0)
            st = lib.vkc_gemm(gpu.handle, _lib.MM_FP32, ta, tb, m, n, k, C.c_float(alpha), a._dptr(), A.shape[1],
                              b._dptr(), B.shape[1], C.c_float(beta), c._dptr(), n)
            assert st == 0, _lib.last_error()
            c._written()
            exp = alpha * e + beta * C0
            tol = (k + 3) * u * abs(alpha) * mag + 3 * u * (np.abs(exp) + abs(beta) * np.abs(C0))
            assert np.all(np.abs(np.asarray(c) - exp) <= tol)
        if not ta and tb:   # Dense forward: bias and activation in the epilogue
            bias = rng.standard_normal(n).astype(np.float32)
            d = vk.Array(gpu, shape=(m, n))
            st = lib.vkc_dense_forward(gpu.handle, _lib.MM_FP32, a._dptr(), b._dptr(), vk.Array(gpu, data=bias)._dptr(),
                                       d._buf.ptr, m, k, n, _lib.ACT_RELU)
            assert st == 0, _lib.last_error()
            d._written()
            assert np.all(np.abs(np.asarray(d) - np.maximum(e + bias, 0)) <= (k + 3) * u * mag + 3 * u * np.abs(e + bias))
    finally:
        lib.vkc_gemm_tune_clear()
        autotune.load_table()


def test_bits_are_the_grouped_tile_code(gpu):
    """Unsplit, the small kernel adds in the order of the 128 x 128 tile (the
    grouped GEMM's code for such products): the same bits."""
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib, autotune
    rng = np.random.default_rng(4)
    pairs = [(rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32))
             for m, n, k in ((65, 100, 127), (40, 300, 700), (130, 33, 64))]
    try:
        for A, B in pairs:
            _lib.lib.vkc_gemm_plan_set(_lib.MM_FP32, A.shape[0], B.shape[1], A.shape[1], 1, 256)
        As, Bs = [vk.Array(gpu, data=A) for A, _ in pairs], [vk.Array(gpu, data=B) for _, B in pairs]
        for got, a, b in zip(vk.vkarray.matmul_grouped(As, Bs, precision="fp32"), As, Bs):
            (m, k), n = a.shape, b.shape[1]
            c = vk.Array(gpu, shape=(m, n))
            st = _lib.lib.vkc_gemm(gpu.handle, _lib.MM_FP32, 0, 0, m, n, k, C.c_float(1.0), a._dptr(), k, b._dptr(), n,
                                   C.c_float(0.0), c._buf.ptr, n)
            assert st == 0, _lib.last_error()
            c._written()
            np.testing.assert_array_equal(np.asarray(c), np.asarray(got))
    finally:
        _lib.lib.vkc_gemm_tune_clear()
        autotune.load_table()
