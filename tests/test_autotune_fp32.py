"""The fp32 entries of the tuning table are those of the FMA GEMM: they are
measured on shapes that run it."""
import pytest


def test_fp32_entries_are_measured_on_shapes_that_run_fmas():
    at = pytest.importorskip("vulkpy_gb300.autotune")
    shapes = at.default_shapes()
    left_out = 0
    for s in shapes:
        f = at.fma_shape(*s)
        if f is None:
            low = [(1 << at.bucket(x)) // 2 + 1 for x in s]
            assert low[0] * low[1] * low[2] >= at.FP32_TENSOR_WORK
            left_out += 1
            continue
        assert f[0] * f[1] * f[2] < at.FP32_TENSOR_WORK
        assert [at.bucket(x) for x in f] == [at.bucket(x) for x in s]
        if s[0] * s[1] * s[2] < at.FP32_TENSOR_WORK:
            assert f == s
    assert 0 < left_out < len(shapes) // 10


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,tensor", [(1024, 1024, 1024, True), (256, 1024, 4096, True), (1024, 1024, 1000, False),
                                          (600, 600, 600, False)])
def test_plan_get_reports_the_kernel_that_runs(gpu, m, n, k, tensor):
    """A width-256 entry sets the FMA GEMM's ranges; the plan of a shape that
    runs on the tensor cores is the three-part product's."""
    import ctypes as C
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib, autotune
    lib = _lib.lib
    a, b, c = (vk.zeros(gpu, shape=s) for s in ((m, k), (n, k), (m, n)))
    got, n0, n1 = C.c_int(), C.c_uint64(), C.c_uint64()
    try:
        assert lib.vkc_gemm_tune_clear() == 0
        assert lib.vkc_gemm_tune_get(gpu.handle, _lib.MM_FP32, m, n, k, C.byref(got)) == 0
        rule = got.value
        assert lib.vkc_gemm_tune_set(_lib.MM_FP32, m, n, k, 13) == 0
        assert lib.vkc_gemm_tune_get(gpu.handle, _lib.MM_FP32, m, n, k, C.byref(got)) == 0
        assert lib.vkc_launch_count(C.byref(n0)) == 0
        assert lib.vkc_gemm(gpu.handle, _lib.MM_FP32, 0, 1, m, n, k, 1.0, a._dptr(), k, b._dptr(), k, 0.0, c._dptr(),
                            n) == 0
        assert lib.vkc_launch_count(C.byref(n1)) == 0
        assert got.value == (rule if tensor else 13)
        assert n1.value - n0.value == (3 if tensor else 2)   # pre-pass, GEMM, repair or reduction; FMAs, reduction
    finally:
        lib.vkc_gemm_tune_clear()
        autotune.load_table()
