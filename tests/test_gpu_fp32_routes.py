"""fp32 products at the edges of the three-part tensor-core path, with the
path checked: it makes three launches (operand pre-pass, GEMM, and repair or
reduction), the FMA GEMMs one or two.

Accuracy as in test_gpu_fp32_tensor.py: relative Frobenius error below one
accumulation's worst case, 4 * 2^-23 < 5e-7."""
import ctypes as C

import numpy as np
import pytest

from oracle.ops import rel_fro
from test_gpu_fp32_tensor import BOUND, _gemm, _operands, _poison, _same, plans, vk  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_plans(vk):
    """Every shape on the built-in rules; the shipped table again afterwards."""
    from vulkpy_gb300 import _lib, autotune
    assert _lib.lib.vkc_gemm_tune_clear() == 0
    yield
    autotune.load_table()


def _launches(gpu, f):
    from vulkpy_gb300 import _lib
    a, b = C.c_uint64(), C.c_uint64()
    assert _lib.lib.vkc_launch_count(C.byref(a)) == 0
    out = f()
    assert _lib.lib.vkc_launch_count(C.byref(b)) == 0
    return b.value - a.value, out


def _product(vk, gpu, A, B):
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    n, c = _launches(gpu, lambda: a @ b)
    return n, np.asarray(c).copy()


# tile edges (128), K-block edges (64) and the small-product span (512), with
# K above 256 (up to there unsplit products of few tiles run on FMAs)
@pytest.mark.parametrize("m,n,k", [(2, 2, 257), (128, 128, 320), (129, 127, 321), (127, 257, 511), (33, 31, 512),
                                   (300, 520, 513), (64, 1000, 1100)])
@pytest.mark.parametrize("splits", [1, 3])
def test_tile_edges(gpu, vk, plans, m, n, k, splits):
    plans(m, n, k, splits)
    A, B = _operands(np.random.default_rng(m + 3 * n + 7 * k), m, n, k, 0, 0)
    launches, got = _product(vk, gpu, A, B)
    assert launches == 3
    assert rel_fro(got, A.astype(np.float64) @ B) < BOUND
    assert gpu.check_errors() == 0


# from m n = 2^24 on K of 16 and more: single K blocks, the last one partial
@pytest.mark.parametrize("k", [16, 17, 63, 64, 65])
def test_single_k_blocks(gpu, vk, no_plans, k):
    m, n = 4097, 4100
    A, B = _operands(np.random.default_rng(k), m, n, k, 0, 0)
    launches, got = _product(vk, gpu, A, B)
    assert launches == 3
    assert rel_fro(got, A.astype(np.float64) @ B) < BOUND
    assert gpu.check_errors() == 0


@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "large", "tiny"])
@pytest.mark.parametrize("splits", [1, 3])
def test_values_outside_the_split(gpu, vk, plans, kind, splits):
    m, n, k = 150, 140, 270
    plans(m, n, k, splits)
    A, B = _operands(np.random.default_rng(11), m, n, k, 0, 0)
    _poison(A, B, kind)
    launches, got = _product(vk, gpu, A, B)
    assert launches == 3
    _same(got, A, B)
    assert gpu.check_errors() == 0


# partial sums recomputed inside the GEMM: each form, with operands that the
# 16-byte loads can and cannot read, remainders of rows, columns and K
@pytest.mark.parametrize("kind", ["nan", "large"])
@pytest.mark.parametrize("m,n,k", [(1040, 1032, 1016), (1041, 1031, 1015)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_partial_sums_outside_the_split(gpu, vk, plans, kind, m, n, k, ta, tb):
    plans(m, n, k, 3)
    A, B = _operands(np.random.default_rng(13), m, n, k, 0, 0)
    _poison(A, B, kind)
    launches, got = _launches(gpu, lambda: _gemm(vk, gpu, np.ascontiguousarray(A.T) if ta else A,
                                                 np.ascontiguousarray(B.T) if tb else B, ta, tb))
    assert launches == 3
    _same(got, A, B)
    assert gpu.check_errors() == 0


def test_partial_sums_outside_the_split_on_every_cta(gpu, vk, plans):
    """More units per CTA than the mask of units to recompute has bits: rows at
    both ends of the matrix, in either K range."""
    m, n, k = 9300, 9200, 128
    plans(m, n, k, 2)
    rng = np.random.default_rng(14)
    A, B = _operands(rng, m, n, k, 0, 0)
    A[5, 100] = np.nan
    A[9299, 3] = np.float32(2.0 ** 103)
    launches, got = _product(vk, gpu, A, B)
    assert launches == 3
    assert np.all(np.isnan(got[5]))
    rows = np.unique(np.concatenate([np.arange(0, 140), rng.integers(140, m, 200), np.arange(m - 140, m)]))
    rows = rows[rows != 5]
    e = A[rows].astype(np.float64) @ B
    scale = np.abs(A[rows]).astype(np.float64) @ np.abs(B)
    assert np.all(np.abs(got[rows] - e) <= (k + 2) * 2.0 ** -24 * scale)
    assert gpu.check_errors() == 0


def test_without_room_for_the_copies(gpu, vk, no_plans):
    """The operand copies cannot be had: the product is computed from the
    operands in place."""
    from vulkpy_gb300 import _lib
    A, B = _operands(np.random.default_rng(1), 300, 200, 300, 0, 0)
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    exp = A.astype(np.float64) @ B
    launches, c = _launches(gpu, lambda: a @ b)
    assert launches == 3 and rel_fro(np.asarray(c), exp) < BOUND
    try:
        assert _lib.lib.vkc_inject_alloc_failure(1) == 0   # the second allocation: after the result's
        launches, c = _launches(gpu, lambda: a @ b)
    finally:
        _lib.lib.vkc_inject_alloc_failure(-1)
    assert launches == 1
    assert rel_fro(np.asarray(c), exp) < 1e-6


def test_without_room_for_the_partial_sums(gpu, vk, no_plans):
    """300 x 300 x 400 in three K ranges: the operand copies can be had, the
    ranges' partial sums cannot; the FMA GEMM needs neither."""
    from vulkpy_gb300 import _lib
    A, B = _operands(np.random.default_rng(3), 300, 300, 400, 0, 0)
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    exp = A.astype(np.float64) @ B
    try:
        assert _lib.lib.vkc_inject_alloc_failure(2) == 0   # the third allocation: after the copies'
        launches, c = _launches(gpu, lambda: a @ b)
    finally:
        _lib.lib.vkc_inject_alloc_failure(-1)
    assert launches == 2                                   # the operand pre-pass, and the FMA GEMM
    assert rel_fro(np.asarray(c), exp) < 1e-6
    launches, c = _launches(gpu, lambda: a @ b)
    assert launches == 3 and rel_fro(np.asarray(c), exp) < BOUND


def test_without_room_in_a_capture(gpu, vk, no_plans):
    """The same while a graph is captured (copies and, in a second product,
    partial sums that cannot be had)."""
    from vulkpy_gb300 import _lib
    A, B = _operands(np.random.default_rng(5), 300, 300, 400, 0, 0)
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    exp = A.astype(np.float64) @ B
    a @ b
    for after, launches in ((1, 1), (2, 2), (-1, 3)):
        g = vk.graph.Graph(gpu)
        try:
            assert _lib.lib.vkc_inject_alloc_failure(after) == 0
            with g:
                n, c = _launches(gpu, lambda: a @ b)
        finally:
            _lib.lib.vkc_inject_alloc_failure(-1)
        assert n == launches
        g.launch()
        assert rel_fro(np.asarray(c), exp) < 1e-6
    big = vk.Array(gpu, data=np.ones((6144, 6144), np.float32))    # 450 MB of copies: with room for them
    big @ big
    g = vk.graph.Graph(gpu)
    with g:
        n, c = _launches(gpu, lambda: big @ big)
    assert n == 3
    g.launch()
    assert np.all(np.asarray(c) == 6144)


def _grouped(vk, gpu, A, B):
    """A @ B as a grouped product of one problem: launches and result."""
    from vulkpy_gb300 import _lib
    (m, k), n = A.shape, B.shape[1]
    a, b, c = vk.Array(gpu, data=A), vk.Array(gpu, data=B), vk.Array(gpu, shape=(m, n))
    p = _lib.GemmProblem(ta=0, tb=0, m=m, n=n, k=k, alpha=1.0, beta=0.0, a=a._dptr(), lda=k, b=b._dptr(), ldb=n,
                         c=c._buf.ptr, ldc=n)
    launches, st = _launches(gpu, lambda: _lib.lib.vkc_gemm_grouped(gpu.handle, _lib.MM_FP32, C.byref(p), 1))
    assert st == 0, _lib.last_error()
    c._written()
    return launches, np.asarray(c).copy()


def test_grouped_without_room_for_the_copies(gpu, vk):
    from vulkpy_gb300 import _lib
    A, B = _operands(np.random.default_rng(2), 1040, 1030, 1010, 0, 0)
    exp = A.astype(np.float64) @ B
    launches, got = _grouped(vk, gpu, A, B)
    assert launches == 3 and rel_fro(got, exp) < BOUND
    a, b, c = vk.Array(gpu, data=A), vk.Array(gpu, data=B), vk.Array(gpu, shape=(1040, 1030))
    p = _lib.GemmProblem(ta=0, tb=0, m=1040, n=1030, k=1010, alpha=1.0, beta=0.0, a=a._dptr(), lda=1010, b=b._dptr(),
                         ldb=1030, c=c._buf.ptr, ldc=1030)
    try:
        assert _lib.lib.vkc_inject_alloc_failure(0) == 0
        launches, st = _launches(gpu, lambda: _lib.lib.vkc_gemm_grouped(gpu.handle, _lib.MM_FP32, C.byref(p), 1))
    finally:
        _lib.lib.vkc_inject_alloc_failure(-1)
    assert st == 0, _lib.last_error()
    c._written()
    assert launches == 1
    assert rel_fro(np.asarray(c), exp) < 1e-6


def test_grouped_and_single_where_the_single_call_splits(gpu, vk, no_plans):
    """256 x 1024 x 4096: the single call splits K, the grouped one does not;
    both are within the path's bound."""
    A, B = _operands(np.random.default_rng(4), 256, 1024, 4096, 0, 0)
    exp = A.astype(np.float64) @ B
    launches, grouped = _grouped(vk, gpu, A, B)
    assert launches == 3 and rel_fro(grouped, exp) < BOUND
    launches, single = _product(vk, gpu, A, B)
    assert launches == 3 and rel_fro(single, exp) < BOUND
    assert gpu.check_errors() == 0
