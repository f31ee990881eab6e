"""fp32 products as six bf16 tensor-core products (three exact parts per
operand), single and grouped.

Accuracy: each hi*hi accumulation makes at most four truncating additions of
at most 2^-23 of the running sum; the blocks are added with round-to-nearest
(2^-24 each).  For random data the relative Frobenius error stays below one
accumulation's worst case, 4 * 2^-23 < 5e-7, at every K.

Results that values outside the split (inf, NaN, |x| >= 2^103) reach, or that
overflow on the way (2^79 and more), are recomputed from the fp32 operands in
order of k, so they behave like float32 FMAs: inf and NaN where float32
arithmetic has them.  Small values, subnormals included, are split exactly."""
import ctypes as C

import numpy as np
import pytest

from oracle.ops import rel_fro

pytestmark = pytest.mark.gpu

BOUND = 5e-7


@pytest.fixture(scope="module")
def vk():
    import vulkpy_gb300
    return vulkpy_gb300


@pytest.fixture
def plans():
    """vkc_gemm_plan_set, and the shipped table again afterwards."""
    from vulkpy_gb300 import _lib, autotune
    yield lambda m, n, k, s: _lib.lib.vkc_gemm_plan_set(_lib.MM_FP32, m, n, k, s, 128)
    _lib.lib.vkc_gemm_tune_clear()
    autotune.load_table()


def _matmul(vk, gpu, A, B):
    return np.asarray(vk.Array(gpu, data=A) @ vk.Array(gpu, data=B)).copy()


def _gemm(vk, gpu, A, B, ta, tb, alpha=1.0, beta=0.0, C0=None):
    from vulkpy_gb300 import _lib
    M, K = A.shape[::-1] if ta else A.shape
    N = B.shape[0] if tb else B.shape[1]
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    c = vk.Array(gpu, data=C0 if C0 is not None else np.zeros((M, N), np.float32))
    st = _lib.lib.vkc_gemm(gpu.handle, _lib.MM_FP32, ta, tb, M, N, K, C.c_float(alpha), a._dptr(), A.shape[1],
                           b._dptr(), B.shape[1], C.c_float(beta), c._dptr(), N)
    assert st == 0, _lib.last_error()
    c._written()
    return np.asarray(c).copy()


def _operands(rng, M, N, K, ta, tb):
    A = rng.standard_normal((K, M) if ta else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if tb else (K, N)).astype(np.float32)
    return A, B


# tile edges (128), K-block edges (64) and the small-product span (512)
@pytest.mark.parametrize("m,n,k", [(2, 2, 64), (128, 128, 64), (129, 127, 65), (127, 257, 511), (33, 31, 512),
                                   (300, 520, 513), (64, 1000, 1100), (1000, 64, 1024), (31, 4099, 577)])
@pytest.mark.parametrize("splits", [1, 3])
def test_accuracy_at_tile_edges(gpu, vk, plans, m, n, k, splits):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    plans(m, n, k, splits)
    A, B = _operands(rng, m, n, k, 0, 0)
    assert rel_fro(_matmul(vk, gpu, A, B), A.astype(np.float64) @ B) < BOUND
    assert gpu.check_errors() == 0


# vkc_gemm takes the path from m n k = 2^30 on: transposes, alpha, beta
@pytest.mark.parametrize("m,n,k", [(1025, 1030, 1100), (513, 4099, 520), (2100, 513, 1024)])
@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_gemm_forms(gpu, vk, plans, m, n, k, splits, ta, tb):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    plans(m, n, k, splits)
    A, B = _operands(rng, m, n, k, ta, tb)
    C0 = rng.standard_normal((m, n)).astype(np.float32)
    e = (A.T if ta else A).astype(np.float64) @ (B.T if tb else B).astype(np.float64)
    assert rel_fro(_gemm(vk, gpu, A, B, ta, tb), e) < BOUND
    assert rel_fro(_gemm(vk, gpu, A, B, ta, tb, 0.5, 2.0, C0), 0.5 * e + 2.0 * C0) < BOUND
    assert gpu.check_errors() == 0


def _poison(A, B, kind):
    """Puts unusual values into rows 1 and 40 of A and column 2 of B; the
    rows and columns of the result they reach."""
    if kind == "inf":
        A[1, 3], A[40, 5] = np.inf, -np.inf
        B[7, 2] = np.inf
    elif kind == "nan":
        A[1, 3], A[40, 64] = np.nan, np.nan
        B[0, 2] = np.nan
    elif kind == "huge":          # overflows in the sum, and hi alone would round to inf
        A[1, 3], A[40, :] = np.float32(3.4e38), np.float32(2e37)
        B[5, 2] = np.float32(-3.3e38)
    elif kind == "large":         # finite results that overflow the scaled accumulators
        A[1, :] *= np.float32(2.0 ** 60)
        A[40, 9] = np.float32(2.0 ** 104)
        B[:, 2] *= np.float32(2.0 ** 20)
    elif kind == "tiny":          # rows and columns down to subnormals
        A[1, :] *= np.float32(2.0 ** -115)
        A[40, ::2] = np.float32(1e-40)
        B[:, 2] *= np.float32(2.0 ** -112)


def _float32_like(A, B):
    """float64 products rounded to float32, overflow and specials included."""
    with np.errstate(all="ignore"):
        return (A.astype(np.float64) @ B.astype(np.float64)).astype(np.float32)


def _same(got, A, B):
    with np.errstate(all="ignore"):
        e = _float32_like(A, B)
        scale = np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64)
    # a sum that overflows on the way may be inf or NaN in float32 although its end value is finite
    sure = np.isfinite(e) & (scale < 3e38)
    K = A.shape[1]
    tol = (K + 2) * 2.0 ** -24 * scale + K * 2.0 ** -149
    assert np.all(np.abs(got[sure].astype(np.float64) - e[sure]) <= tol[sure])
    np.testing.assert_array_equal(np.isnan(got)[np.isnan(e)], True)
    assert not np.any(np.isfinite(got[~np.isfinite(e)]))
    inputs_inf = np.isinf(e) & (~np.isfinite(scale) | (scale < 1e38))
    np.testing.assert_array_equal(got[inputs_inf], e[inputs_inf])


@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "large", "tiny"])
@pytest.mark.parametrize("splits", [1, 2])
def test_values_outside_the_split(gpu, vk, plans, kind, splits):
    rng = np.random.default_rng(11)
    m, n, k = 150, 140, 200
    plans(m, n, k, splits)
    A, B = _operands(rng, m, n, k, 0, 0)
    _poison(A, B, kind)
    _same(_matmul(vk, gpu, A, B), A, B)
    assert gpu.check_errors() == 0


@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "large", "tiny"])
@pytest.mark.parametrize("splits", [1, 2])
def test_values_outside_the_split_in_gemm(gpu, vk, plans, kind, splits):
    rng = np.random.default_rng(12)
    m, n, k = 1040, 1030, 1010
    plans(m, n, k, splits)
    A, B = _operands(rng, m, n, k, 0, 0)
    _poison(A, B, kind)
    _same(_gemm(vk, gpu, np.ascontiguousarray(A.T), np.ascontiguousarray(B.T), 1, 1), A, B)
    # beta: C is read once, by whichever kernel computes the result
    got = _gemm(vk, gpu, A, B, 0, 0, 1.0, 1.0, np.full((m, n), 3.0, np.float32))
    clean = np.ones((m, n), bool)
    clean[[1, 40], :] = False
    clean[:, 2] = False
    e = _float32_like(A, B)
    np.testing.assert_allclose(got[clean], e[clean] + 3.0, rtol=1e-5, atol=1e-4)
    if kind == "tiny":
        np.testing.assert_allclose(got, e + 3.0, rtol=1e-5, atol=1e-4)
    assert gpu.check_errors() == 0


@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "large", "tiny"])
def test_grouped_equals_single_with_unusual_values(gpu, vk, plans, kind):
    """Grouped products (swapped ones among them: m <= 64 < n) give
    vkc_gemm's bits, recomputed results included."""
    rng = np.random.default_rng(3)
    As, Bs, ref = [], [], []
    for m, n, k in ((1040, 1030, 1010), (64, 4200, 4100), (50, 129, 64), (2100, 520, 1000)):
        plans(m, n, k, 1)
        A, B = _operands(rng, m, n, k, 0, 0)
        if k > 64:
            _poison(A, B, kind)
        As.append(vk.Array(gpu, data=A))
        Bs.append(vk.Array(gpu, data=B))
        ref.append(_gemm(vk, gpu, A, B, 0, 0))
    for got, e in zip(vk.vkarray.matmul_grouped(As, Bs, precision="fp32"), ref):
        np.testing.assert_array_equal(np.asarray(got), e)
    assert gpu.check_errors() == 0


def test_without_room_for_the_copies(gpu, vk):
    """The operand copies cannot be had: the product is computed from the
    operands in place."""
    from vulkpy_gb300 import _lib
    rng = np.random.default_rng(1)
    A, B = _operands(rng, 300, 200, 150, 0, 0)
    a, b = vk.Array(gpu, data=A), vk.Array(gpu, data=B)
    try:
        assert _lib.lib.vkc_inject_alloc_failure(1) == 0   # the second allocation: after the result's
        c = a @ b
    finally:
        _lib.lib.vkc_inject_alloc_failure(-1)
    assert rel_fro(np.asarray(c), A.astype(np.float64) @ B) < 1e-6
