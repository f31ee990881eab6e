"""Reductions and arg-reductions at the edges of their kernels' splits: axes
around the slices of 4 / 8 / 16 / 32 warps, rows around a group of 16
elements per thread, widths that are and are not multiples of 4.

Sums are compensated, so their error is a few roundings of the result plus
2^-24 of the mean absolute term: |err| <= 2^-22 sum|x| is far above it and
far below any wrong or missing term."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vk():
    import vulkpy_gb300
    return vulkpy_gb300


@pytest.mark.parametrize("prev,axis,post", [(1, 37, 33153), (3, 16, 5000), (2, 63, 20001), (2, 64, 8004), (1, 65, 16000),
                                            (1, 127, 4097), (7, 257, 129), (5, 513, 36), (1, 3000, 1501), (2, 2500, 4100)])
def test_middle_axis(gpu, vk, prev, axis, post):
    rng = np.random.default_rng(prev + axis + post)
    a = rng.standard_normal((prev, axis, post)).astype(np.float32)
    x = vk.Array(gpu, data=a)
    a64 = a.astype(np.float64)
    tol = 2.0 ** -22 * np.abs(a64).sum(axis=1)
    assert np.all(np.abs(np.asarray(x.sum(axis=1)) - a64.sum(axis=1)) <= tol)
    np.testing.assert_array_equal(np.asarray(x.maximum(axis=1)), a.max(axis=1))
    np.testing.assert_array_equal(np.asarray(x.minimum(axis=1)), a.min(axis=1))
    e = np.exp(a * np.float32(1e-3))
    np.testing.assert_allclose(np.asarray(vk.Array(gpu, data=e).prod(axis=1)), e.astype(np.float64).prod(axis=1),
                               rtol=1e-6)
    got = np.asarray(x.sum(axis=1, rebroadcast=True))
    assert got.shape == a.shape and np.all(np.abs(got - a64.sum(axis=1, keepdims=True)) <= tol[:, None, :])


@pytest.mark.parametrize("rows,length", [(5, 2048), (3, 2049), (2, 4095), (2, 16384), (2, 16388), (3, 20001), (700, 100)])
@pytest.mark.parametrize("kind", ["normal", "equal", "worst", "nan_late", "nan_all", "zeros"])
def test_arg_rows(gpu, vk, rows, length, kind):
    rng = np.random.default_rng(rows * length)
    a = rng.standard_normal((rows, length)).astype(np.float32)
    if kind == "equal":
        a[:] = 1.5
    elif kind == "worst":          # nothing but the value a search starts from, then with one better at the end
        a[:] = -np.inf
        a[-1, -1] = -3.0
    elif kind == "nan_late":
        a[:, length - 2:] = np.nan
    elif kind == "nan_all":
        a[:] = np.nan
    elif kind == "zeros":
        a[:] = np.where(rng.random(a.shape) < 0.5, np.float32(0.0), np.float32(-0.0))
    for b in (a, -a):
        x = vk.Array(gpu, data=b)
        np.testing.assert_array_equal(np.asarray(x.argmax(axis=1)), np.argmax(b, axis=1).astype(np.uint32))
        np.testing.assert_array_equal(np.asarray(x.argmin(axis=1)), np.argmin(b, axis=1).astype(np.uint32))
        assert int(np.asarray(x.argmax())[0]) == int(np.argmax(b))
        assert int(np.asarray(x.argmin())[0]) == int(np.argmin(b))
