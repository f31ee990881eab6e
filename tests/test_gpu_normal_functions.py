"""The functions inside the normal generator, each over all its 2^23
arguments.  A state (0, 1, 0, w) gives the raw output rotl(w, 7), so that any
pair of uniforms can be put in.

Bounds, in ulps of the exact value: sin and cos 1.55 (the reduced argument is
rounded once, half an ulp, which is one of the result's where that lies a
binade below; half an ulp for the result; 0.05 for the polynomial), the radius
1.5 (logf's 1 ulp, half of it after the square root, which is one of the
result's in a lower binade; half an ulp for the result)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 23


def _pairs(gpu, k0, k1, mean=0.0, stddev=1.0):
    """Box-Muller pairs of the uniforms k0 / 2^23 and k1 / 2^23."""
    import vulkpy_gb300 as vk
    n = len(k0)
    r = vk.random.Xoshiro128pp(gpu, size=2 * n, seed=1)
    st = np.zeros((2 * n, 4), np.uint32)
    st[:, 1] = 1
    for half, k in ((0, k0), (1, k1)):
        w = k.astype(np.uint32) << np.uint32(9)
        st[half::2, 3] = (w >> np.uint32(7)) | (w << np.uint32(25))
    r._state[:] = st.reshape(-1)
    r._state._dptr()
    z = np.array(r.normal(shape=(2 * n,), mean=mean, stddev=stddev))
    return z[0::2], z[1::2]


def _ulps(got, exact):
    own = np.exp2(np.floor(np.log2(np.abs(exact))) - 23)
    return np.abs(got.astype(np.float64) - exact) / own


@pytest.fixture(scope="module")
def every():
    return np.arange(N, dtype=np.uint32)


def test_radius(gpu, every):
    _, z = _pairs(gpu, every, np.zeros(N, np.uint32))       # angle 0: cos is 1
    exact = np.sqrt(-2 * np.log1p(-every[1:].astype(np.float64) / N))
    assert _ulps(z[1:], exact).max() < 1.5


def test_radius_zero_gives_the_mean(gpu, every):
    """u0 = 0: log(1) is 0, so both numbers are the mean."""
    k1 = every[::4097]
    for mean in (0.0, 1.5, 1e-20):
        for z in _pairs(gpu, np.zeros(len(k1), np.uint32), k1, mean=mean, stddev=3.0):
            np.testing.assert_array_equal(z, np.float32(mean))


def test_sin_and_cos(gpu, every):
    half = np.full(1, N // 2, np.uint32)
    r = _pairs(gpu, half, np.zeros(1, np.uint32))[1][0]
    sd = np.float32(1.0) / r
    while _pairs(gpu, half, np.zeros(1, np.uint32), stddev=float(sd))[1][0] != 1.0:   # fl(r stddev) = 1
        sd = np.nextafter(sd, np.float32(9))
        assert sd < 2 / r
    s, c = _pairs(gpu, np.full(N, N // 2, np.uint32), every, stddev=float(sd))
    a = (np.float32(6.28318530718) * (every.astype(np.float32) / np.float32(N))).astype(np.float64)
    assert s[0] == 0.0 and c[0] == 1.0
    assert _ulps(s[1:], np.sin(a[1:])).max() < 1.55
    assert _ulps(c, np.cos(a)).max() < 1.55
    assert np.abs(s).max() <= 1.0 and np.abs(c).max() <= 1.0
