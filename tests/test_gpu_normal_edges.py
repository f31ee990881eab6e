"""Normal numbers at the edges of the pairwise kernel: one or two pair steps,
an odd count (the last pair half inside the output), a buffer that is not
8-byte aligned (element stores instead of pair stores), serial and segmented.

Against the oracle's float32 restatement: log within 0.9 ulp, sin and cos
within 1.8 ulp and a correctly rounded angle give at most a few ulp of r
(<= 6 stddev) either side: rtol 2e-6, atol 4e-6 for stddev 2."""
import ctypes as C

import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,n", [(64, 1), (64, 63), (64, 64), (64, 129), (64, 130), (64, 193), (256, 5000), (64, 4097),
                                    (4096, 12289), (4, 70001)])
@pytest.mark.parametrize("offset", [0, 1])
def test_normal_pair_edges(gpu, size, n, offset):
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import _lib
    ref = O.Xoshiro128pp(9, size)
    r = vk.random.Xoshiro128pp(gpu, size=size, seed=9)
    buf = vk.Array(gpu, data=np.full(n + 3, 77.0, np.float32))
    for _ in range(2):  # the second call starts from the advanced states
        exp = ref.normal(n, 1.5, 2.0)
        st = _lib.lib.vkc_xoshiro_normal(gpu.handle, r._state._dptr(), size, buf._dptr() + 4 * offset, n,
                                         C.c_float(1.5), C.c_float(2.0))
        assert st == 0, _lib.last_error()
        r._state._written()
        buf._written()
        got = np.asarray(buf).copy()
        np.testing.assert_allclose(got[offset:offset + n], exp, rtol=2e-6, atol=4e-6)
        np.testing.assert_array_equal(got[:offset], 77.0)
        np.testing.assert_array_equal(got[offset + n:], 77.0)
        np.testing.assert_array_equal(r.state().reshape(-1), ref.state)
