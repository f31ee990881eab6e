"""A large fp32 product returns to the caller before the GPU has computed it,
also the first of its form in a process: none of its kernels is loaded behind
running ones (loading waits for them)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import ctypes as C
import sys

import numpy as np

import vulkpy_gb300 as vk
from vulkpy_gb300 import _lib

lib = _lib.lib
gpu = vk.GPU()
form = sys.argv[1]
n = 8192                                      # 1.1e12 multiply-adds: milliseconds
m, k = (1024, 1 << 17) if form == "split" else (n, n)
a, b, c = vk.zeros(gpu, shape=(m, k)), vk.zeros(gpu, shape=(k, m)), vk.Array(gpu, shape=(m, m))
pa, pb, pc = a._dptr(), b._dptr(), c._dptr()
ta, tb = (int(v) for v in form) if form.isdigit() else (0, 0)
gpu.wait()
if form == "grouped":
    p = _lib.GemmProblem(ta=0, tb=0, m=m, n=m, k=k, alpha=1.0, beta=0.0, a=pa, lda=k, b=pb, ldb=m, c=pc, ldc=m)
    st = lib.vkc_gemm_grouped(gpu.handle, _lib.MM_FP32, C.byref(p), 1)
else:
    st = lib.vkc_gemm(gpu.handle, _lib.MM_FP32, ta, tb, m, m, k, 1.0, pa, m if ta else k, pb, k if tb else m, 0.0, pc, m)
assert st == 0, _lib.last_error()
job = C.c_void_p()
assert lib.vkc_job_record(gpu.handle, C.byref(job)) == 0
done = C.c_int(-1)
assert lib.vkc_job_query(job, C.byref(done)) == 0
assert lib.vkc_job_wait(job, -1) == 0
lib.vkc_job_destroy(job)
assert gpu.check_errors() == 0
print("done" if done.value else "running")
"""


# the four forms of a single product (the digits: A, B transposed), one whose
# K is split over a reduction, and a grouped one
@pytest.mark.parametrize("form", ["00", "01", "10", "11", "split", "grouped"])
def test_first_large_product_of_a_process_is_queued(form):
    r = subprocess.run([sys.executable, "-c", SCRIPT, form], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "running"
