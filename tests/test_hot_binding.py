"""The CPython binding of the per-operation calls uses the library that ctypes
has loaded, also when VULKPY_GB300_LIB names another file."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import vulkpy_gb300
print(*sorted({l.split()[-1] for l in open("/proc/self/maps") if "libvulkpy_gb300" in l}), sep="\n")
"""


def test_one_copy_of_the_library(tmp_path):
    _lib = pytest.importorskip("vulkpy_gb300._lib")
    other = tmp_path / "libvulkpy_gb300_copy.so"
    shutil.copy(_lib.LIB_PATH, other)
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env={**os.environ, "VULKPY_GB300_LIB": str(other)},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == [str(other)]


def test_binding_is_named_for_the_interpreter():
    """An interpreter with another ABI must not load it."""
    import sysconfig
    _lib = pytest.importorskip("vulkpy_gb300._lib")
    name = os.path.basename(_lib._hot.__file__)
    assert name == "_hot" + sysconfig.get_config_var("EXT_SUFFIX") != "_hot.so"
    assert not os.path.exists(os.path.join(os.path.dirname(_lib._hot.__file__), "_hot.so"))
