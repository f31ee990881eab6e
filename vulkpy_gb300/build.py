"""Build the native library ``libvulkpy_gb300.so`` in-tree for sm_103a.

Every ``csrc/*.cu`` file is compiled by nvcc in parallel (one ``-gencode``
for ``compute_103a``/``sm_103a``) and linked into one shared library next to
this file.  Objects go to ``_build/`` and are rebuilt only when a source or
header is newer than the object.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
INCLUDE = HERE.parent / "include"
BUILD = HERE / "_build"
LIB = HERE / "libvulkpy_gb300.so"
# the CPython binding of the per-operation calls, named for the interpreter it
# is compiled for (another one does not load it)
HOT = HERE / ("_hot" + sysconfig.get_config_var("EXT_SUFFIX"))

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = [
    "-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    f"-I{INCLUDE}",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build vulkpy_gb300")


def _stale(obj: Path, src: Path, headers: list[Path]) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return any(p.stat().st_mtime > t for p in [src, *headers])


def build(verbose: bool = False, jobs: int | None = None) -> Path:
    """Compile the CUDA sources and link the shared library; returns its path."""
    nvcc = _nvcc()
    BUILD.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + sorted(INCLUDE.glob("*.h"))
    objs = []
    todo = []
    for src in sources:
        obj = BUILD / (src.stem + ".o")
        objs.append(obj)
        if _stale(obj, src, headers):
            todo.append((src, obj))

    def compile_one(item):
        src, obj = item
        cmd = [nvcc, *ARCH, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{r.stdout}\n{r.stderr}")
        return src.name

    if todo:
        with cf.ThreadPoolExecutor(max_workers=jobs or min(len(todo), os.cpu_count() or 4)) as ex:
            for name in ex.map(compile_one, todo):
                if verbose:
                    print(f"compiled {name}", flush=True)
    if todo or not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
        tmp = LIB.with_suffix(".so.tmp")
        cmd = [nvcc, *ARCH, "-shared", "-o", str(tmp), *map(str, objs), "-lcudart_static", "-lrt", "-ldl", "-lpthread"]
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
        os.replace(tmp, LIB)
    (HERE / "_hot.so").unlink(missing_ok=True)  # any interpreter would load it
    src = CSRC / "hot.c"
    if _stale(HOT, src, sorted(INCLUDE.glob("*.h"))):
        tmp = HOT.with_suffix(".so.tmp")
        cmd = [os.environ.get("CC", "gcc"), "-O2", "-std=c11", "-shared", "-fPIC", f"-I{sysconfig.get_paths()['include']}",
               str(src), "-o", str(tmp)]
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"compiling hot.c failed:\n{r.stdout}\n{r.stderr}")
        os.replace(tmp, HOT)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
