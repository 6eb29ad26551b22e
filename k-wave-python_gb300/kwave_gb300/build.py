"""In-tree build of libkwave_gb300.so for sm_103a (nvcc, no cmake).

Translation units compile in parallel, then link into
``kwave_gb300/libkwave_gb300.so``.  Rebuilds only when a source is newer than
the library (or ``force=True``).
"""
from __future__ import annotations

import os
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR.parent / "csrc"
INCLUDE = PKG_DIR.parent.parent / "include"
BUILD_DIR = PKG_DIR.parent / "_build"
LIB = PKG_DIR / "libkwave_gb300.so"
SOURCES = ["kw_kernels.cu", "kw_generic_fft2.cu", "kw_axis_tma.cu", "kw_axis_tma_plain.cu", "kw_axis_tma_ops.cu", "kw_axis_tma_ops2.cu",
           "kw_mr_axis.cu", "kw_mr_axis_fwd.cu", "kw_mr_axis_inv.cu", "kw_mr_axis_grad.cu", "kw_mr_axis_div.cu", "kw_mr_axis_nab.cu", "kw_mr_axis_gen.cu",
           "kw_mr_rows.cu", "kw_mr_rows1.cu", "kw_mr_rows2.cu", "kw_mr_rows3.cu", "kw_mr_rows4.cu", "kw_mr_rows5.cu",
           "kw_rows_reg.cu", "kw_rows_reg2.cu", "kw_rows_reg3.cu", "kw_rows_tma.cu", "kw_plan.cu", "kw_noalloc.cu", "kw_unet.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
# (device code is stored as it is: unpacking its line tables when a kernel is first used
# took longer than running it -- first 375 x 324 transmit of a process 46 ms, so 23)
NVCC_FLAGS = ["-O3", "-lineinfo", "--compress-mode=none", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "--extended-lambda"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def _sources():
    return [s for s in SOURCES if (CSRC / s).exists()]


def _stale():
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = [CSRC / s for s in _sources()] + list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not _stale():
        return LIB
    nvcc = _nvcc()
    BUILD_DIR.mkdir(exist_ok=True)
    objs = []

    def compile_one(src):
        obj = BUILD_DIR / (Path(src).stem + ".o")
        cmd = [nvcc, *ARCH, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", str(CSRC / src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stderr}")
        if verbose and r.stderr:
            print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(len(_sources()), max(2, os.cpu_count() or 2))) as ex:
        objs = list(ex.map(compile_one, _sources()))
    tmp = LIB.with_suffix(".so.tmp")
    cmd = [nvcc, *ARCH, "-shared", "-o", str(tmp), *map(str, objs), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))
