"""Builds the shared libraries in this directory with nvcc for sm_100a.

    python -m pratchya_b200.csrc.build [--force] [-v]

libpratchya_b200.so is the product, _native.so the host side of its ops for torch (native.cc, a CPython extension).  libpratchya_b200_diag.so is the same sources compiled with
-DPB_DIAGNOSTICS plus selftest.cu: cycle counters, timing experiments, environment switches, the
fault injection of the abort-path test and the device self-checks live there only, and only the
tests load it.  Both are kept in-tree next to their sources; nothing is installed anywhere.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
INCLUDE = HERE.parent.parent / "include"
LIB = HERE / "libpratchya_b200.so"
DIAG_LIB = HERE / "libpratchya_b200_diag.so"
NATIVE = HERE / "_native.so"
SOURCES = ["api.cu", "quantize.cu", "dequantize.cu", "transpose_quantize.cu", "optimizer.cu", "gemm_sm100.cu", "dense_dot.cu", "split_dot.cu", "wkv7.cu", "rwkv_glue.cu", "rwkv_norms.cu", "loss.cu"]
DIAG_SOURCES = SOURCES + ["selftest.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--cudart", "static",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(d).stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False, diagnostics: bool = False) -> Path:
    """Compiles what is stale and links the product library (or, with `diagnostics`, the diagnostics one)."""
    names = DIAG_SOURCES if diagnostics else SOURCES
    lib = DIAG_LIB if diagnostics else LIB
    extra = ["-DPB_DIAGNOSTICS"] if diagnostics else []
    srcs = [HERE / s for s in names if (HERE / s).exists()]
    headers = list(HERE.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    objdir = HERE / ("build_diag" if diagnostics else "build")
    objdir.mkdir(exist_ok=True)
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in srcs:
        obj = objdir / (src.stem + ".o")
        objs.append(obj)
        if force or _stale(obj, [src, *headers]):
            cmd = [nvcc, *NVCC_FLAGS, *extra, f"-I{INCLUDE}", f"-I{HERE}", "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd), flush=True)
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{out}")
    if force or procs or _stale(lib, objs):
        cmd = [nvcc, "-shared", "--cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
               "-o", str(lib), *map(str, objs), "-ldl", "-lpthread"]
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}")
    if not diagnostics:
        build_native(force, verbose)
    return lib


NATIVE_MADE_FOR = HERE / "build" / "native.made_for"


def _native_made_for() -> str:
    """The torch and the Python that native.cc is compiled against: another of either needs another _native.so."""
    import torch
    return f"torch {torch.__version__} {torch.version.git_version}, python {sys.version}"


def native_stale() -> bool:
    return (_stale(NATIVE, [HERE / "native.cc", INCLUDE / "pratchya_b200.h"]) or not NATIVE_MADE_FOR.exists()
            or NATIVE_MADE_FOR.read_text() != _native_made_for())


def build_native(force: bool = False, verbose: bool = False) -> Path:
    """Compiles native.cc against torch's headers (the library it calls, libpratchya_b200.so, is found next to it)."""
    import sysconfig

    import torch
    src = HERE / "native.cc"
    if not (force or native_stale()):
        return NATIVE
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include", f"-I{INCLUDE}",
           str(src), "-o", str(NATIVE), f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python",
           f"-L{HERE}", "-l:libpratchya_b200.so", "-Wl,-rpath,$ORIGIN"]
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed on native.cc:\n{r.stdout}")
    NATIVE_MADE_FOR.parent.mkdir(exist_ok=True)
    NATIVE_MADE_FOR.write_text(_native_made_for())
    return NATIVE


def build_all(force: bool = False, verbose: bool = False):
    return build(force, verbose), build(force, verbose, diagnostics=True)


if __name__ == "__main__":
    print(*build_all(force="--force" in sys.argv, verbose="-v" in sys.argv))
