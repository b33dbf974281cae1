"""Builds libmuser_cuda.so in-tree with nvcc for sm_100a (cross-compiles without a GPU)."""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libmuser_cuda.so"
CALL = PKG / ("_call" + sysconfig.get_config_var("EXT_SUFFIX"))  # the Python binding's per-call half (csrc/host_call.c), for this Python
SOURCES = ["api.cu", "repack.cu", "kquant_decode.cu", "kquant_tc.cu", "kquant_mma.cu", "nvfp4_quant.cu", "nvfp4_gemm.cu", "nvfp4_static.cu", "nvfp4_a16.cu", "collective.cu", "layer_ops.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def nvcc() -> str:
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def _newest(paths) -> float:
    return max(p.stat().st_mtime for p in paths)


def build_call(force: bool = False) -> Path | None:
    src, include = CSRC / "host_call.c", Path(sysconfig.get_paths()["include"])
    (PKG / "_call.so").unlink(missing_ok=True)  # (its former name, which any Python takes for its own)
    if not (include / "Python.h").exists():
        print(f"{include} has no Python.h: calls from Python go through ctypes (_call_py.py), some microseconds slower", file=sys.stderr)
        return None
    if not force and CALL.exists() and CALL.stat().st_mtime >= _newest([src, PKG.parent / "include" / "muser_cuda.h"]):
        return CALL
    cmd = [nvcc(), "-shared", "-cudart", "none", "-O2", "-Xcompiler", "-fPIC,-Wall,-Wno-unused-parameter", f"-I{include}", str(src), "-o", str(CALL), "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for host_call.c:\n" + r.stderr[-4000:])
    return CALL


def build(force: bool = False, verbose: bool = False) -> Path:
    build_call(force)
    srcs = [CSRC / s for s in SOURCES]
    deps = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + [PKG.parent / "include" / "muser_cuda.h"]
    if not force and LIB.exists() and LIB.stat().st_mtime >= _newest(srcs + deps):
        return LIB
    objdir = CSRC / "build"
    objdir.mkdir(exist_ok=True)

    def compile_one(src: Path) -> Path:
        obj = objdir / (src.stem + ".o")
        if not force and obj.exists() and obj.stat().st_mtime >= _newest([src] + deps):
            return obj
        extra = os.environ.get("MUSER_CUDA_NVCC_EXTRA", "").split()  # e.g. -DMUSER_GEMM_WAIT_PROFILE for a development build
        cmd = [nvcc(), *NVCC_FLAGS, *extra, "-Xptxas", "-v", "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        (objdir / (src.stem + ".ptxas.log")).write_text(r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stderr[-4000:]}")
        if verbose:
            print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    cmd = [nvcc(), "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
           "-Xlinker", "--version-script=" + str(CSRC / "exports.map"), "-lcudart_static", "-ldl", "-lrt", "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stderr[-4000:])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
