"""Build libquik_b200.so in-tree with nvcc for sm_100a, and the CPython module _host (csrc/host_ext.cpp) with g++.

    python -m quik_b200.build            # build if sources are newer than the library
    python -m quik_b200.build --force

The library is a plain C-ABI shared object (see include/quik_b200.h); it links the CUDA
runtime statically and needs no GPU to build or to load.  _host is built against the headers and libraries of the torch that
is installed; neither depends on the other at link time.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libquik_b200.so")
HOST_EXT = os.path.join(HERE, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))     # native host path (csrc/host_ext.cpp)
SOURCES = ["abi.cu", "quantize.cu", "dequantize.cu", "gemm_mma_sync.cu", "gemm_tcgen05.cu", "gemm_tcgen05_ts.cu", "smallm.cu", "stream_w.cu", "stream_w_mma.cu", "selftest.cu", "rotary.cu", "peer_copy.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def needs_build() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(HOST_EXT):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST_EXT))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "quik_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _build_host_ext() -> None:
    """g++ against the headers of torch, CPython and the CUDA runtime."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    inc = [sysconfig.get_paths()["include"], os.path.join(root, "include"),
           os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{d}" for d in inc], os.path.join(CSRC, "host_ext.cpp"), "-o", HOST_EXT,
           "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for host_ext.cpp:\n{r.stdout}\n{r.stderr}")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)

    def compile_one(src: str) -> str:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as pool:
        ext = pool.submit(_build_host_ext)
        objs = list(pool.map(compile_one, SOURCES))
        ext.result()
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
