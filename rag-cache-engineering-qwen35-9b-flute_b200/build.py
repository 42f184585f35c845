"""Build libb200lut.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

python build.py            # incremental: recompiles sources newer than their object
python build.py --force
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libb200lut.so")
HOST = os.path.join(HERE, "_b200lut_host.so")      # native host layer (torch C++), links LIB
SOURCES = ("api.cu", "layout.cu", "gemv.cu", "fht.cu", "gemm_tc.cu", "gemm_cluster.cu", "peer.cu", "residual.cu", "elementwise.cu", "embed.cu", "gemv_kgrouped.cu")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA library cannot be built")
    return exe


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src: str, force: bool) -> str:
    obj = os.path.join(OBJ, os.path.splitext(src)[0] + ".o")
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh") or f == src]
    deps.append(os.path.join(HERE, "..", "include", "b200_lut.h"))
    if force or _stale(obj, deps):
        extra = os.environ.get("B200LUT_NVCC_EXTRA", "").split()
        cmd = [_nvcc(), *NVCC_FLAGS, *extra, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        with open(obj + ".log", "w") as f:
            f.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    return obj


def _compile_host(force: bool) -> str:
    import sysconfig

    import torch
    src = os.path.join(CSRC, "host")
    obj = os.path.join(OBJ, "host.o")
    deps = [os.path.join(src, f) for f in os.listdir(src)] + [os.path.join(HERE, "..", "include", "b200_lut.h")]
    if force or _stale(obj, deps):
        inc = os.path.join(os.path.dirname(torch.__file__), "include")
        cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"), "-isystem", cuda,
               "-I", sysconfig.get_paths()["include"], "-c", os.path.join(src, "host.cpp"), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"g++ failed on host.cpp:\n{r.stdout}\n{r.stderr}")
    return obj


def _link_host(obj: str, force: bool) -> None:
    import torch
    if not (force or _stale(HOST, [obj, LIB])):
        return
    tl = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "lib64")
    cmd = ["g++", "-shared", "-o", HOST, obj, "-L", HERE, "-l:libb200lut.so", "-L", tl, "-lc10", "-ltorch_cpu", "-ltorch",
           "-ltorch_python", "-lc10_cuda", "-ltorch_cuda", "-L", cuda, "-lcudart", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link of the host layer failed:\n{r.stdout}\n{r.stderr}")


def build_library(force: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    with concurrent.futures.ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as ex:
        host = ex.submit(_compile_host, force)
        objs = list(ex.map(lambda s: _compile(s, force), SOURCES))
    if force or _stale(LIB, objs):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _link_host(host.result(), force)
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv))
