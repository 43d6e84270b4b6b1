"""Builds ``libugache_b200.so`` (CUDA kernels + C ABI) in-tree with nvcc for sm_100a.

The library links the CUDA runtime statically and nothing else from CUDA, so it loads on a
machine without a GPU or driver (host-side entry points work there; device entry points
return an error status).
"""
import hashlib
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libugache_b200.so")
FAST = os.path.join(HERE, "_fast.so")  # the Python face's per-step calls (links against torch)
STAMP = os.path.join(HERE, "build", "stamp.txt")

CUDA_SOURCES = ["kernels.cu", "api.cu"]
HOST_SOURCES = ["placement.cc", "compat_api.cc"]
FAST_SOURCE = "pyfast.cc"
HEADERS = ["device_types.h", "kernels.cuh", "placement.h", "../../include/ugache_b200.h",
           "../../include/coll_cache_api.h", "../../include/coll_cache_lib/facade.h"]

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC,-fopenmp,-Wall", "-Xptxas", "-v"]


def _nvcc():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: the CUDA extension cannot be built")
    return nvcc


def _fingerprint():
    h = hashlib.sha256()
    for name in CUDA_SOURCES + HOST_SOURCES + [FAST_SOURCE] + HEADERS:
        path = os.path.join(CSRC, name)
        if os.path.exists(path):
            with open(path, "rb") as f:
                h.update(name.encode())
                h.update(f.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def _build_fast():
    """The extension module for the interpreter and torch that run this."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI, os.path.join(CSRC, FAST_SOURCE), "-o", FAST]
    for i in inc:
        cmd += ["-isystem", i]
    cmd += ["-L" + tlib, "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed on %s:\n%s" % (FAST_SOURCE, r.stderr))


def build(force=False, verbose=False):
    """Compile the shared library and the extension module if sources changed.  Returns the library's path."""
    fp = _fingerprint()
    if not force and all(map(os.path.exists, (LIB, FAST, STAMP))):
        with open(STAMP) as f:
            if f.read().strip() == fp:
                return LIB
    nvcc = _nvcc()
    bdir = os.path.join(HERE, "build")
    os.makedirs(bdir, exist_ok=True)
    objs = []
    log = []
    for src in CUDA_SOURCES + HOST_SOURCES:
        path = os.path.join(CSRC, src)
        if not os.path.exists(path):
            continue
        obj = os.path.join(bdir, os.path.splitext(src)[0] + ".o")
        cmd = [nvcc] + NVCC_FLAGS + ["-c", path, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        log.append(r.stderr)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed on %s:\n%s" % (src, r.stderr))
        objs.append(obj)
    cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-cudart", "static", "-Xcompiler", "-fopenmp",
                                                  "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s" % r.stderr)
    _build_fast()
    with open(os.path.join(bdir, "ptxas.log"), "w") as f:
        f.write("\n".join(log))
    with open(STAMP, "w") as f:
        f.write(fp)
    if verbose:
        print("\n".join(log))
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
