"""Builds ``libugache_b200.so`` (CUDA kernels + C ABI) in-tree with nvcc for sm_100a.

The library links the CUDA runtime statically and nothing else from CUDA, so it loads on a
machine without a GPU or driver (host-side entry points work there; device entry points
return an error status).
"""
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libugache_b200.so")
FAST = os.path.join(HERE, "_fast.so")  # the Python face's per-step calls (links against torch)
STAMP = os.path.join(HERE, "build", "stamp.txt")
FAST_STAMP = os.path.join(HERE, "build", "fast_stamp.txt")

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


def _fingerprint(names, command):
    h = hashlib.sha256()
    for name in names:
        path = os.path.join(CSRC, name)
        if os.path.exists(path):
            with open(path, "rb") as f:
                h.update(name.encode())
                h.update(f.read())
    h.update(" ".join(command).encode())
    return h.hexdigest()


def _up_to_date(path, stamp, fp):
    if not (os.path.exists(path) and os.path.exists(stamp)):
        return False
    with open(stamp) as f:
        return f.read().strip() == fp


def _write(path, text):
    with open(path, "w") as f:
        f.write(text)


FAST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
FAST_LIBS = ["-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def build_fast(force=False):
    """Compile the extension module if its source, the interpreter or torch changed; without torch there is
    none (the C library does not need it)."""
    try:
        import torch

        from ._lib import fast_abi
        abi = fast_abi()
    except ImportError as e:
        print("ugache_b200: %s is not built, torch cannot be imported (%s)" % (os.path.basename(FAST), e), file=sys.stderr)
        return
    fp = _fingerprint([FAST_SOURCE, "../../include/ugache_b200.h"], [abi] + FAST_FLAGS + FAST_LIBS)
    if not force and _up_to_date(FAST, FAST_STAMP, fp):
        return
    import sysconfig

    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = ["g++"] + FAST_FLAGS + ['-DUGC_BUILT_FOR="%s"' % abi,
                                  "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI]
    cmd += [os.path.join(CSRC, FAST_SOURCE), "-o", FAST]
    for i in inc:
        cmd += ["-isystem", i]
    cmd += ["-L" + os.path.join(os.path.dirname(torch.__file__), "lib")] + FAST_LIBS
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed on %s:\n%s" % (FAST_SOURCE, r.stderr))
    _write(FAST_STAMP, fp)


def build(force=False, verbose=False):
    """Compile the shared library and the extension module if sources changed.  Returns the library's path."""
    os.makedirs(os.path.dirname(STAMP), exist_ok=True)
    fp = _fingerprint(CUDA_SOURCES + HOST_SOURCES + HEADERS, NVCC_FLAGS)
    if force or not _up_to_date(LIB, STAMP, fp):
        log = _build_library()
        _write(STAMP, fp)
        if verbose:
            print("\n".join(log))
    build_fast(force)
    return LIB


def _build_library():
    nvcc = _nvcc()
    bdir = os.path.join(HERE, "build")
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
    _write(os.path.join(bdir, "ptxas.log"), "\n".join(log))
    return log


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
