"""Ahead-of-time build of ``libnmg_b200.so`` (the C-ABI CUDA library) for sm_100a and of ``_nmg_host.so`` (the CPython
extension that checks tensors, allocates and calls the library).

    python -m sten_b200.build [--force] [--verbose]

Every translation unit under ``csrc/`` is compiled with
``nvcc -gencode arch=compute_100a,code=sm_100a -lineinfo`` (cross-compiles without a GPU) and linked into
``sten_b200/libnmg_b200.so`` next to this file, so the library travels with the source tree.  There is no
run-time code generation: shapes are kernel arguments, (n, m) specialisations are template instances.
"""
import argparse
import concurrent.futures
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libnmg_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "nmg_host.cpp")
HOST_LIB = os.path.join(HERE, "_nmg_host.so")
OBJ_DIR = os.path.join(HERE, "csrc", "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(exe):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stamp():
    h = hashlib.sha256()
    for root in (CSRC, os.path.join(os.path.dirname(HERE), "include")):
        for f in sorted(os.listdir(root)):
            p = os.path.join(root, f)
            if os.path.isfile(p) and f.endswith((".cu", ".cuh", ".h")):
                h.update(f.encode())
                with open(p, "rb") as fh:
                    h.update(fh.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def build_host(force=False, verbose=False):
    """The host extension: one C++ file against the Python and torch headers, linked to the library next to it."""
    import torch
    from torch.utils import cpp_extension
    h = hashlib.sha256(torch.__version__.encode() + sys.version.encode())
    for p in (HOST_SRC, os.path.join(os.path.dirname(HERE), "include", "nmg_b200.h")):
        with open(p, "rb") as fh:
            h.update(fh.read())
    stamp, stamp_file = h.hexdigest(), os.path.join(OBJ_DIR, "stamp_host")
    if not force and os.path.isfile(HOST_LIB) and os.path.isfile(stamp_file) and open(stamp_file).read() == stamp:
        return HOST_LIB
    tmp = HOST_LIB + f".{os.getpid()}.tmp"
    include = [sysconfig.get_paths()["include"], *cpp_extension.include_paths("cuda")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{p}" for p in include], HOST_SRC, "-o", tmp, *[f"-L{p}" for p in cpp_extension.library_paths("cuda")], f"-L{HERE}",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-l:libnmg_b200.so", "-Wl,-rpath,$ORIGIN"]
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on {HOST_SRC}:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, HOST_LIB)
    with open(stamp_file, "w") as f:
        f.write(stamp)
    return HOST_LIB


def build(force=False, verbose=False):
    lib = build_lib(force, verbose)
    build_host(force, verbose)
    return lib


def build_lib(force=False, verbose=False):
    stamp_file = os.path.join(OBJ_DIR, "stamp")
    stamp = _stamp()
    if not force and os.path.isfile(LIB) and os.path.isfile(stamp_file) and open(stamp_file).read() == stamp:
        return LIB
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src):
        obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    tmp = LIB + f".{os.getpid()}.tmp"
    cmd = [nvcc, "-shared", "-Xlinker", "-soname=libnmg_b200.so", "-o", tmp, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, LIB)
    with open(stamp_file, "w") as f:
        f.write(stamp)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", "-v", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
    sys.exit(0)
