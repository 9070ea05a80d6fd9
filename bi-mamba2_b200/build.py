"""Build libbissd.so (the CUDA kernels + C ABI) and _bissd_torch.so (the operator's native host path) in-tree.

    python bi-mamba2_b200/build.py [--force] [--verbose]

Both land in bi-mamba2_b200/ssd/_lib/.  libbissd.so is compiled by nvcc for sm_100a and has no PyTorch in it (the
package also loads it with ctypes); _bissd_torch.so is a Python extension compiled by g++ against the installed PyTorch
and linked to libbissd.so.  Neither needs a GPU to build.
"""
import argparse
import concurrent.futures
import os
import re
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "ssd", "_lib")
OUT = os.path.join(OUT_DIR, "libbissd.so")
SOURCES = ["bissd_api.cu", "bissd_layer.cu", "bissd_simt.cu"]
TORCH_SRC = os.path.join(CSRC, "torch_ops.cpp")
TORCH_OUT = os.path.join(OUT_DIR, "_bissd_torch.so")


def _newest_source_mtime(source):
    """Newest of a source file and what it includes from this repository, directly or not."""
    seen, todo = set(), [os.path.join(CSRC, source)]
    while todo:
        path = todo.pop()
        if path not in seen:
            seen.add(path)
            with open(path) as f:
                names = re.findall(r'^#include "([^"]+)"', f.read(), flags=re.M)
            todo += [os.path.normpath(os.path.join(os.path.dirname(path), n)) for n in names]
    return max(os.path.getmtime(p) for p in seen)


def _run(cmd, verbose, what):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed building {what}")


def build_torch(force=False, verbose=False):
    """The extension depends on its own source and the C header only: libbissd.so may be rebuilt beneath it."""
    header = os.path.join(os.path.dirname(HERE), "include", "bissd.h")
    newest = max(os.path.getmtime(TORCH_SRC), os.path.getmtime(header))
    if not force and os.path.exists(TORCH_OUT) and os.path.getmtime(TORCH_OUT) >= newest:
        return TORCH_OUT
    import torch
    from torch.utils import cpp_extension
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_bissd_torch"]
    for path in cpp_extension.include_paths() + [os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]:
        cmd += ["-isystem", path]
    cmd += [TORCH_SRC, "-o", TORCH_OUT, "-L" + OUT_DIR, "-l:libbissd.so", "-Wl,-rpath,$ORIGIN"]
    cmd += ["-L" + os.path.join(os.path.dirname(torch.__file__), "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch",
            "-ltorch_python"]
    _run(cmd, verbose, os.path.basename(TORCH_OUT))
    return TORCH_OUT


def build(force=False, verbose=False):
    os.makedirs(OUT_DIR, exist_ok=True)
    build_library(force, verbose)
    build_torch(force, verbose)
    return OUT


def build_library(force=False, verbose=False):
    if not force and os.path.exists(OUT) and os.path.getmtime(OUT) >= max(map(_newest_source_mtime, SOURCES)):
        return OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    flags = ["-std=c++17", "-O3", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
             "--extended-lambda", "-Xcompiler", "-fPIC"] + (["-Xptxas", "-v"] if verbose else [])
    objs = [os.path.join(OUT_DIR, s.replace(".cu", ".o")) for s in SOURCES]
    stale = [(s, o) for s, o in zip(SOURCES, objs) if force or not os.path.exists(o) or os.path.getmtime(o) < _newest_source_mtime(s)]
    with concurrent.futures.ThreadPoolExecutor() as pool:                # one nvcc per translation unit, side by side
        list(pool.map(lambda so: _run([nvcc, *flags, "-c", "-o", so[1], os.path.join(CSRC, so[0])], verbose, so[0]), stale))
    _run([nvcc, "-shared", "-o", OUT, *objs], verbose, os.path.basename(OUT))
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
