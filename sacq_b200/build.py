"""Builds ``libsacq_b200.so`` in-tree with nvcc for sm_100a, and ``_native.so``, the host side of the
layer calls as a CPython extension (g++ against the installed PyTorch), beside it.

    python -m sacq_b200.build [--force] [--verbose]

One object per ``csrc/*.cu`` (compiled in parallel), linked into
``sacq_b200/libsacq_b200.so``.  nvcc cross-compiles without a GPU, so this
also serves as the "does it build" check on a CPU-only machine.
"""
from __future__ import annotations

import argparse
import concurrent.futures
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(HERE, "build")
LIB_PATH = os.path.join(HERE, "libsacq_b200.so")
NATIVE_SRC = os.path.join(CSRC, "host", "native_calls.cpp")
NATIVE_PATH = os.path.join(HERE, "_native.so")
NATIVE_KEY_PATH = os.path.join(OBJ_DIR, "native.key")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the sacq_b200 CUDA library cannot be built")
    return exe


def _sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps():
    return _sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "host", "*.h")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h")) + [os.path.abspath(__file__)]


def up_to_date() -> bool:
    if not os.path.exists(LIB_PATH):
        return False
    t = os.path.getmtime(LIB_PATH)
    return all(os.path.getmtime(p) <= t for p in _deps())


def native_key() -> str:
    """What a build of the extension module is bound to, besides its sources: one Python and one PyTorch."""
    import torch
    return f"{sys.version}\n{torch.__version__} {torch.version.git_version} {torch.compiled_with_cxx11_abi()}\n"


def native_up_to_date() -> bool:
    deps = [NATIVE_SRC, os.path.join(CSRC, "host", "internal.h"), os.path.abspath(__file__)] + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    if not os.path.exists(NATIVE_PATH) or any(os.path.getmtime(p) > os.path.getmtime(NATIVE_PATH) for p in deps):
        return False
    try:
        with open(NATIVE_KEY_PATH) as f:
            return f.read() == native_key()
    except OSError:
        return False


def build_native(force: bool = False) -> str:
    """Compile the extension module if its source or the public header is newer, or if it was built for another Python or
    PyTorch.  Returns its path."""
    if not force and native_up_to_date():
        return NATIVE_PATH
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include",
           f"-I{sysconfig.get_paths()['include']}", NATIVE_SRC, "-o", NATIVE_PATH,
           f"-L{root}/lib", f"-L{HERE}", "-l:libsacq_b200.so", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed for %s:\n%s\n%s" % (NATIVE_SRC, res.stdout, res.stderr))
    os.makedirs(OBJ_DIR, exist_ok=True)
    with open(NATIVE_KEY_PATH, "w") as f:
        f.write(native_key())
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> str:
    """Compile and link the library (and the extension module) where a source is newer.  Returns the library's path."""
    if not force and up_to_date():
        build_native()
        return LIB_PATH
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    flags = list(NVCC_FLAGS) + (["-Xptxas", "-v"] if ptxas_info else []) + os.environ.get("SACQ_NVCC_EXTRA", "").split()

    def compile_one(src):
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc] + flags + ["-c", src, "-o", obj]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, res.stdout, res.stderr))
        if verbose or ptxas_info:
            sys.stderr.write(res.stderr)
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, _sources()))
    cmd = [nvcc, "-shared", "-o", LIB_PATH] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("link failed:\n%s\n%s" % (res.stdout, res.stderr))
    build_native(force)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--ptxas-info", action="store_true", help="print registers/spills/shared memory per kernel")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose, ptxas_info=a.ptxas_info))
