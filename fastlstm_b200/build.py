"""Build libfastlstm_b200.so (nvcc, sm_100a) and the CPython extension _host in-tree.

    python -m fastlstm_b200.build [--force] [--verbose]

The library is plain CUDA C++ behind an extern "C" ABI (include/fastlstm_b200.h) and does not link libtorch;
_host (csrc/host.cpp) is the host side of the layer operators and does.  Both build offline in about a minute.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libfastlstm_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_PATH = os.path.join(PKG_DIR, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))
HEADERS = glob.glob(os.path.join(PKG_DIR, "..", "include", "*.h"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared", "--threads", "0",     # one compiler process per source file
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; cannot build libfastlstm_b200.so")
    return exe


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target, deps):
    return not os.path.exists(target) or any(os.path.getmtime(p) > os.path.getmtime(target) for p in deps)


def _run(cmd, what, verbose):
    if verbose:
        print(" ".join(cmd))
    p = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)

    def finish():
        log, _ = p.communicate()
        sys.stderr.write(log)                 # (silent but for warnings and errors)
        if p.returncode != 0:
            raise RuntimeError(f"compiler failed building {what}")
    return finish


def _host_cmd():
    import torch
    from torch.utils import cpp_extension as ext
    lib_dirs = [os.path.join(os.path.dirname(torch.__file__), "lib"), os.path.join(os.path.dirname(_nvcc()), "..", "lib64")]
    return ([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-Wall",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_host"]
            + [f"-I{d}" for d in ext.include_paths(device_type="cuda") + [sysconfig.get_paths()["include"]]]
            + ["-o", HOST_PATH, HOST_SRC, f"-L{PKG_DIR}", "-l:libfastlstm_b200.so", "-Wl,-rpath,$ORIGIN"]
            + [f"-L{d}" for d in lib_dirs] + ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-lcudart"])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library, and _host; returns the library's path."""
    lib_deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + HEADERS
    if force or _stale(LIB_PATH, lib_deps):
        _run([_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] + sources() + ["-lcuda"],
             "libfastlstm_b200.so", verbose)()
    if force or _stale(HOST_PATH, [HOST_SRC] + HEADERS):
        _run(_host_cmd(), "_host", verbose)()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
