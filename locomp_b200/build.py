"""Build the CUDA shared library in-tree: locomp_b200/_lcq.so (sm_100a only), and the extension
module locomp_b200/_torch_calls (host C++) that calls it with torch tensors.

    python -m locomp_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
# LOCOMP_B200_LIB selects another build of the library (e.g. one compiled with different tuning macros)
LIB_PATH = os.environ.get("LOCOMP_B200_LIB") or os.path.join(PKG_DIR, "_lcq.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
    # a host-only constexpr function called from device code compiles to a trap: make that an error
    "-Werror", "cross-execution-space-call",
]

# the host path for torch tensors: plain C++ against the headers of the torch that is installed
CALLS_SOURCE = os.path.join(CSRC, "torch_calls.cpp")
CALLS_PATH = os.path.join(PKG_DIR, "_torch_calls" + sysconfig.get_config_var("EXT_SUFFIX"))


def _sources():
    out = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))]
    out.append(os.path.join(INCLUDE, "locomp_b200.h"))
    return out


def _older(path: str, sources) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(s) > t for s in sources)


def _calls_sources():
    return [CALLS_SOURCE, os.path.join(INCLUDE, "locomp_b200.h")]


def needs_build() -> bool:
    return _older(LIB_PATH, _sources()) or _older(CALLS_PATH, _calls_sources())


def _run(what: str, cmd, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + proc.stdout + proc.stderr)


def _build_calls(verbose: bool) -> None:
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    include = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_path("include"), os.path.join(cuda, "include")]
    _run("g++", [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
                 f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f"-I{d}" for d in include] +
         ["-o", CALLS_PATH, CALLS_SOURCE, "-L" + os.path.join(base, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
          "-lc10_cuda", "-lc10", "-ldl"], verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile csrc/lib.cu (which includes every kernel header) into _lcq.so, and csrc/torch_calls.cpp."""
    if force or _older(CALLS_PATH, _calls_sources()):
        _build_calls(verbose)
    if not force and not _older(LIB_PATH, _sources()):
        return LIB_PATH
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build locomp_b200/_lcq.so")
    _run("nvcc", [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH, os.path.join(CSRC, "lib.cu")], verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
