"""Build the CUDA library in-tree with nvcc for sm_100a, and the native host path beside it.

    python -m simplicial_attention_b200.build [--force] [--verbose]

Produces ``simplicial_attention_b200/libsa2.so`` (C ABI in ``include/sa2.h``) and ``_sa2_torch.<versions>.so`` (the argument
blocks, allocations and autograd nodes of the Python entry points in C++, against torch's headers).
nvcc cross-compiles without a GPU, so this also serves as the build check.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libsa2.so")

ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA library cannot be built")


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _inputs() -> list[str]:
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")]
    files.append(os.path.join(ROOT, "include", "sa2.h"))
    files.append(os.path.abspath(__file__))
    return files


def is_stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(f) > t for f in _inputs())


def ext_path() -> str:
    """The extension is C++ against the headers of one Python and one torch: their versions are part of its name, so that
    another torch in the same tree builds its own instead of loading this one's."""
    import sysconfig

    import torch
    tag = f"{sysconfig.get_config_var('SOABI')}-torch{torch.__version__}-cxx11abi{int(torch._C._GLIBCXX_USE_CXX11_ABI)}"
    return os.path.join(PKG, f"_sa2_torch.{tag.replace('+', '_')}.so")


def ext_is_stale() -> bool:
    path = ext_path()
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(f) > t for f in (os.path.join(CSRC, "sa2_torch.cpp"), os.path.join(ROOT, "include", "sa2.h"),
                                                 os.path.abspath(__file__)))


def build_ext(force: bool = False) -> str:
    """Compile the extension if it is missing or older than its sources (host code only, so g++)."""
    path = ext_path()
    if not force and not ext_is_stale():
        return path
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = [os.path.join(ROOT, "include"), *cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    tmp = path + f".{os.getpid()}.tmp"
    cmd = [
        shutil.which("g++") or "g++", "-shared", "-fPIC", "-O2", "-std=c++17", "-DTORCH_EXTENSION_NAME=_sa2_torch", "-DTORCH_API_INCLUDE_EXTENSION_H",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[x for d in includes for x in ("-isystem", d)],
        os.path.join(CSRC, "sa2_torch.cpp"), "-o", tmp,
        "-L" + lib_dir, "-Wl,-rpath," + lib_dir, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python",
    ]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
    os.replace(tmp, path)
    return path


def build(force: bool = False, verbose: bool = False, out: str = LIB, defines: tuple[str, ...] = ()) -> str:
    """Compile libsa2.so if it is missing or older than its sources.  ``out`` and ``defines`` make a second
    build beside it (the diagnostic build with wait accounting, see waitprof.py); such a build is always redone."""
    if out == LIB and not force and not is_stale():
        return LIB
    cmd = [
        _nvcc(), "-shared", "-Xcompiler", "-fPIC", "-O3", "-std=c++17", "-lineinfo",
        *ARCH_FLAGS,
        "-I", os.path.join(ROOT, "include"), "-I", CSRC,
        "--expt-relaxed-constexpr", *["-D" + d for d in defines],
        "-o", out, *sources(),
    ]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
        print(" ".join(cmd), file=sys.stderr)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr, file=sys.stderr)
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_ext(force="--force" in sys.argv))
