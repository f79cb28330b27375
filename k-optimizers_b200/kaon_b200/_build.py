"""Build libkaon_b200.so in-tree with nvcc for sm_100a.

    python -m kaon_b200._build [--force] [-v]     (from the directory that holds the package)

Every .cu file is compiled to an object of its own (in parallel, only when it or a header changed) and
the objects are linked into the shared library.  host_ext.cpp becomes the CPython module _kaon_host (the
per-tensor host work of a step), against the installed torch's headers.
-fmad=false: the kernels spell out every fused multiply-add the reference's torch ops perform and
must not get any other.  The library has no torch dependency: it is loaded with ctypes.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(PKG), "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(PKG, "libkaon_b200.so")
HOST_SRC = os.path.join(CSRC, "host_ext.cpp")
HOST_LIB = os.path.join(PKG, "_kaon_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-fmad=false",
    "-Xcompiler", "-fPIC",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def headers() -> list[str]:
    deps = glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    deps += glob.glob(os.path.join(os.path.dirname(os.path.dirname(PKG)), "include", "*.h"))
    return deps


def _obj(src: str) -> str:
    return os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")


def needs_build() -> bool:
    if not os.path.exists(LIB) or _host_stale():
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(d) > t for d in sources() + headers())


def host_abi() -> str:
    """What the host module is compiled for: it reads tensor objects by torch's layout of them."""
    import torch
    return f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"


def _host_stale() -> bool:
    """Missing, older than its source, or compiled for another torch or Python (its `abi` string, as the file holds it)."""
    if not os.path.exists(HOST_LIB) or os.path.getmtime(HOST_LIB) < os.path.getmtime(HOST_SRC):
        return True
    with open(HOST_LIB, "rb") as f:
        return f"kaon host module for {host_abi()}\0".encode() not in f.read()


def _build_host(env: dict) -> None:
    """The host module: torch's headers for the layout of a tensor object, its libraries for the symbols
    (they are loaded by ``import torch`` before the module is)."""
    import torch
    from torch.utils.cpp_extension import include_paths
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.check_call(
        ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f'-DKAON_HOST_ABI="{host_abi()}"', f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
         *[f"-I{p}" for p in include_paths()], f"-I{sysconfig.get_paths()['include']}", HOST_SRC, "-o", HOST_LIB,
         f"-L{libs}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", f"-Wl,-rpath,{libs}"], env=env)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    env = dict(os.environ)
    env.pop("CC", None)   # let nvcc pick its default host compiler
    env.pop("CXX", None)
    os.makedirs(OBJ, exist_ok=True)
    hdr_time = max(os.path.getmtime(h) for h in headers())

    def compile_one(src: str) -> str:
        obj = _obj(src)
        if (not force and os.path.exists(obj)
                and os.path.getmtime(obj) > max(os.path.getmtime(src), hdr_time)):
            return obj
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
            print(" ".join(cmd), flush=True)
        subprocess.check_call(cmd, env=env)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        host = pool.submit(_build_host, env) if force or _host_stale() else None
        objs = list(pool.map(compile_one, sources()))
        if host is not None:
            host.result()
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "--shared", "-o", LIB, *objs],
                          env=env)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
