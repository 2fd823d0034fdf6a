"""Build libmoe_b200.so in-tree with nvcc for sm_100a, and the host extension _host.so with g++.

    python -m moe_routers_b200.build [--force] [--verbose]

The library is a plain C-ABI shared object (see include/moe_b200.h); it links
the CUDA runtime statically and resolves the one driver entry point it needs
(cuTensorMapEncodeTiled) at run time, so it builds on a machine without a GPU
or driver.
"""
from __future__ import annotations

import glob
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libmoe_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_PATH = os.path.join(PKG, "_host.so")
HOST_STAMP = os.path.join(LIB_DIR, "host_stamp.txt")  # what _host.so was built for
INCLUDE = os.path.join(os.path.dirname(PKG), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: libmoe_b200.so cannot be built")
    return cand


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(INCLUDE, "*.h"))
    return any(os.path.getmtime(p) > t for p in deps)


def _host_stamp() -> str:
    """What _host.so depends on besides its source: it reads torch's and Python's own structures."""
    return f"torch {importlib.metadata.version('torch')} {sysconfig.get_config_var('SOABI')}\n"


def _host_fresh(stamp: str) -> bool:
    if not os.path.exists(HOST_PATH) or os.path.getmtime(HOST_PATH) < max(
            os.path.getmtime(p) for p in [HOST_SRC] + glob.glob(os.path.join(INCLUDE, "*.h"))):
        return False
    try:
        with open(HOST_STAMP) as f:
            return f.read() == stamp
    except FileNotFoundError:
        return False


def build_host(force: bool = False) -> str:
    """Compile csrc/host.cpp against the installed torch's headers into the extension module _host.so (no-op if it
    is newer than its source and was built for this torch and this Python)."""
    stamp = _host_stamp()
    if not force and _host_fresh(stamp):
        return HOST_PATH
    import torch

    torch_dir = os.path.dirname(torch.__file__)
    includes = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
                sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for path in includes:
        cmd += ["-isystem", path]
    cmd += [HOST_SRC, "-o", HOST_PATH, "-L", os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError(f"g++ failed on {HOST_SRC}")
    os.makedirs(LIB_DIR, exist_ok=True)
    with open(HOST_STAMP, "w") as f:
        f.write(stamp)
    return HOST_PATH


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into lib/libmoe_b200.so, and where torch is installed host.cpp into _host.so
    (no-op if fresh)."""
    path = _build_cuda(force, verbose)
    if importlib.util.find_spec("torch") is not None:
        build_host(force)
    return path


def _build_cuda(force: bool, verbose: bool) -> str:
    if not force and not _stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    nvcc = _nvcc()
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    procs = []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if (not force and os.path.exists(obj)
                and os.path.getmtime(obj) > max(os.path.getmtime(p) for p in
                                                [src] + glob.glob(os.path.join(CSRC, "*.cuh"))
                                                + glob.glob(os.path.join(INCLUDE, "*.h")))):
            continue
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objs]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError("link of libmoe_b200.so failed")
    return LIB_PATH


if __name__ == "__main__":
    path = build_library(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
