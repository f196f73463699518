"""Build recipe of the CUDA library (nvcc, sm_100a only, in-tree output)."""

from __future__ import annotations

import glob
import os
import subprocess
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
LIB_PATH = os.path.join(PKG_DIR, "libturboquant_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "tq_host.cpp")
HOST_PATH = os.path.join(PKG_DIR, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC", "--threads", "0",      # the .cu files compile in parallel
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def needs_build() -> bool:
    headers = glob.glob(os.path.join(INCLUDE, "*.h"))
    return (_stale(LIB_PATH, sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + headers)
            or _stale(HOST_PATH, [HOST_SRC] + headers))


def _stale(target: str, deps: list[str]) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(p) > os.path.getmtime(target) for p in deps)


def _host_command() -> list[str]:
    """g++ line of the CPython extension: torch's headers and libraries, the CUDA library next to it."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-I", INCLUDE, "-I", os.path.join(root, "include"), "-I", sysconfig.get_paths()["include"],
            "-I", os.path.join(cuda, "include"), "-o", HOST_PATH, HOST_SRC,
            "-L", PKG_DIR, "-lturboquant_b200", "-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10",
            "-lc10_cuda", "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + os.path.join(root, "lib")]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into libturboquant_b200.so next to this file, and the host extension."""
    if not force and not needs_build():
        return LIB_PATH
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-I", CSRC, "-o", LIB_PATH, *sources()]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)
    host = subprocess.run(_host_command(), capture_output=True, text=True)
    if host.returncode != 0:
        raise RuntimeError("the host extension did not compile:\n" + host.stdout + host.stderr)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
