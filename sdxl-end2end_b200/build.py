"""Builds, in-tree, libsdxlq.so (the C-ABI library with the sm_100a kernels, nvcc) and _front.<tag>.so (the
Python mirror's native front over that ABI, g++)."""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
import warnings

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBRARY = os.path.join(HERE, "libsdxlq.so")
FRONT_SOURCES = ["torch_front.cpp", os.path.join("..", "..", "include", "sdxlq.h")]
SOURCES = ["capi.cu", "gemm_umma.cu", "quantize.cu", "quantize_int8_fast.cu", "linear_small.cu", "linear_skinny.cu", "layer_norm.cu", "harness_norm.cu"]
HEADERS = ["internal.cuh", "ptx.cuh", "quantize.cuh", "fp8_math.cuh", "int8_math.cuh", os.path.join("..", "..", "include", "sdxlq.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++20",
    "-Xcompiler", "-fPIC", "-shared",
    "--fmad=true",
]


def _newest(paths) -> float:
    return max(os.path.getmtime(p) for p in paths)


def needs_build() -> bool:
    if not os.path.exists(LIBRARY):
        return True
    inputs = [os.path.join(CSRC, s) for s in SOURCES] + [os.path.join(CSRC, h) for h in HEADERS]
    return _newest(inputs) > os.path.getmtime(LIBRARY)


def front_path() -> str:
    """The native front's file. It holds for one torch and one Python ABI, which its name states."""
    import torch
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    return os.path.join(HERE, f"_front.torch-{torch.__version__}-abi{abi}.{sysconfig.get_config_var('SOABI')}.so")


def build_front(force: bool = False) -> str:
    """Compiles the native front against the installed torch. Returns its path."""
    path = front_path()
    inputs = [os.path.join(CSRC, s) for s in FRONT_SOURCES]
    if not force and os.path.exists(path) and _newest(inputs) <= os.path.getmtime(path):
        return path
    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    include, libraries = os.path.join(root, "include"), os.path.join(root, "lib")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    command = ["g++", "-O2", "-std=c++20", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               "-I", sysconfig.get_paths()["include"], "-isystem", include,
               "-isystem", os.path.join(include, "torch", "csrc", "api", "include"), "-isystem", os.path.join(cuda, "include"),
               "-o", path, inputs[0], "-L", libraries, "-lc10", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        sys.stderr.write(result.stdout + result.stderr)
        raise RuntimeError("g++ failed building the native front")
    return path


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles every CUDA source for sm_100a into one shared library, then the native front (without which the mirror
    issues its calls through ctypes: a warning). Returns the library's path."""
    if force or needs_build():
        _build_library(verbose)
    try:
        build_front(force)
    except (OSError, RuntimeError) as error:
        warnings.warn(f"the native front was not built, calls go through ctypes: {error}", RuntimeWarning)
    return LIBRARY


def _build_library(verbose: bool) -> None:
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    command = [nvcc, *NVCC_FLAGS]
    if verbose:
        command += ["-Xptxas", "-v"]
    command += ["-o", LIBRARY] + [os.path.join(CSRC, s) for s in SOURCES]
    result = subprocess.run(command, capture_output=True, text=True)
    if verbose or result.returncode != 0:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode != 0:
        raise RuntimeError("nvcc failed building libsdxlq.so")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
