"""Builds ``liblloom_b200.so`` (nvcc, sm_100a only) and the Python binding ``_native.so`` (g++) in-tree, no JIT cache."""
from __future__ import annotations

import os
import shutil
import subprocess

_PKG = os.path.dirname(os.path.abspath(__file__))
SRC_DIR = os.path.join(_PKG, "csrc")
LIB_PATH = os.path.join(_PKG, "liblloom_b200.so")
NATIVE_PATH = os.path.join(_PKG, "_native.so")
NATIVE_SRC = os.path.join(SRC_DIR, "python", "native.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--shared", "-Xcompiler", "-fPIC",
    "-Xcompiler", "-ffp-contract=off",  # host-side quantizers: strict sequential f32, like the reference
]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build liblloom_b200.so")
    return nvcc


def sources() -> list[str]:
    out = []
    for root, _, files in os.walk(SRC_DIR):
        out += [os.path.join(root, f) for f in files if f.endswith((".cu", ".cuh", ".h", ".hpp", ".cpp"))]
    inc = os.path.join(os.path.dirname(_PKG), "include")
    out += [os.path.join(inc, f) for f in os.listdir(inc) if f.endswith(".h")]
    return sorted(out)


def is_stale() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(NATIVE_PATH):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(NATIVE_PATH))
    return any(os.path.getmtime(s) > t for s in sources())


def translation_units() -> list[str]:
    """Every .cu / .cpp under csrc/: the kernels are split over several units so that they compile in parallel."""
    out = []
    for root, _, files in os.walk(SRC_DIR):
        out += [os.path.join(root, f) for f in files if f.endswith((".cu", ".cpp"))]
    return sorted(p for p in out if p != NATIVE_SRC)


def native_command(obj: str) -> list[str]:
    """Compiler command of the Python binding: a plain extension module against torch's C++ API."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext

    cuda_home = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [*ext.include_paths(), os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[f for p in inc for f in ("-isystem", p)], "-c", NATIVE_SRC, "-o", obj]


def native_link_command(obj: str) -> list[str]:
    from torch.utils import cpp_extension as ext

    libs = [f for p in ext.library_paths() for f in (f"-L{p}", f"-Wl,-rpath,{p}")]
    return ["g++", "-shared", "-o", NATIVE_PATH, obj, *libs, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch",
            "-ltorch_python", f"-L{_PKG}", "-l:liblloom_b200.so", "-Wl,-rpath,$ORIGIN"]


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source of the package (one object per translation unit, in parallel), link them into one
    shared library and the Python binding against it; returns the library's path."""
    if not force and not is_stale():
        return LIB_PATH
    from concurrent.futures import ThreadPoolExecutor

    obj_dir = os.path.join(_PKG, "build")
    os.makedirs(obj_dir, exist_ok=True)
    compile_flags = [f for f in NVCC_FLAGS if f != "--shared"]

    def compile_unit(src: str) -> tuple[str, str]:
        obj = os.path.join(obj_dir, os.path.basename(src) + ".o")
        if src == NATIVE_SRC:
            res = subprocess.run(native_command(obj), capture_output=True, text=True)
            if res.returncode != 0:
                raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
            return obj, res.stderr
        cmd = [_nvcc(), *compile_flags, "-c", src, "-o", obj]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
        return obj, res.stderr

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        results = list(pool.map(compile_unit, [NATIVE_SRC, *translation_units()]))
    if verbose:
        for _, log in results:
            print(log)
    cmd = [_nvcc(), "--shared", "-o", LIB_PATH, *[obj for obj, _ in results[1:]]]
    for cmd in (cmd, native_link_command(results[0][0])):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    return LIB_PATH


if __name__ == "__main__":
    import sys

    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
