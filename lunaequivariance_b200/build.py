"""Builds the C-ABI shared library ``_lib/libluna_b200.so`` from ``csrc/*.cu`` with nvcc for sm_100a, and the PyTorch
launch path ``_lib/luna_torch.so`` from ``csrc/torch_binding.cpp`` with the host compiler.

Usage: ``python -m lunaequivariance_b200.build [--force] [--verbose] [--lineinfo]``.  Objects are rebuilt only when a
source, a header or this file is newer; files compile in parallel.  No GPU is needed to build.
"""

from __future__ import annotations

import argparse
import concurrent.futures
import os
import shutil
import subprocess
import sys

PACKAGE_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PACKAGE_DIR, "csrc")
LIB_DIR = os.path.join(PACKAGE_DIR, "_lib")
BUILD_DIR = os.path.join(PACKAGE_DIR, "_lib", "obj")
LIBRARY = os.path.join(LIB_DIR, "libluna_b200.so")
BINDING = os.path.join(LIB_DIR, "luna_torch.so")

# Line tables are left out by default: they made the library four times as large (the edge kernels are unrolled into very many
# lines).  --lineinfo brings them back for profiling.
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
    # It made a library of 101 MB one of 20; with the kernels of three channels per lane it is 28.  A module is unpacked when its
    # first kernel is loaded: the first call of a layer takes 3.2 ms instead of 1.4, once for each kind of layer.
    "--compress-mode=size",
]


def find_nvcc() -> str:
    for candidate in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if candidate and os.path.exists(candidate):
            return candidate
    raise RuntimeError("nvcc not found; set NVCC or CUDA_HOME")


# uvu_edge_inst.cu is compiled once per (element type, channels per lane, shape); the shapes are those of uvu_edge.cuh
EDGE_SOURCE = "uvu_edge_inst.cu"
EDGE_LANES = (("float", 1), ("float", 2), ("float", 3), ("float", 4), ("double", 1), ("double", 2), ("double", 3))
EDGE_SHAPES = 11


def units() -> list[tuple[str, str, list[str]]]:
    """(source, object, extra flags) of everything the library is made of."""
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        source = os.path.join(CSRC, name)
        if name != EDGE_SOURCE:
            found.append((source, os.path.join(BUILD_DIR, name[:-3] + ".o"), []))
            continue
        for shape in reversed(range(EDGE_SHAPES)):
            for kind, lanes in EDGE_LANES:
                obj = os.path.join(BUILD_DIR, f"{name[:-3]}_{kind}{lanes}_{shape}.o")
                found.append((source, obj, [f"-DLUNA_EDGE_T={kind}", f"-DLUNA_EDGE_CPL={lanes}",
                                            f"-DLUNA_EDGE_SHAPE={shape}"]))
    # the longest to compile first
    return sorted(found, key=lambda unit: not unit[2])


def headers_mtime() -> float:
    paths = [os.path.join(CSRC, n) for n in os.listdir(CSRC) if n.endswith((".h", ".cuh"))]
    paths.append(os.path.join(os.path.dirname(PACKAGE_DIR), "include", "luna_b200.h"))
    paths.append(os.path.abspath(__file__))  # the flags
    return max(os.path.getmtime(p) for p in paths if os.path.exists(p))


def compile_one(nvcc: str, unit: tuple[str, str, list[str]], verbose: bool, ptxas_info: bool,
                lineinfo: bool) -> tuple[str, str]:
    source, obj, flags = unit
    command = [nvcc, *NVCC_FLAGS, *(["-lineinfo"] if lineinfo else []), *flags, "-c", source, "-o", obj]
    if ptxas_info:
        command[1:1] = ["-Xptxas", "-v"]
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"nvcc failed for {source} {flags}:\n{result.stdout}\n{result.stderr}")
    return obj, result.stderr if (verbose or ptxas_info) else ""


def build_binding(nvcc: str, newest_header: float, force: bool) -> None:
    """The torch extension: host code only; it finds the library's entry points at load time."""
    import sysconfig

    import torch

    source = os.path.join(CSRC, "torch_binding.cpp")
    if not force and os.path.exists(BINDING) and os.path.getmtime(BINDING) >= max(os.path.getmtime(source), newest_header):
        return
    root = torch.__path__[0]
    cuda_include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               cuda_include, "/usr/local/cuda/include", sysconfig.get_paths()["include"]]
    # The compiler that nvcc uses for its host code, and not CXX: a compiler that links the C++ runtime statically gives
    # the module a second copy of it beside torch's, and streams (error texts with sizes in them) then crash.
    command = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared",
               "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=luna_torch",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{path}" for path in include),
               source, "-o", BINDING, f"-L{os.path.join(root, 'lib')}", "-ltorch", "-ltorch_cpu", "-ltorch_python",
               "-lc10", "-lc10_cuda", "-ldl"]
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"building {BINDING} failed:\n{result.stdout}\n{result.stderr}")


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False, lineinfo: bool = False) -> str:
    nvcc = find_nvcc()
    os.makedirs(BUILD_DIR, exist_ok=True)
    newest_header = headers_mtime()
    todo, objects = [], []
    for source, obj, flags in units():
        objects.append(obj)
        stale = (force or ptxas_info or lineinfo or not os.path.exists(obj)
                 or os.path.getmtime(obj) < max(os.path.getmtime(source), newest_header))
        if stale:
            todo.append((source, obj, flags))
    workers = max(1, os.cpu_count() or 2)
    with concurrent.futures.ThreadPoolExecutor(max_workers=workers) as pool:
        binding = pool.submit(build_binding, nvcc, newest_header, force)
        if todo:
            for obj, log in pool.map(lambda unit: compile_one(nvcc, unit, verbose, ptxas_info, lineinfo), todo):
                if log:
                    print(log, file=sys.stderr)
        binding.result()
    wanted = {os.path.basename(o) for o in objects}
    for name in os.listdir(BUILD_DIR):  # drop objects of deleted sources
        if name.endswith(".o") and name not in wanted:
            os.remove(os.path.join(BUILD_DIR, name))
    if todo or not os.path.exists(LIBRARY):
        link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                "-o", LIBRARY, *objects]
        result = subprocess.run(link, capture_output=True, text=True)
        if result.returncode != 0:
            raise RuntimeError(f"link failed:\n{result.stdout}\n{result.stderr}")
    return LIBRARY


if __name__ == "__main__":
    parser = argparse.ArgumentParser()
    parser.add_argument("--force", action="store_true")
    parser.add_argument("--verbose", action="store_true")
    parser.add_argument("--ptxas-info", action="store_true", help="print registers/spills/shared memory per kernel")
    parser.add_argument("--lineinfo", action="store_true", help="rebuild with line tables, for profiling")
    arguments = parser.parse_args()
    print(build(arguments.force, arguments.verbose, arguments.ptxas_info, arguments.lineinfo))
