"""In-tree build of the three shared libraries (no cmake, no JIT cache).

* ``lib/libdtq_b200.so``   -- the torch-free CUDA kernels and their C ABI
  (``include/dtq_b200.h``), built with nvcc for sm_100a only.
* ``lib/libdriss_torch.so`` -- ``register_ops.cpp``: the ``TORCH_LIBRARY(DrissTorch)``
  registration that binds the C ABI into the PyTorch dispatcher, built with g++.
* ``lib/_direct.<python ABI>.so`` -- ``direct_calls.cpp``: the operators as plain Python functions (an extension
  module), built with g++.

``python driss_torch_b200/build.py`` builds all; objects are rebuilt only when a
source or header is newer, the two that are linked to torch also for another torch, Python or command.  The reference builds one ``libdriss_torch.so`` through
scikit-build/CMake with the same architecture flags (CMakeLists.txt:25-27).
"""
from __future__ import annotations

import importlib.machinery
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB = PKG / "lib"
OBJ = PKG / "build"
INCLUDE = ROOT / "include"

CUDA_HOME = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
NVCC = str(CUDA_HOME / "bin" / "nvcc")

KERNEL_SOURCES = [
    "common.cu",
    "saturated_cast.cu",
    "saturated_cast_t.cu",
    "amax.cu",
    "dynamic_scaled_quant.cu",
    "rowwise_quant.cu",
    "mx_cast.cu",
    "mx_cast_tma.cu",
    "mx_cast_dual.cu",
    "mx_cast_formats.cu",
    "mx_cast_amax.cu",
    "mx_gemm.cu",
]

NVCC_FLAGS = [
    "-std=c++17",
    "-O3",
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-Xcompiler",
    "-fPIC",
    "-Xptxas",
    "-v",
    "--cudart",
    "shared",
]


def _newest(paths) -> float:
    return max(p.stat().st_mtime for p in paths)


def _headers():
    return list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))


def _run(cmd, log: Path | None = None) -> None:
    proc = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if log is not None:
        log.write_text(proc.stdout)
    if proc.returncode != 0:
        sys.stderr.write(proc.stdout)
        raise RuntimeError("build step failed: " + " ".join(map(str, cmd)))


def build_kernels(force: bool = False, extra_flags=()) -> Path:
    LIB.mkdir(exist_ok=True)
    OBJ.mkdir(exist_ok=True)
    dep_time = _newest(_headers() + [Path(__file__)])
    jobs = []
    objs = []
    for name in KERNEL_SOURCES:
        src = CSRC / name
        obj = OBJ / (src.stem + ".o")
        objs.append(obj)
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, dep_time):
            cmd = [NVCC, *NVCC_FLAGS, *extra_flags, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
            jobs.append((cmd, OBJ / (src.stem + ".ptxas.log")))
    with ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as pool:
        list(pool.map(lambda j: _run(*j), jobs))
    so = LIB / "libdtq_b200.so"
    if force or jobs or not so.exists():
        _run([NVCC, "-shared", "--cudart", "shared", "-o", str(so), *map(str, objs),
              "-Xlinker", "-rpath", "-Xlinker", str(CUDA_HOME / "lib64")])
    return so


def made_for(cmd) -> str:
    """What a library linked to torch was made with: it has to be made again for any other."""
    import torch

    return "\n".join([f"torch {torch.__version__} {torch.version.git_version}", sysconfig.get_config_var("SOABI"), " ".join(map(str, cmd))])


def out_of_date(target: Path, sources, stamp: Path, wanted: str) -> bool:
    if not target.exists() or target.stat().st_mtime < _newest(sources):
        return True
    return not stamp.exists() or stamp.read_text() != wanted


def _build_torch_library(source: str, target: str, libs, force: bool) -> Path:
    import torch
    from torch.utils.cpp_extension import include_paths

    LIB.mkdir(exist_ok=True)
    OBJ.mkdir(exist_ok=True)
    src = CSRC / source
    so = LIB / target
    torch_lib = Path(torch.__file__).parent / "lib"
    incs = [f"-I{p}" for p in include_paths("cuda")] + [f"-I{INCLUDE}", f"-I{sysconfig.get_paths()['include']}"]
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    cmd = [
        "g++", "-std=c++17", "-O2", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={abi}", *incs, str(src),
        "-o", str(so),
        f"-L{LIB}", f"-L{torch_lib}", *libs,
        "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_lib}", f"-Wl,-rpath,{CUDA_HOME / 'lib64'}",
    ]
    stamp, wanted = OBJ / (target + ".stamp"), made_for(cmd)
    if force or out_of_date(so, [src, *INCLUDE.glob("*.h")], stamp, wanted):
        _run(cmd)
        stamp.write_text(wanted)
    return so


def build_torch_binding(force: bool = False) -> Path:
    assert (LIB / "libdtq_b200.so").exists(), "build the kernel library first"
    so = _build_torch_library("register_ops.cpp", "libdriss_torch.so",
                              ["-ldtq_b200", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-L{CUDA_HOME / 'lib64'}", "-lcudart"],
                              force)
    (LIB / "_direct.so").unlink(missing_ok=True)  # its name once, which any Python would load
    _build_torch_library("direct_calls.cpp", "_direct" + importlib.machinery.EXTENSION_SUFFIXES[0],
                         ["-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10"], force)
    return so


def build_all(force: bool = False) -> None:
    build_kernels(force)
    build_torch_binding(force)


if __name__ == "__main__":
    build_all(force="--force" in sys.argv)
    print("built:", *(p.name for p in sorted(LIB.glob("*.so"))))
