"""In-tree build of the native libraries (nvcc for the sm_100a kernels, g++ for the host-only accountant).

The shared objects are written next to the Python package (``opake_b200/_C``) so that they travel with a
snapshot of the source tree; nothing is installed into site-packages and no JIT cache is used.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "csrc"
OUT = Path(__file__).resolve().parent / "_C"

KERNEL_LIB = OUT / "libopake_kernels.so"
# same sources with -DOPK_DEBUG_BOUNDS: data-dependent indices are checked, a bad one is recorded and its access skipped
KERNEL_LIB_DEBUG = OUT / "libopake_kernels_debug.so"
ACCOUNTING_LIB = OUT / ("_opake_accounting" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-DOPK_SM100A",
]


def _newer(target: Path, sources: list[Path]) -> bool:
    if not target.exists():
        return False
    t = target.stat().st_mtime
    return all(s.stat().st_mtime <= t for s in sources)


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; cannot build the sm_100a kernels")
    return exe


def build_kernels(force: bool = False, verbose: bool = False, debug_bounds: bool = False) -> Path:
    """Compile every ``csrc/kernels/*.cu`` into one shared library for sm_100a (``debug_bounds``: the checked variant)."""
    src_dir = CSRC / "kernels"
    target = KERNEL_LIB_DEBUG if debug_bounds else KERNEL_LIB
    extra = ["-DOPK_DEBUG_BOUNDS"] if debug_bounds else []
    suffix = ".dbg.o" if debug_bounds else ".o"
    cu = sorted(src_dir.glob("*.cu"))
    deps = cu + sorted(src_dir.glob("*.cuh")) + sorted(src_dir.glob("*.h"))
    if not force and _newer(target, deps):
        return target
    OUT.mkdir(parents=True, exist_ok=True)
    objs = []
    jobs = []
    for f in cu:
        obj = OUT / (f.stem + suffix)
        if not force and _newer(obj, [f] + [d for d in deps if d.suffix in (".cuh", ".h")]):
            objs.append(obj)
            continue
        cmd = [_nvcc(), *NVCC_FLAGS, *extra, "-c", str(f), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        jobs.append((f, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for f, proc in jobs:
        out, _ = proc.communicate()
        if verbose and out:
            print(out)
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed for {f.name}:\n{out}")
    link = [_nvcc(), "-shared", "-o", str(target), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
            "-Xcompiler", "-fPIC"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    return target


def build_accounting(force: bool = False) -> Path:
    """Compile the torch-free C++ privacy accountant (pybind11 module)."""
    src_dir = CSRC / "accounting"
    cpp = sorted(src_dir.glob("*.cpp"))
    if not cpp:
        return ACCOUNTING_LIB
    deps = cpp + sorted(src_dir.glob("*.hpp"))
    if not force and _newer(ACCOUNTING_LIB, deps):
        return ACCOUNTING_LIB
    import pybind11

    OUT.mkdir(parents=True, exist_ok=True)
    cmd = [
        os.environ.get("CXX", "g++"), "-O3", "-std=c++17", "-shared", "-fPIC", "-pthread", "-fvisibility=hidden",
        f"-I{pybind11.get_include()}", f"-I{sysconfig.get_paths()['include']}", f"-I{src_dir}",
        *map(str, cpp), "-o", str(ACCOUNTING_LIB),
    ]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"accountant build failed:\n{r.stdout}")
    return ACCOUNTING_LIB


def nodes_lib() -> Path:
    """The autograd nodes of the operators of ops/nodes.py: the one library here that is compiled against torch's headers. Its name tells
    the torch and the source that it was built from, so one of another torch or of an older source is never taken for it."""
    import hashlib

    import torch

    source = hashlib.sha256((CSRC / "host" / "nodes.cpp").read_bytes()).hexdigest()[:12]
    torch_version = "".join(c if c.isalnum() or c == "." else "_" for c in torch.__version__)
    return OUT / f"_opake_nodes-torch{torch_version}-{source}{sysconfig.get_config_var('EXT_SUFFIX') or '.so'}"


def build_nodes(force: bool = False) -> Path:
    """Compile the autograd nodes of the dispatcher operators (host code on torch's C++ API). The library appears whole or not at all:
    several ranks may look for it, and build it, at once."""
    src, target = CSRC / "host" / "nodes.cpp", nodes_lib()
    if not force and target.exists():
        return target
    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    part = target.with_name(f"{target.name}.{os.getpid()}.part")

    OUT.mkdir(parents=True, exist_ok=True)
    cmd = [
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-DTORCH_EXTENSION_NAME=_opake_nodes",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{p}" for p in include_paths()),
        f"-I{sysconfig.get_paths()['include']}", str(src), "-o", str(part), *(f"-L{p}" for p in library_paths()),
        "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10",
    ]
    try:
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"build of the autograd nodes failed:\n{r.stdout}")
        os.replace(part, target)
    except OSError as exc:
        raise RuntimeError(f"build of the autograd nodes failed: no C++ compiler ({exc})") from exc
    finally:
        part.unlink(missing_ok=True)
    return target


def build_all(force: bool = False, verbose: bool = False) -> None:
    build_kernels(force=force, verbose=verbose)
    build_kernels(force=force, debug_bounds=True)
    build_nodes(force=force)
    build_accounting(force=force)


if __name__ == "__main__":
    build_all(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print("built:", KERNEL_LIB, ACCOUNTING_LIB if ACCOUNTING_LIB.exists() else "(no accountant sources yet)")
