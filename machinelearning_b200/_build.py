"""Builds ``libnlfa.so`` (the C-ABI attention library) in-tree with nvcc, and ``_host.so`` (its
torch-facing call path, ``csrc/host.cpp``) with g++ against torch's headers.

    python -m machinelearning_b200._build [--force] [--verbose]

sm_100a only: ``-gencode arch=compute_100a,code=sm_100a``.  Same flag policy as
the reference's JIT build (``nanolab/flash_cuda.py:116-124``): ``-O3 -lineinfo``
and no ``--use_fast_math``.  nvcc cross-compiles without a GPU, so this also
runs on a CPU-only machine.
"""
from __future__ import annotations

import concurrent.futures
import os
import pathlib
import shutil
import subprocess
import sys

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "_obj"
LIB = PKG / "libnlfa.so"
HOST = PKG / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found")
    return exe


def sources() -> list[pathlib.Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale(target: pathlib.Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    """Compile every ``csrc/*.cu`` and link ``libnlfa.so``; returns its path."""
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    headers = list(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "nlfa.h"]
    jobs = []
    for src in sources():
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{r.stdout}\n{r.stderr}")
        (OBJ / (src.stem + ".ptxas.txt")).write_text(r.stderr)
        return src.name, r.stderr

    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for name, log in ex.map(compile_one, jobs):
                if verbose:
                    print(f"== {name}\n{log}")
    objs = [OBJ / (s.stem + ".o") for s in sources()]
    if force or jobs or _stale(LIB, objs):
        def link(out):
            cmd = [nvcc, "-shared", "-o", str(out), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
        _into_place(LIB, link)
    build_host(force)
    return LIB


def _into_place(target: pathlib.Path, make) -> None:
    """``make(path)`` under a name of this process's own, then one rename: another process that starts at the same time
    loads the whole file or none."""
    part = target.with_name(f"{target.name}.{os.getpid()}.part")
    try:
        make(part)
        os.replace(part, target)
    finally:
        part.unlink(missing_ok=True)


def _host_stamp() -> str:
    """What ``_host.so`` was compiled against; ``host.cpp`` carries it as a string."""
    import torch
    return f"nlfa host module for torch {torch.__version__}, python {sys.version_info[0]}.{sys.version_info[1]};"


def host_fits() -> bool:
    """Whether ``_host.so`` is there and was compiled against this torch and this Python (it uses torch's C++ interface,
    which no other build shares)."""
    return HOST.exists() and _host_stamp().encode() in HOST.read_bytes()


def build_host(force: bool = False) -> pathlib.Path:
    """Compile ``csrc/host.cpp``; it finds ``libnlfa.so`` next to itself."""
    src = CSRC / "host.cpp"
    if not force and not _stale(HOST, [src, PKG.parent / "include" / "nlfa.h"]) and host_fits():
        return HOST
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    cuda = pathlib.Path(_nvcc()).resolve().parent.parent
    include = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda / "include")]
    libs = pathlib.Path(torch.__file__).parent / "lib"

    def compile_to(out):
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-w",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f'-DNLFA_HOST_STAMP="{_host_stamp()}"',
               *(f"-isystem{p}" for p in include), str(src), "-o", str(out),
               f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
               f"-L{PKG}", "-l:libnlfa.so", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"g++ failed on host.cpp:\n{r.stdout}\n{r.stderr}")
    _into_place(HOST, compile_to)
    return HOST


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
