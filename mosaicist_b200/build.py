"""Builds libmosaicist_sm100a.so in-tree with nvcc.

    python -m mosaicist_b200.build [--force] [--debug]

`--debug` also builds libmosaicist_sm100a_debug.so with -DMSC_DEBUG: the same kernels plus
per-CTA clock stamps (clock64 and the global nanosecond timer) and pipeline-stage skip flags,
used by `python -m mosaicist_b200.profile_stage --in-kernel-clock`; nothing else loads it.

The library is compiled for sm_100a only.  nvcc cross-compiles without a GPU, so this
runs on a CPU-only machine; the resulting .so is what the GPU machine loads.
"""

from __future__ import annotations

import contextlib
import fcntl
import hashlib
import os
import pathlib
import re
import shutil
import subprocess
import sys

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libmosaicist_sm100a.so"
HEADER = PKG.parent / "include" / "mosaicist_sm100a.h"
PTXAS_LOG = PKG / "libmosaicist_sm100a.ptxas.log"
DEBUG_LIB = PKG / "libmosaicist_sm100a_debug.so"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo"]


def sources() -> list[pathlib.Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale() -> bool:
    if not LIB.exists():
        return True
    built = LIB.stat().st_mtime
    deps = list(CSRC.glob("*")) + [HEADER]
    return any(p.stat().st_mtime > built for p in deps)


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    """Compile every .cu under csrc/ into one shared library (and the native host path beside
    it); returns its path."""
    build_host_ops(force)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not force and not _stale():
        return LIB
    if not pathlib.Path(nvcc).exists():
        if LIB.exists():
            return LIB  # prebuilt library on a machine without the toolkit
        raise RuntimeError("nvcc not found and no prebuilt libmosaicist_sm100a.so")
    srcs = [str(s) for s in sources()]
    cmd = [nvcc, *ARCH, *COMMON, f'-DMSC_ABI="{abi()}"', "-Xptxas", "-v", "-t", "0", "-shared", "-Xcompiler", "-fPIC",
           "-cudart", "static", "-o", str(LIB), *srcs, "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    PTXAS_LOG.write_text(res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stderr[-4000:])
    if verbose:
        print(res.stderr)
    return LIB


HOST_OPS_SRC = PKG / "host_ops" / "host_ops.cpp"
HOST_OPS = PKG / "_host_ops.so"
HOST_OPS_STAMP = PKG / "_host_ops.stamp"


def abi() -> str:
    """Digest of what the header declares, comments left out: the library and the host path were built
    for each other if theirs are equal."""
    text = re.sub(r"/\*.*?\*/|//[^\n]*", " ", HEADER.read_text(), flags=re.S)
    return hashlib.sha256(" ".join(text.split()).encode()).hexdigest()[:16]


def host_ops_stamp() -> str:
    """What an existing host path must have been built from: its source, the header, and the torch and
    Python whose C++ interfaces it is tied to."""
    import torch

    source = hashlib.sha256(HOST_OPS_SRC.read_bytes()).hexdigest()[:16]
    return f"source {source} header {abi()} torch {torch.__version__} python {sys.version_info[:2]} {sys.platform}"


def host_ops_current() -> bool:
    try:
        return HOST_OPS.exists() and HOST_OPS_STAMP.read_text() == host_ops_stamp()
    except OSError:
        return False


@contextlib.contextmanager
def _locked(path: pathlib.Path):
    """One process at a time; the others wait."""
    with open(path, "a") as f:
        fcntl.flock(f, fcntl.LOCK_EX)
        try:
            yield
        finally:
            fcntl.flock(f, fcntl.LOCK_UN)


def build_host_ops(force: bool = False) -> pathlib.Path:
    """The native host path of the operators (host_ops/host_ops.cpp), a Python extension module
    against torch's C++ interface; returns its path.  Ranks that start together build it once: they
    take turns, and the module appears in place when it is complete."""
    if not force and host_ops_current():
        return HOST_OPS
    gxx = shutil.which("g++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if gxx is None:
        raise RuntimeError("g++ not found and no _host_ops.so that fits this source, torch and Python")
    import sysconfig

    import torch

    root = pathlib.Path(torch.__file__).resolve().parent
    cuda = pathlib.Path(nvcc).resolve().parents[1]
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include",
                sysconfig.get_paths()["include"]]
    with _locked(PKG / "_host_ops.lock"):
        if not force and host_ops_current():
            return HOST_OPS
        stamp = host_ops_stamp()
        part = PKG / f"_host_ops.{os.getpid()}.part"
        cmd = [gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", f'-DMSC_ABI="{abi()}"',
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{i}" for i in includes],
               "-o", str(part), str(HOST_OPS_SRC), f"-L{root / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu",
               "-ltorch_cuda", "-lc10", "-lc10_cuda"]
        try:
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                raise RuntimeError("g++ failed on the host operators:\n" + res.stderr[-4000:])
            os.replace(part, HOST_OPS)
            part.write_text(stamp)
            os.replace(part, HOST_OPS_STAMP)
        finally:
            part.unlink(missing_ok=True)
    return HOST_OPS


CUPTI_SHIM = PKG / "cupti_shim" / "libmsc_cupti.so"


def build_cupti_shim(force: bool = False) -> pathlib.Path | None:
    """The small C++ library behind the stand-in `cupti` package (cupti_shim/): kernel activity
    records from libcupti for the reference's tracer, where cupti-python is not installed.
    Returns None (and builds nothing) where the toolkit's CUPTI headers or g++ are missing."""
    src = PKG / "cupti_shim" / "cupti_shim.cpp"
    if not force and CUPTI_SHIM.exists() and CUPTI_SHIM.stat().st_mtime >= src.stat().st_mtime:
        return CUPTI_SHIM
    gxx = shutil.which("g++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = pathlib.Path(nvcc).resolve().parents[1]
    if gxx is None or not (cuda / "include" / "cupti.h").exists():
        return CUPTI_SHIM if CUPTI_SHIM.exists() else None
    libdir = cuda / "lib64"
    cmd = [gxx, "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{cuda / 'include'}", "-o", str(CUPTI_SHIM), str(src),
           f"-L{libdir}", "-lcupti", f"-Wl,-rpath,{libdir}"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed on the CUPTI shim:\n" + res.stderr[-2000:])
    return CUPTI_SHIM


def build_debug(force: bool = False) -> pathlib.Path:
    """The -DMSC_DEBUG build (clock stamps, skip flags); returns its path."""
    deps = list(CSRC.glob("*")) + [HEADER]
    if not force and DEBUG_LIB.exists() and all(p.stat().st_mtime <= DEBUG_LIB.stat().st_mtime for p in deps):
        return DEBUG_LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cmd = [nvcc, *ARCH, *COMMON, f'-DMSC_ABI="{abi()}"', "-DMSC_DEBUG", "-shared", "-Xcompiler", "-fPIC", "-cudart", "static",
           "-o", str(DEBUG_LIB), *[str(s) for s in sources()], "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stderr[-4000:])
    return DEBUG_LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose=True)
    print("built", path)
    print("built", build_host_ops(force="--force" in sys.argv))
    print("built", build_cupti_shim(force="--force" in sys.argv))
    if "--debug" in sys.argv:
        print("built", build_debug(force="--force" in sys.argv))
