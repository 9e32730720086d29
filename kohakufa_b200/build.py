"""Builds ``libkfa.so`` (the CUDA kernels + C ABI) in-tree with nvcc for sm_100a, and ``_kfa_host.so`` (the C++
launch path of the torch ops) with the host compiler.

    python -m kohakufa_b200.build            # rebuild if a source is newer than the library
    python -m kohakufa_b200.build --force

No GPU is needed to build (nvcc cross-compiles). The library is never built implicitly at
import time on a machine without nvcc: ``kohakufa_b200._lib`` raises instead.
"""

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libkfa.so"
# The same library with every pipeline wait limited to a few hundred cycles, so that the first wait for
# a copy from global memory runs out by itself: what tests/test_abort.py loads to see the kernels'
# give-up path (status word, NaN outputs, clean teardown) run on a device without hanging anything.
LIB_SHORT_WAIT = PKG / "libkfa_shortwait.so"
SHORT_WAIT_FLAGS = ["-DKFA_WAIT_CYCLES=300ll"]
HOST = PKG / "_kfa_host.so"
HOST_SOURCES = [CSRC / "kfa_host.cpp", PKG.parent / "include" / "kfa.h"]
SOURCES = [CSRC / "kfa_api.cu"]
HEADERS = [
    CSRC / "kfa_ptx.cuh",
    CSRC / "kfa_fwd.cuh",
    CSRC / "kfa_bwd.cuh",
    CSRC / "kfa_bwd_fused.cuh",
    CSRC / "kfa_selftest.cuh",
    CSRC / "kfa_cp.cuh",
    CSRC / "kfa_mask.cuh",
    CSRC / "kfa_scores.cuh",
    PKG.parent / "include" / "kfa.h",
]
NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "-shared",
    "-Xcompiler",
    "-fPIC",
    "-Xptxas",
    "-v",
]


def nvcc_path() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found: cannot build libkfa.so")
    return found


def host_stamp() -> bytes:
    """The torch and the Python a host extension is built for: it is compiled against their C++ headers, whose inlined
    accessors fit no other. The stamp is a string in the extension."""
    import torch

    return f"_kfa_host for torch {torch.__version__} {torch.version.git_version}, {sysconfig.get_config_var('SOABI')}".encode()


def host_fits(lib: Path) -> bool:
    return host_stamp() in lib.read_bytes()


def stale(lib: Path = LIB) -> bool:
    if not lib.exists() or (lib == HOST and not host_fits(lib)):
        return True
    built = lib.stat().st_mtime
    return any(p.stat().st_mtime > built for p in (HOST_SOURCES if lib == HOST else SOURCES + HEADERS))


def _run(cmd, log: str, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    (PKG / log).write_text(" ".join(cmd) + "\n" + proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n{proc.stdout}\n{proc.stderr}")
    if verbose:
        print(proc.stderr)


def _compile(lib: Path, extra, log: str, verbose: bool) -> None:
    _run([nvcc_path(), *NVCC_FLAGS, *extra, "-o", str(lib), *map(str, SOURCES)], log, verbose)


def _compile_host() -> None:
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc_path()).resolve().parent.parent
    include = [sysconfig.get_paths()["include"], root / "include", root / "include/torch/csrc/api/include", cuda / "include"]
    abi = int(torch.compiled_with_cxx11_abi())
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-DNDEBUG", f"-D_GLIBCXX_USE_CXX11_ABI={abi}"]
    cmd.append(f'-DKFA_HOST_STAMP="{host_stamp().decode()}"')
    cmd += [f"-I{d}" for d in include] + ["-o", str(HOST), str(HOST_SOURCES[0]), f"-L{root / 'lib'}"]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    _run(cmd, "build_host.log", False)


def build(force: bool = False, verbose: bool = False, short_wait: bool = True) -> Path:
    """Compile the library, the host extension (and, with ``short_wait``, the library's short-wait test twin) if
    missing or older than the sources; returns the library's path."""
    jobs = [(LIB, [], "build.log")] + ([(LIB_SHORT_WAIT, SHORT_WAIT_FLAGS, "build_shortwait.log")] if short_wait else [])
    if force or stale(HOST):
        _compile_host()
    for lib, extra, log in jobs:
        if force or stale(lib):
            _compile(lib, extra, log, verbose and lib is LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
