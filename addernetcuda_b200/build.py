"""Builds libadder_b200.so in-tree with nvcc for sm_100a (no libtorch, no Python headers), and the extension _adder_host.so
on top of it with the C++ compiler (libtorch and Python headers: the host path of the eager layer calls).  Where torch or
a header is missing only the extension is, with a warning: layers then go through the Python layer.

    python -m addernetcuda_b200.build [--force] [--verbose]

The library is placed next to this file so that it travels with the source tree.  It links the
CUDA runtime statically and exports only the extern "C" entry points of include/adder_b200.h.
A second library, libadder_b200_tuning.so, is linked from the same objects with the C-ABI layer compiled
with -DADDER_B200_TUNING: it adds the tile-override setters that parameter sweeps and some tests use and
that the product library deliberately lacks.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import warnings
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIB = PKG / "libadder_b200.so"
HOST_LIB = PKG / "_adder_host.so"              # csrc/host.cpp
TUNING_LIB = PKG / "libadder_b200_tuning.so"   # same objects, api.cu compiled with -DADDER_B200_TUNING
SOURCES = ["api.cu", "adder_fwd.cu", "adder_fwd_gather.cu", "adder_bwd_input.cu", "adder_gx_gather.cu", "adder_bwd_weight.cu", "adder_gw_mma.cu", "adder_bwd_weight_pipe.cu", "adder_bwd_weight_tma.cu", "tma_host.cu", "adder_bwd_weight_1x1.cu", "adder_pointwise.cu", "static_scratch.cu", "batchnorm.cu", "peer_allreduce.cu"]
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def find_nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found (set NVCC or add it to PATH)")
    return cand


def _older(libs, deps) -> bool:
    """One of the built files is missing or older than a source."""
    if not all(p.exists() for p in libs):
        return True
    t = min(p.stat().st_mtime for p in libs)
    return any(d.stat().st_mtime > t for d in deps)


def _headers() -> list:
    return list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))


def _stale() -> bool:
    return _older((LIB, TUNING_LIB), list(CSRC.glob("*.cu")) + _headers())


def _host_mark() -> str:
    """Stands in the extension: the torch that it was linked with, whose C++ interface differs from version to version."""
    import torch
    return f"adder_host for torch {torch.__version__}"


def host_usable() -> bool:
    """The extension is there and was linked with the torch that is installed."""
    return HOST_LIB.exists() and _host_mark().encode() in HOST_LIB.read_bytes()


def _host_stale() -> bool:
    return not host_usable() or _older((HOST_LIB,), [CSRC / "host.cpp", *INCLUDE.glob("*.h")])


def _shared_libstdcxx() -> list:
    """The C++ runtime that torch runs on, named before the compiler's own.  A compiler that has only a static one would put a
    second copy into the extension, and streams of one copy cannot format with the locale of the other: an error
    message with a number in it ended the process."""
    import torch  # noqa: F401  (loads it)
    try:
        maps = Path("/proc/self/maps").read_text()
    except OSError:
        return []
    return sorted({line.split()[-1] for line in maps.splitlines() if "/libstdc++.so" in line})[:1]


def _host_command(out: Path) -> list:
    """Compile and link csrc/host.cpp against the installed torch."""
    import sysconfig
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(find_nvcc()).resolve().parent.parent
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include", INCLUDE,
           Path(sysconfig.get_paths()["include"])]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wno-interference-size",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DADDER_HOST_MARK="{_host_mark()}"', *(f"-I{p}" for p in inc), str(CSRC / "host.cpp"),
            "-o", str(out), *_shared_libstdcxx(), f"-L{root / 'lib'}", "-lc10", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda",
            f"-L{cuda / 'lib64'}", "-lcudart"]


def _temporary(lib: Path) -> Path:
    """Where a library is linked before it takes its name: another process never loads half a file."""
    return lib.with_name(f".{os.getpid()}.{lib.name}")


def _start_host():
    """(process, its output file) of the extension's compilation, or None with a warning where it cannot be started."""
    tmp = _temporary(HOST_LIB)
    try:
        return subprocess.Popen(_host_command(tmp), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), tmp
    except (ImportError, OSError, RuntimeError) as e:
        warnings.warn(f"{HOST_LIB.name} is not built ({e}): eager layer calls go through the Python layer")
        return None


def _finish_host(started) -> bool:
    if started is None:
        return False
    proc, tmp = started
    out, _ = proc.communicate()
    if proc.returncode != 0:
        tmp.unlink(missing_ok=True)
        warnings.warn(f"{HOST_LIB.name} is not built: eager layer calls go through the Python layer\n{out[-2000:]}")
        return False
    os.replace(tmp, HOST_LIB)
    return True


def build_host() -> bool:
    """Build the extension alone."""
    return _finish_host(_start_host())


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile what is out of date (every translation unit in parallel) and link the libraries."""
    try:
        host_stale = force or _host_stale()
    except ImportError:
        host_stale = True
    host = _start_host() if host_stale else None
    if force or _stale():
        _build_libraries(verbose)
    if host_stale:
        _finish_host(host)
    return LIB


def _build_libraries(verbose: bool) -> None:
    nvcc = find_nvcc()
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    common = [nvcc, "-O3", "-std=c++17", "-lineinfo", *ARCH_FLAGS, "-Xcompiler", "-fPIC,-fvisibility=hidden",
              "-I", str(INCLUDE), "-I", str(CSRC)]
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    objs = []
    for src in SOURCES:
        obj = objdir / (src[:-3] + ".o")
        objs.append(str(obj))
        procs.append((src, subprocess.Popen(common + ["-c", str(CSRC / src), "-o", str(obj)],
                                            stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    # the tuning variant of the C-ABI layer: the only translation unit that differs between the two libraries
    api_tuning = objdir / "api_tuning.o"
    procs.append(("api.cu (tuning)", subprocess.Popen(common + ["-DADDER_B200_TUNING", "-c", str(CSRC / "api.cu"), "-o", str(api_tuning)],
                                                      stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"--- nvcc failed on {src} ---\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src} ---\n{out}\n")
    if failed:
        raise RuntimeError("nvcc compilation failed")
    tuning_objs = [str(api_tuning) if o.endswith("/api.o") else o for o in objs]
    for lib, members in ((LIB, objs), (TUNING_LIB, tuning_objs)):
        tmp = _temporary(lib)
        subprocess.run([nvcc, "-shared", *ARCH_FLAGS, "-o", str(tmp), *members, "-cudart", "static"], check=True)
        os.replace(tmp, lib)


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true", help="print ptxas register/shared-memory usage")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
