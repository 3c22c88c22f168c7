"""Build recipe of the CUDA library: nvcc, sm_100a only, one shared object next to the package; and of the Python extension beside it
(csrc/host.cpp against torch's C++ interface: the host side of small calls).

    python sm120-fp4_b200/build.py [--verbose]

The library exports the C ABI declared in include/b200moe.h and nothing else that a caller needs.
"""
from __future__ import annotations

import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libb200moe.so"
SOURCES = ["capi.cu", "layout_quant.cu", "route.cu", "decode.cu", "decode_tc.cu", "prefill.cu", "ep.cu", "umma_probe.cu", "stream_probe.cu"]
FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-Xcompiler", "-fPIC",
         "--expt-relaxed-constexpr", "-Xptxas", "-v"]


DIAG = "--diag" in sys.argv or os.environ.get("B200MOE_DIAG") == "1"
if DIAG:
    # diagnostic build (libb200moe_diag.so, loaded with B200MOE_LIB=<path>): per-worker cycle counters in the decode kernel and
    # the entry points of include/b200moe_diag.h. Not the library that ships.
    FLAGS += ["-DB200_TIMERS", "-DB200_DIAGNOSTICS"]
    LIB = PKG / "libb200moe_diag.so"


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def sources() -> list[Path]:
    return [CSRC / s for s in SOURCES if (CSRC / s).exists()] + sorted(p for p in CSRC.glob("*.cu") if p.name not in SOURCES)


# The extension inlines torch's C++ interface and knows the interpreter's: its name carries the interpreter's ABI, its code the version of torch (which
# _lib.host() compares), and it is built again whenever the command would be another one.
HOST_SRC, HOST = CSRC / "host.cpp", PKG / f"_host{sysconfig.get_config_var('EXT_SUFFIX')}"
HOST_BUILT_BY = PKG / "build" / "host.command"


def host_command(out: Path) -> list[str]:
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc()).resolve().parent.parent
    return [os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
            f'-DB200_TORCH_VERSION="{torch.__version__}"',
            f"-I{root / 'include'}", f"-I{cuda / 'include'}", f"-I{sysconfig.get_paths()['include']}", str(HOST_SRC), "-o", str(out),
            f"-L{root / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def host_record() -> str:
    return "\n".join(host_command(HOST)).replace(str(PKG), ".")      # (the folder may be moved)


def host_stale() -> bool:
    if not HOST.exists() or HOST.stat().st_mtime <= HOST_SRC.stat().st_mtime or not HOST_BUILT_BY.exists():
        return True
    return HOST_BUILT_BY.read_text() != host_record()


def build_host(verbose: bool = False, force: bool = False) -> Path:
    if force or host_stale():
        new = HOST.with_name(HOST.name + f".{os.getpid()}")      # put in place whole: another process may be loading the old one
        r = subprocess.run(host_command(new), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if verbose or r.returncode:
            print(f"--- {HOST_SRC.name}\n{r.stdout}", file=sys.stderr)
        if r.returncode:
            raise RuntimeError(f"{HOST_SRC.name} failed")
        HOST_BUILT_BY.parent.mkdir(exist_ok=True)
        HOST_BUILT_BY.unlink(missing_ok=True)
        os.replace(new, HOST)
        HOST_BUILT_BY.write_text(host_record())
    return HOST


def stale() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    return any(p.stat().st_mtime > t for p in list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")))


def build(verbose: bool = False, force: bool = False) -> Path:
    """The library, and where torch is installed the host extension."""
    build_library(verbose, force)
    if importlib.util.find_spec("torch"):
        build_host(verbose, force)
    return LIB


def build_library(verbose: bool = False, force: bool = False) -> Path:
    if not force and not stale():
        return LIB
    objs = []
    out_dir = PKG / ("build_diag" if DIAG else "build")
    out_dir.mkdir(exist_ok=True)
    procs = []
    for src in sources():
        obj = out_dir / (src.stem + ".o")
        objs.append(obj)
        if obj.exists() and obj.stat().st_mtime > max(p.stat().st_mtime for p in [src] + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))) and not force:
            continue
        cmd = [nvcc(), *FLAGS, "-c", str(src), "-o", str(obj)]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, pr in procs:
        log, _ = pr.communicate()
        if verbose or pr.returncode:
            print(f"--- {src.name}\n{log}", file=sys.stderr)
        if pr.returncode:
            raise RuntimeError(f"nvcc failed on {src.name}")
    cmd = [nvcc(), "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode:
        print(r.stdout, file=sys.stderr)
        raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
