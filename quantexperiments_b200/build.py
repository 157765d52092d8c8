"""In-tree build of libcbl.so (hand-written CUDA for sm_100a behind a C ABI) and of _cblhost.so (the native call path
between torch and it, csrc/host.cpp).

    python -m quantexperiments_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU; the shared object is written next to this file so that it
travels with the source tree. Nothing is cached outside the tree."""

from __future__ import annotations

import re
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libcbl.so"
HOST = PKG / "_cblhost.so"
STAMP = PKG / "_cblhost.stamp"           # the torch that the host extension was built against
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "cbl.h"]
    return any(p.stat().st_mtime > t for p in deps)


def build_host(force: bool = False, verbose: bool = False) -> Path:
    """Compile csrc/host.cpp against the installed torch; returns the extension module's path."""
    import sysconfig
    import torch
    src, deps = CSRC / "host.cpp", [CSRC / "host.cpp", PKG.parent / "include" / "cbl.h"]
    if not force and HOST.exists() and STAMP.exists() and STAMP.read_text() == torch.__version__ and all(p.stat().st_mtime <= HOST.stat().st_mtime for p in deps):
        return HOST
    root = Path(torch.__file__).resolve().parent
    cuda = Path("/usr/local/cuda")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DCBL_TORCH="{torch.__version__}"', "-isystem", str(root / "include"),
           "-isystem", str(root / "include" / "torch" / "csrc" / "api" / "include"), "-isystem", str(cuda / "include"),
           "-isystem", sysconfig.get_paths()["include"], str(src), "-o", str(HOST), f"-L{PKG}", "-l:libcbl.so", "-Wl,-rpath,$ORIGIN", f"-L{root / 'lib'}",
           "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", f"-L{cuda / 'lib64'}", "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError(f"g++ failed ({r.returncode}): {' '.join(cmd)}")
    STAMP.write_text(torch.__version__)
    return HOST


def check_registers(log: str) -> None:
    """The one-token kernel shares the registers of its launch out among its roles (setmaxnreg): it must have been compiled to the number
    that its source states (in eights), or its warps would wait for registers that do not exist.  `log`: ptxas -v."""
    want = int(re.search(r"L8_REGS_LAUNCH = (\d+)", (CSRC / "cbl_gemv1.cu").read_text()).group(1))
    m = re.search(r"Compiling entry function '[^']*k_gemv_l8[^']*'.*?Used (\d+) registers", log, re.S)
    if m is None or -(-int(m.group(1)) // 8) * 8 != want:
        raise RuntimeError(f"k_gemv_l8 uses {m and m.group(1)} registers, its source counts on {want}")


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every kernel for sm_100a into libcbl.so, and the host extension; returns the library's path."""
    if not force and not _stale():
        build_host(False, verbose)
        return LIB
    cmd = ["nvcc", *ARCH, "-O3", "-std=c++17", "-lineinfo", "-shared", "-Xcompiler", "-fPIC", "--threads", "0",
           "-I", str(PKG.parent / "include"), "-Xptxas", "-v",
           *[str(s) for s in sources()], "-o", str(LIB)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError(f"nvcc failed ({r.returncode}): {' '.join(cmd)}\n{r.stderr if not verbose else ''}")
    try:
        check_registers(r.stderr + r.stdout)
    except RuntimeError:
        LIB.unlink()
        raise
    build_host(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
