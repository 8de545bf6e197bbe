"""Build, in-tree, libfxpr_b200.so (csrc/*.cu with nvcc, sm_100a only: the C ABI) and
libfxpr_torch.so (csrc/torch_ops.cpp with g++: the torch operators over it).

Usage: ``python build.py [--force] [--verbose]``.  Objects go to ``build/``, the
shared libraries to ``lib/`` next to this file.  A source is recompiled when it or
any header is newer than its object, the operator library also when its command line
or the installed torch is another one than it was built with (``build/torch_ops.stamp``).
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent
CSRC = ROOT / "csrc"
OBJ = ROOT / "build"
LIB = ROOT / "lib" / "libfxpr_b200.so"
TORCH_LIB = ROOT / "lib" / "libfxpr_torch.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    # no implicit fused multiply-add: the exact kernels must equal a CPU doing
    # single IEEE operations; kernels that want an FMA ask for it explicitly
    "-fmad=false",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; cannot build libfxpr_b200.so")
    return exe


def _stale(src: Path, obj: Path, headers: list[Path]) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return any(p.stat().st_mtime > t for p in [src, *headers])


def _torch_cmd(src: Path) -> list[str]:
    """g++ line of the operator library, against the torch that is installed."""
    import torch
    from torch.utils import cpp_extension as ce

    cuda = Path(_nvcc()).resolve().parent.parent
    inc = [f"-I{p}" for p in [*ce.include_paths(), cuda / "include"]]
    lib = Path(torch.__file__).resolve().parent / "lib"
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc, str(src), "-o", str(TORCH_LIB),
            f"-L{LIB.parent}", f"-L{lib}", f"-L{cuda / 'lib64'}", "-lfxpr_b200", "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-lcudart", "-Wl,-rpath,$ORIGIN"]


def _torch_stamp(cmd: list[str]) -> str:
    """What the operator library's binary interface depends on besides its sources."""
    import torch

    return "\n".join([torch.__version__, str(torch.version.git_version), *cmd]) + "\n"


def _link(nvcc: str, sources: list[Path]) -> None:
    objs = [str(OBJ / (s.stem + ".o")) for s in sources]
    cmd = [nvcc, "-shared", "-o", str(LIB), *objs, "-lcudart_static", "-lpthread", "-ldl", "-lrt",
           "-Xlinker", "-soname=libfxpr_b200.so", "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    LIB.parent.mkdir(exist_ok=True)
    headers = (sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.inl")) + sorted(CSRC.glob("*.h"))
               + sorted((ROOT.parent / "include").glob("*.h")))
    sources = sorted(CSRC.glob("*.cu"))
    jobs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        if force or _stale(src, obj, headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append((src, cmd))

    def run(job):
        src, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(f"--- {src.name}\n{r.stdout}{r.stderr}\n")
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src.name}")
    if jobs or not LIB.exists():
        _link(nvcc, sources)
    src = CSRC / "torch_ops.cpp"
    deps = [src, CSRC / "host_policy.h", *(ROOT.parent / "include").glob("*.h")]
    cmd, stamp_file = _torch_cmd(src), OBJ / "torch_ops.stamp"
    stamp = _torch_stamp(cmd)
    same = stamp_file.exists() and stamp_file.read_text() == stamp
    if force or not same or not TORCH_LIB.exists() or any(p.stat().st_mtime > TORCH_LIB.stat().st_mtime for p in deps):
        stamp_file.unlink(missing_ok=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("g++ failed on torch_ops.cpp")
        stamp_file.write_text(stamp)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
