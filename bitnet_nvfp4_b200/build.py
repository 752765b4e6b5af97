"""In-tree build of libbnf4.so (sm_100a only) with nvcc, and of the host extension _host (the Python-side call path over it) with g++.

    python -m bitnet_nvfp4_b200.build            # incremental
    python -m bitnet_nvfp4_b200.build --force    # rebuild everything

nvcc cross-compiles without a GPU. The shared object is placed next to this file so that it travels
with the source tree; it is not installed into site-packages.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libbnf4.so"
HOST = PKG / f"_host{sysconfig.get_config_var('EXT_SUFFIX')}"  # (another interpreter does not take it for its own)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    f"-I{ROOT / 'include'}", f"-I{CSRC}",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libbnf4 has no CPU build")
    return exe


def _host_compiler_args() -> list[str]:
    # some images export CXX to a wrapper that lacks its runtime specs; prefer the system compiler
    return ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []


def _newer(src: Path, dst: Path, deps: list[Path]) -> bool:
    if not dst.exists():
        return True
    t = dst.stat().st_mtime
    return any(p.stat().st_mtime > t for p in [src, *deps])


def build(force: bool = False, verbose: bool = False) -> Path:
    OBJ.mkdir(exist_ok=True)
    nvcc = _nvcc()
    headers = sorted(CSRC.glob("*.h")) + sorted(CSRC.glob("*.cuh")) + sorted((ROOT / "include").glob("*.h"))
    sources = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp"))
    jobs = []
    objs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        objs.append(obj)
        if force or _newer(src, obj, headers):
            cmd = [nvcc, *_host_compiler_args(), *NVCC_FLAGS, "-x", "cu", "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append((src, cmd))

    def run(job):
        src, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(f"--- {src.name}\n{r.stdout}{r.stderr}\n")
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src.name}")

    if force or jobs or not LIB.exists():
        cmd = [nvcc, *_host_compiler_args(), "-shared", "-o", str(LIB), *map(str, objs)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of libbnf4.so failed")
    build_host(force)
    return LIB


def build_host(force: bool = False) -> Path:
    """The host extension: a CPython extension on torch's C++ tensors, linked to the libbnf4.so beside it. It holds for one torch and one
    interpreter only, so both are noted with the command that built it, and it is built again when any of them changes."""
    src = CSRC / "binding" / "host_calls.cpp"
    import torch
    from torch.utils import cpp_extension

    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    cuda = Path(_nvcc()).resolve().parent.parent / "include"
    torch_lib = Path(torch.__file__).resolve().parent / "lib"
    cmd = [gxx, "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-isystem{d}" for d in [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], cuda]], f"-I{ROOT / 'include'}", str(src),
           "-o", str(HOST), f"-L{PKG}", "-l:libbnf4.so", "-Wl,-rpath,$ORIGIN", f"-L{torch_lib}", "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10",
           "-lc10_cuda"]
    stamp, built = OBJ / "_host.stamp", "\n".join([torch.__version__, sys.version, *cmd]).replace(str(ROOT), "")
    if not force and not _newer(src, HOST, [ROOT / "include" / "bnf4.h"]) and stamp.exists() and stamp.read_text() == built:
        return HOST
    (PKG / "_host.so").unlink(missing_ok=True)  # the name it had before
    stamp.unlink(missing_ok=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"build of {HOST.name} failed")
    OBJ.mkdir(exist_ok=True)
    stamp.write_text(built)
    return HOST


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
