"""Ahead-of-time build of libreskv_b200.so for sm_100a.

    python -m reskv_b200.csrc.build [--force] [--verbose]

One ``nvcc`` invocation per ``.cu`` file (object files under ``build/``), then a
shared link next to this file.  The library does not link against torch or Python: it
is plain CUDA runtime code behind the C ABI of ``include/reskv_b200.h``.  Next to it
``_host.so`` is built from ``host.cpp``: the CPython module that takes torch tensors
and calls that ABI.  nvcc cross-compiles, so no GPU is needed to build.  ``RESKV_NVCC_FLAGS`` (environment) adds compiler flags; use it
together with ``--force``.
"""

from __future__ import annotations

import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
LIB = HERE / "libreskv_b200.so"
HOST = HERE / "_host.so"
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("CUDA_HOME", "") + "/bin/nvcc", "/usr/local/cuda/bin/nvcc", shutil.which("nvcc") or ""):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: set CUDA_HOME")


def sources() -> list[Path]:
    return sorted(HERE.glob("*.cu"))


def _stale(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    objdir = HERE / "build"
    objdir.mkdir(exist_ok=True)
    headers = sorted(HERE.glob("*.cuh")) + [HERE.parent.parent / "include" / "reskv_b200.h"]
    extra = os.environ.get("RESKV_NVCC_FLAGS", "").split()
    jobs = []
    for src in sources():
        obj = objdir / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            cmd = [nvcc, *ARCH_FLAGS, *COMMON, *extra, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)
    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError(f"nvcc failed on {cmd[-3]}")
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        list(pool.map(run, jobs))
    objs = [objdir / (s.stem + ".o") for s in sources()]
    if force or jobs or _stale(LIB, objs):
        run([nvcc, *ARCH_FLAGS, "-shared", "-Xlinker=-soname=libreskv_b200.so", "-o", str(LIB), *map(str, objs), "-lcudart"])
    command, record = _host_command(nvcc), objdir / "_host.txt"
    if force or _host_stale([HERE / "host.cpp", headers[-1]], command, record):
        run(command)
        record.write_text(_host_record(command))
    return LIB


def _host_record(command: list[str]) -> str:
    """What ``_host.so`` depends on besides its sources: the command line (interpreter and torch by path) and torch's
    version, whose internal headers it compiles against."""
    version = _torch_dir() / "version.py"
    return " ".join(command) + "\n" + (version.read_text() if version.exists() else "")


def _host_stale(deps: list[Path], command: list[str], record: Path) -> bool:
    return _stale(HOST, deps) or not record.exists() or record.read_text() != _host_record(command)


def _torch_dir() -> Path:
    """torch is only located, not imported: its headers and libraries sit in the package, and at run time they are already
    loaded."""
    return Path(importlib.util.find_spec("torch").origin).parent


def _host_command(nvcc: str) -> list[str]:
    """g++ for the tensor-facing module."""
    torch = _torch_dir()
    cuda = Path(nvcc).resolve().parent.parent
    includes = [torch / "include", torch / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"]]
    libs = ["c10", "c10_cuda", "torch_cpu", "torch_cuda", "torch_python"]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", *(f"-I{d}" for d in includes), str(HERE / "host.cpp"), "-o",
            str(HOST), f"-L{torch / 'lib'}", *(f"-l{lib}" for lib in libs), f"-L{cuda / 'lib64'}", "-lcudart", f"-L{HERE}",
            "-lreskv_b200", "-Wl,-rpath,$ORIGIN"]


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
