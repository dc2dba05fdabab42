"""Builds libllmmm_b200.so (the C-ABI library) in-tree with nvcc for sm_100a and, where torch is installed, _binding.so
(its calls for Python).

Usage: python -m llmmm_b200.build [--force] [--verbose] [--profile]

--profile builds a second library, libllmmm_b200_profile.so, from the same sources with -DLLMMM_PROFILE: the
kernels then record %globaltimer / clock64 stamps at their hand-off points and the library exports
llmmm_profile_dump_* functions that print them (load that library instead of the regular one, run the shape,
call the dump function).  The regular library contains none of this.
"""
from __future__ import annotations

import concurrent.futures as cf
import importlib.util
import os
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libllmmm_b200.so"
BINDING = PKG / "_binding.so"
PROFILE_LIB = PKG / "libllmmm_b200_profile.so"
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


# Kernels whose hot loop has no register to spare: the build fails if ptxas reports spills for them.
NO_SPILL = ("fp8_blockwise_gemm",)
# (no instantiation is exempt)
SPILL_TOLERATED: tuple[str, ...] = ()


def spilling_kernels(ptxas_log: str, patterns: tuple[str, ...]) -> list[str]:
    """Entry functions matching `patterns` for which `-Xptxas -v` reports spill stores or loads."""
    bad, current = [], None
    for line in ptxas_log.splitlines():
        if "Compiling entry function" in line or "Function properties for" in line:
            current = line.split("'")[1] if "'" in line else line.rsplit(" ", 1)[-1]
        elif "bytes spill stores" in line and current and any(p in current for p in patterns):
            if "0 bytes spill stores, 0 bytes spill loads" not in line and not any(t in current for t in SPILL_TOLERATED):
                bad.append(current)
    return sorted(set(bad))


def _newer(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return False
    t = target.stat().st_mtime
    return all(d.stat().st_mtime <= t for d in deps)


def build_library(force: bool = False, verbose: bool = False, profile: bool = False) -> Path:
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.h")) + sorted(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "llmmm_c.h"]
    obj_dir = OBJ / "profile" if profile else OBJ
    lib = PROFILE_LIB if profile else LIB
    flags = FLAGS + (["-DLLMMM_PROFILE"] if profile else [])
    obj_dir.mkdir(parents=True, exist_ok=True)

    def compile_one(src: Path) -> tuple[Path, str]:
        obj = obj_dir / (src.stem + ".o")
        if not force and _newer(obj, [src] + headers):
            return obj, ""
        cmd = [NVCC, *flags, "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        spilled = [] if profile else spilling_kernels(r.stderr, NO_SPILL)
        if spilled:
            obj.unlink(missing_ok=True)
            raise RuntimeError(f"{src.name}: ptxas spilled registers in {spilled}; these kernels lose a third of their "
                               "speed to a few spilled bytes (change the setmaxnreg split until -Xptxas -v shows 0)")
        return obj, r.stderr

    with cf.ThreadPoolExecutor(max_workers=min(8, len(sources))) as ex:
        results = list(ex.map(compile_one, sources))
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            if log:
                sys.stderr.write(log)
    if force or not _newer(lib, objs):
        cmd = [NVCC, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(lib), *map(str, objs), "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if not profile and importlib.util.find_spec("torch") is not None:  # (a C or C++ host needs the library alone)
        build_binding(force)
    return lib


def binding_built_for() -> str:
    """What _binding.so is built against; capi.py does not use one that says otherwise."""
    import torch
    return f"torch {torch.__version__}, python {sys.version_info.major}.{sys.version_info.minor}"


def build_binding(force: bool = False) -> Path:
    """_binding.so: the native form of the calls in capi.py, against the headers of the torch it will run with."""
    src = CSRC / "binding.cpp"
    built_for = binding_built_for()
    if not force and _newer(BINDING, [src, PKG.parent / "include" / "llmmm_c.h"]) and built_for.encode() + b"\0" in BINDING.read_bytes():
        return BINDING
    import torch
    root = Path(torch.__file__).resolve().parent
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f'-DLLMMM_BUILT_FOR="{built_for}"', f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{root / 'include'}", f"-I{root / 'include/torch/csrc/api/include'}", f"-I{Path(NVCC).resolve().parent.parent / 'include'}",
           f"-I{sysconfig.get_paths()['include']}", str(src), "-o", str(BINDING), f"-L{root / 'lib'}", "-ltorch_python", "-ltorch",
           "-ltorch_cpu", "-lc10", "-lc10_cuda", f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{src.name}: {r.stdout}\n{r.stderr}")
    return BINDING


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="--verbose" in sys.argv, profile="--profile" in sys.argv))
