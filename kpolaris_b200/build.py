"""Builds the in-tree CUDA library kpolaris_b200/lib/libkpolaris_b200.so for
sm_100a with nvcc.  Each translation unit carries its own floating-point
flags: the FP64 kernels are compiled with --fmad=false (reference rounding),
the mixed-precision kernels with FMA contraction enabled.

    python -m kpolaris_b200.build [--force] [-j N]

It also builds the command-line image tool kpolaris_b200/bin/kp_model_image
(host C++, kpolaris_b200/host/) against that library.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
INCLUDE = ROOT / "include"
BUILD = PKG / "_build"
LIB = PKG / "lib" / "libkpolaris_b200.so"
HOST = PKG / "host"
TOOL = PKG / "bin" / "kp_model_image"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC,-ffp-contract=off",
          f"-I{INCLUDE}", f"-I{CSRC}", "-Xptxas", "-warn-spills"]

FP64 = ["--fmad=false"]
MIXED = ["--fmad=true", "--use_fast_math"]


def _lanes(policy: str, scene: str, *more: str):
    return [*(FP64 if policy == "FP64" else MIXED), f"-DKP_LANES_POLICY=Policy{policy}", f"-DKP_LANES_SCENE=Scene{scene}", *more]


# translation unit, with the name of its build where it has several -> extra flags
UNITS = {
    "kp_lanes.cu fp64": _lanes("FP64", "Riaf", "-DKP_LANES_IMAGE"),
    "kp_lanes.cu grmhd": _lanes("FP64", "Grmhd"),
    "kp_lanes.cu grmhd_slow": _lanes("FP64", "GrmhdSlow"),
    "kp_lanes.cu bl": _lanes("FP64", "RiafBL"),
    "kp_lanes.cu grmhd_mixed": _lanes("Mixed", "Grmhd"),
    "kp_lanes.cu grmhd_slow_mixed": _lanes("Mixed", "GrmhdSlow"),
    "kp_lanes.cu bl_mixed": _lanes("Mixed", "RiafBL"),
    "kp_kernels_fp64.cu": FP64,
    "kp_kernels_mixed.cu": MIXED,
    "kp_kernels_grmhd.cu": FP64,
    "kp_kernels_grmhd_mixed.cu": MIXED,
    "kp_kernels_grmhd_slow.cu": FP64,
    "kp_kernels_bl.cu": FP64,
    "kp_kernels_bl_mixed.cu": MIXED,
    "kp_kernels_grmhd_slow_mixed.cu": MIXED,
    "kp_capi.cu": FP64,
    "kp_reorder.cu": FP64,
    "kp_noalloc.cu": FP64,
    "kp_server.cu": FP64,
    "kp_peak.cu": [],
    "kp_io.cu": [f"-I{HOST}"],
}


def nvcc() -> str:
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return path


def _headers():
    return (list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(HOST.glob("*.hpp")) +
            [INCLUDE / "kpolaris_b200.h"])


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(d).stat().st_mtime > t for d in deps)


def _object(unit: str) -> Path:
    return BUILD / (unit.replace(" ", ".") + ".o")


def _compile(unit: str, flags, verbose: bool) -> Path:
    src = CSRC / unit.split()[0]
    obj = _object(unit)
    cmd = [nvcc(), *ARCH, *COMMON, *flags, "-c", str(src), "-o", str(obj)]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError(f"nvcc failed for {unit}")
    return obj


def build(force: bool = False, jobs: int = 4, verbose: bool = False) -> Path:
    BUILD.mkdir(parents=True, exist_ok=True)
    LIB.parent.mkdir(parents=True, exist_ok=True)
    headers = _headers()
    todo = []
    objs = []
    for unit, flags in UNITS.items():
        src = CSRC / unit.split()[0]
        if not src.exists():
            continue
        obj = _object(unit)
        objs.append(obj)
        if force or _stale(obj, [src, *headers, Path(__file__)]):
            todo.append((unit, flags))
    if todo:
        with ThreadPoolExecutor(max_workers=max(1, jobs)) as ex:
            list(ex.map(lambda uf: _compile(uf[0], uf[1], verbose), todo))
    if force or todo or _stale(LIB, objs):
        cmd = [nvcc(), *ARCH, "-shared", "-o", str(LIB), *map(str, objs), "-lz"]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    build_tool(force=force, verbose=verbose)
    return LIB


def build_tool(force: bool = False, verbose: bool = False) -> Path:
    """The image tool: host C++ over the C ABI, found next to the library
    through its run path."""
    TOOL.parent.mkdir(parents=True, exist_ok=True)
    src = HOST / "kp_model_image.cpp"
    deps = [src, HOST / "kpolaris_image_options.hpp", HOST / "kp_image_h5.hpp", HOST / "kp_hdf5.hpp",
            INCLUDE / "kpolaris_b200.h", LIB]
    if not force and not _stale(TOOL, deps):
        return TOOL
    cxx = shutil.which("g++") or "g++"
    cmd = [cxx, "-std=c++17", "-O2", "-Wall", f"-I{INCLUDE}", f"-I{HOST}", str(src), f"-L{LIB.parent}",
           "-lkpolaris_b200", "-Wl,-rpath,$ORIGIN/../lib", "-o", str(TOOL)]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("kp_model_image build failed")
    return TOOL


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-j", "--jobs", type=int, default=os.cpu_count() or 4)
    ap.add_argument("-v", "--verbose", action="store_true")
    a = ap.parse_args(argv)
    print(build(force=a.force, jobs=a.jobs, verbose=a.verbose))


if __name__ == "__main__":
    main()
