"""Build libmixlab_b200.so in-tree with nvcc for sm_100a, and the native half of the torch front end with g++.

    python -m mixlab_b200.build [--force] [--verbose]

The library has no Python or torch dependency: it is a plain CUDA shared
object exporting the C ABI of include/mixlab_b200.h.  _front.so (csrc/front.cpp)
is a Python extension over torch that calls it.
"""
from __future__ import annotations

import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libmixlab_b200.so")
FRONT = os.path.join(PKG, "_front.so")
SOURCES = ["capi.cu", "dp_grad.cu", "gdn_block.cu", "gdn_chain.cu", "gdn_decode.cu", "gdn_f32io.cu", "gdn_simt.cu", "gdn_static_scratch.cu", "gdn_tc.cu", "gdn_tc64.cu", "gdn_tc_bwd.cu", "mamba3.cu", "mamba3_block.cu", "mamba3_head.cu", "mamba3_ssd.cu", "mamba3_windows.cu", "umma_selftest.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "--std=c++17",
    "--extended-lambda", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC)")


def _front_cmd() -> list[str]:
    torch = importlib.util.find_spec("torch").submodule_search_locations[0]
    inc = os.path.join(torch, "include")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-I" + inc,
            "-I" + os.path.join(inc, "torch", "csrc", "api", "include"), "-I" + sysconfig.get_paths()["include"],
            "-I" + os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"), os.path.join(CSRC, "front.cpp"),
            "-o", FRONT, "-L" + os.path.join(torch, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu",
            "-lc10_cuda", "-lc10"]


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(FRONT):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(FRONT))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(os.path.dirname(PKG), "include", "mixlab_b200.h"))
    return any(os.path.getmtime(p) > t for p in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    nvcc = _nvcc()
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    objs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    procs.append(("front.cpp", subprocess.Popen(_front_cmd(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"--- {src} failed ---\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(out)
    if failed:
        raise RuntimeError("compilation failed")
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs]
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
