"""Build libfat_b200.so (the C-ABI library, nvcc for sm_100a) and libfat_torch_ops.so (the torch.library operators, g++) in-tree.

    python -m fastalgebraictransformer_b200.build [--force] [--verbose]

Every .cu under csrc/ is compiled to an object in csrc/_obj/ (in parallel) and linked into
fastalgebraictransformer_b200/libfat_b200.so.  nvcc cross-compiles, so no GPU is needed.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(PKG, "libfat_b200.so")
OPS_SRCS = [os.path.join(CSRC, n) for n in ("torch_ops.cpp", "torch_autograd.cpp")]
OPS_LIB = os.path.join(PKG, "libfat_torch_ops.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put the CUDA toolkit on PATH")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile and link the library if any source is newer than it.  Returns the .so path."""
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + \
        sorted(glob.glob(os.path.join(PKG, "..", "include", "*.h")))
    if not sources:
        raise RuntimeError(f"no CUDA sources under {CSRC}")
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src] + headers):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-Xptxas", "-v", "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for src, r in ex.map(compile_one, jobs):
                if verbose or r.returncode:
                    sys.stderr.write(r.stdout + r.stderr)
                if r.returncode:
                    raise RuntimeError(f"nvcc failed on {src}")
    objs = [os.path.join(OBJ, os.path.basename(s)[:-3] + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of libfat_b200.so failed")
    build_ops(force, verbose)
    build_wait_test(force, verbose)
    build_fill_shared(force)
    return LIB


WAIT_TEST_LIB = os.path.join(PKG, "..", "tests", "_build", "libfat_b200_waittest.so")
WAIT_TEST_FLAGS = ["-DFAT_TEST_WITHHOLD_V_TILE=0", "-DFAT_TEST_CE_WITHHOLD_ROW=4", "-DFAT_TEST_LM_WITHHOLD_UNIT=0", "-DFAT_TEST_LM_NO_RING_WAIT=301",
                   "-DFAT_WAIT_HINT_NS=100000",
                   "-DFAT_WAIT_SPINS=30", "-DFAT_LM_POLL_LIMIT=4096"]
WAIT_TEST_SOURCES = ("attn_tc_fwd.cu", "loss.cu", "lm_decode.cu")


def build_wait_test(force: bool = False, verbose: bool = False) -> str:
    """A TEST-ONLY variant of the library (tests/_build/, never loaded by the package): the attention forward is compiled
    so that its producer leaves out one V tile, the staged loss kernel so that its first block never requests the copy of
    one row, the language model's decode step so that one unit of its first projection is never handed on and, with a vocabulary of 301, no
    warp waits for its weights, and every bounded wait gives up after ~3 ms.  tests/test_wait_timeout.py uses it to run the give-up paths once (status word, NaN losses or
    logits, teardown, TMEM release).  Only those sources are recompiled; the other objects are the shipped ones."""
    srcs = [os.path.join(CSRC, n) for n in WAIT_TEST_SOURCES]
    headers = sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + sorted(glob.glob(os.path.join(PKG, "..", "include", "*.h")))
    out_dir = os.path.dirname(WAIT_TEST_LIB)
    os.makedirs(out_dir, exist_ok=True)
    objs = [os.path.join(out_dir, n[:-3] + "_waittest.o") for n in WAIT_TEST_SOURCES]
    others = [os.path.join(OBJ, os.path.basename(s)[:-3] + ".o") for s in sorted(glob.glob(os.path.join(CSRC, "*.cu")))
              if os.path.basename(s) not in WAIT_TEST_SOURCES]
    if not (force or _stale(WAIT_TEST_LIB, srcs + headers + others)):
        return WAIT_TEST_LIB
    nvcc = _nvcc()
    cmds = [[nvcc, *NVCC_FLAGS, *WAIT_TEST_FLAGS, "-c", src, "-o", obj] for src, obj in zip(srcs, objs)]
    link = [nvcc, "-shared", "-o", WAIT_TEST_LIB, *objs, *others, "-gencode", "arch=compute_100a,code=sm_100a"]

    def run(cmd):
        return subprocess.run(cmd, capture_output=True, text=True)

    with cf.ThreadPoolExecutor(max_workers=len(cmds)) as ex:
        results = list(ex.map(run, cmds))
    if all(r.returncode == 0 for r in results):
        results.append(run(link))
    for r in results:
        if verbose or r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError("build of the wait-timeout test library failed")
    return WAIT_TEST_LIB


FILL_SHARED_LIB = os.path.join(PKG, "..", "tests", "_build", "libfill_shared.so")


def build_fill_shared(force: bool = False) -> str:
    """The tests' kernel that fills shared memory (tests/fill_shared.cu -> tests/_build/, never loaded by the package)."""
    src = os.path.join(PKG, "..", "tests", "fill_shared.cu")
    if os.path.exists(src) and (force or _stale(FILL_SHARED_LIB, [src])):
        os.makedirs(os.path.dirname(FILL_SHARED_LIB), exist_ok=True)
        r = subprocess.run([_nvcc(), *NVCC_FLAGS, "-shared", src, "-o", FILL_SHARED_LIB], capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("build of the tests' libfill_shared.so failed")
    return FILL_SHARED_LIB


def build_ops(force: bool = False, verbose: bool = False) -> str:
    """Compile the C++ registration of the torch.library operators (csrc/torch_ops.cpp) and their autograd nodes and Python
    entry points (csrc/torch_autograd.cpp) against the installed torch and link them to libfat_b200.so; the result is also
    an extension module.  Host code only: g++, no nvcc."""
    header = os.path.join(PKG, "..", "include", "fat_b200.h")
    if not (force or _stale(OPS_LIB, [*OPS_SRCS, header, LIB])):
        return OPS_LIB
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ce
    cuda_home = os.environ.get("CUDA_HOME") or os.path.dirname(os.path.dirname(_nvcc()))
    cxx = os.environ.get("CXX") or shutil.which("g++") or "g++"
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
             "-I" + os.path.join(cuda_home, "include"), "-I" + sysconfig.get_paths()["include"]]
    flags += ["-I" + p for p in ce.include_paths()]
    objs = [os.path.join(OBJ, os.path.basename(src)[:-4] + ".o") for src in OPS_SRCS]
    cmds = [[cxx, *flags, "-c", src, "-o", obj] for src, obj in zip(OPS_SRCS, objs) if force or _stale(obj, [src, header])]
    link = [cxx, "-shared", *objs, "-o", OPS_LIB] + ["-L" + p for p in ce.library_paths()]
    link += ["-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python", "-L" + PKG, "-lfat_b200", "-Wl,-rpath,$ORIGIN"]
    # the C++ library of the process, by name: a compiler that only has the static one would put a second copy into this module,
    # whose stream facets are not the process's (writing a number into an error text crashed)
    link.append("-l:libstdc++.so.6")

    def run(cmd):
        return subprocess.run(cmd, capture_output=True, text=True)

    with cf.ThreadPoolExecutor(max_workers=2) as ex:
        results = list(ex.map(run, cmds))
    if all(r.returncode == 0 for r in results):
        results.append(run(link))
    for r in results:
        if verbose or r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError("build of libfat_torch_ops.so failed")
    return OPS_LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
