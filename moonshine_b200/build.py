"""Build the native library in-tree with nvcc for sm_100a.

``python -m moonshine_b200.build`` compiles every ``csrc/*.cu`` into
``moonshine_b200/libk3moe.so`` and ``csrc/k3_pyops.cpp``, the CPython bindings of
its entry points, into ``moonshine_b200/_k3ops.so`` (without a C++ compiler or Python's
headers that step is left out with a warning: the calls then go through ctypes).  Object files are cached
under ``moonshine_b200/_build`` and rebuilt when a source or header is newer.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libk3moe.so")
BINDINGS = os.path.join(HERE, "_k3ops.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall", "--expt-relaxed-constexpr",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _newest_header() -> float:
    hdrs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(ROOT, "include", "*.h"))
    return max(os.path.getmtime(h) for h in hdrs)


def build(verbose: bool = False, force: bool = False, ptxas_info: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    if not sources:
        raise RuntimeError("no CUDA sources under " + CSRC)
    hdr_time = _newest_header()
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if ptxas_info:
                cmd[1:1] = ["-Xptxas", "-v"]
            jobs.append(cmd)

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or res.returncode != 0 or ptxas_info:
            sys.stderr.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
        if res.returncode != 0:
            raise RuntimeError("compilation failed: " + " ".join(cmd))

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        list(pool.map(run, jobs))
    if jobs or not os.path.exists(LIB):
        link = [nvcc, "-shared", "-o", LIB, *objs, "-lcuda"]
        res = subprocess.run(link, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    src = os.path.join(CSRC, "k3_pyops.cpp")
    if force or not os.path.exists(BINDINGS) or os.path.getmtime(BINDINGS) < max(os.path.getmtime(src), hdr_time):
        try:
            run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall",
                 "-I", os.path.join(ROOT, "include"), "-I", sysconfig.get_paths()["include"], "-o", BINDINGS, src,
                 "-L", HERE, "-l:libk3moe.so", "-Wl,-rpath,$ORIGIN"])
        except (OSError, RuntimeError) as e:
            if os.path.exists(BINDINGS):               # one built for other headers must not stay
                os.remove(BINDINGS)
            sys.stderr.write(f"warning: no CPython bindings, operator calls go through ctypes ({e})\n")
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv, ptxas_info="-p" in sys.argv))
