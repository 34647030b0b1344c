"""In-tree build of libmw3gpu.so for sm_103a (nvcc, no cmake).

The translation units compile in parallel; objects and the shared library go
to madwave3_gb300/_build/ (git-ignored).  Nothing here falls back to another
architecture or to a CPU path.
"""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "_build")
LIB = os.path.join(OUT, "libmw3gpu.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
SOURCES = ["mw3_api.cu", "mw3_kernels.cu", "mw3_setup.cu", "mw3_tc.cu", "mw3_tc_ang.cu", "mw3_tc_dst2d.cu",
           "mw3_fx.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
# host code without FMA contraction: the reference's x86-64 build never contracts,
# and set-up tables (absorber start, flux line) must not depend on the host CPU
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-ffp-contract=off", "-I" + INCLUDE]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _deps():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "mw3gpu.h")]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False, extra_flags=()):
    """Compile every CUDA translation unit and link libmw3gpu.so; returns its path."""
    os.makedirs(OUT, exist_ok=True)
    deps = _deps()
    if not force and not _stale(LIB, deps):
        return LIB
    nvcc = _nvcc()

    def compile_one(src):
        obj = os.path.join(OUT, src.replace(".cu", ".o"))
        cmd = [nvcc] + ARCH + NVCC_FLAGS + list(extra_flags) + ["-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed for %s:\n%s%s" % (src, r.stdout, r.stderr))
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    tmp = LIB + ".tmp"
    cmd = [nvcc] + ARCH + ["-shared", "-o", tmp] + objs
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s%s" % (r.stdout, r.stderr))
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
