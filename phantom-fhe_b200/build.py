"""Builds libb200fhe.so in-tree with nvcc for sm_100a (cross-compiles without a GPU)."""
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
SRCS = [os.path.join(HERE, "csrc", f) for f in ("b200fhe.cu", "ntt_whole.cu")]  # compiled side by side
OUT = os.path.join(HERE, "libb200fhe.so")
DEPS = glob.glob(os.path.join(HERE, "csrc", "*")) + [os.path.join(os.path.dirname(HERE), "include", "b200fhe.h")]
FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-Xcompiler", "-fPIC,-fopenmp"]


def build_native(force=False, verbose=False):
    if not force and os.path.exists(OUT) and all(os.path.getmtime(OUT) >= os.path.getmtime(d) for d in DEPS if not d.endswith(".o")):
        return OUT
    objs = [s[:-3] + ".o" for s in SRCS]
    procs = [subprocess.Popen(["nvcc"] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", "-o", o, s]) for s, o in zip(SRCS, objs)]
    codes = [p.wait() for p in procs]
    if any(codes):
        raise subprocess.CalledProcessError(next(c for c in codes if c), "nvcc -c")
    subprocess.check_call(["nvcc"] + FLAGS + ["-shared", "-lgomp", "-o", OUT] + objs)
    return OUT


if __name__ == "__main__":
    print(build_native(force="--force" in sys.argv, verbose="-v" in sys.argv))
