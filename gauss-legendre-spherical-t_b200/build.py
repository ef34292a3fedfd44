"""Build step: compile the CUDA engine into ``libglst_b200.so`` (in place).

    python build.py            # or glst_b200.build.build()

nvcc cross-compiles for sm_100a without a GPU.  The shared library is written
next to this file, where the ctypes loader looks for it.
"""
import glob
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libglst_b200.so")
# (source, defines); the slowest first, all compiled at the same time
UNITS = [("far_field.cu", ["-DGLST_PART=%d" % i]) for i in range(5)] + [
    ("engine.cu", []), ("noalloc.cu", []), ("planner.cpp", [])]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc():
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.exists(c) or c == "nvcc"):
            return c
    return "nvcc"


def inputs():
    """Every file the library is built from."""
    return [os.path.join(CSRC, s) for s in dict(UNITS)] + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(
        os.path.join(CSRC, "*.hpp")) + [os.path.join(ROOT, "include", "glst_c.h"), os.path.abspath(__file__)]


def up_to_date(lib=LIB):
    if not os.path.exists(lib):
        return False
    t = os.path.getmtime(lib)
    return all(os.path.getmtime(s) <= t for s in inputs())


def build(force=False, verbose=False, lib=LIB, defines=()):
    """Compile to `lib`, with extra -D options `defines`; returns its path."""
    if not force and up_to_date(lib):
        return lib
    base = [nvcc(), "-std=c++17", "-O3", "-lineinfo", *ARCH, "-Xcompiler", "-fPIC", *defines]
    with tempfile.TemporaryDirectory() as tmp:
        jobs = []
        for i, (src, part) in enumerate(UNITS):
            obj = os.path.join(tmp, "%d.o" % i)
            cmd = base + part + ["-I" + os.path.join(ROOT, "include"), "-c", os.path.join(CSRC, src), "-o", obj]
            if verbose:
                print(" ".join(cmd), flush=True)
            jobs.append((obj, cmd, subprocess.Popen(cmd)))
        failed = [cmd for _, cmd, p in jobs if p.wait() != 0]
        if failed:
            raise subprocess.CalledProcessError(1, failed[0])
        cmd = base + ["-shared", "-o", lib + ".tmp"] + [obj for obj, _, _ in jobs]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    os.replace(lib + ".tmp", lib)
    return lib


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIB)
