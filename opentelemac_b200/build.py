"""Build the native library libbief_b200.so (sm_100a) in-tree.

The library is plain CUDA C++ with an extern "C" interface
(include/bief_b200.h); it does not link against torch.
"""
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libbief_b200.so")

SOURCES = ["bief_api.cu", "bief_krylov.cu", "bief_noalloc.cu", "bief_resident.cu"]
HEADERS = ["bief_device.cuh", "bief_kernels.cuh", "bief_batch.cuh", "bief_krylov.h",
           "bief_resident.h"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False, defines=(), out=None):
    os.makedirs(LIBDIR, exist_ok=True)
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    deps = srcs + [os.path.join(CSRC, h) for h in HEADERS] + [
        os.path.join(ROOT, "include", "bief_b200.h"), __file__]
    target = out or LIB
    if not force and not _stale(target, deps):
        return target
    # the sources compile side by side, then link
    base = [nvcc(), *ARCH, "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC"]
    opts = ["-I", os.path.join(ROOT, "include"), *[f"-D{d}" for d in defines]]
    if verbose:
        opts.insert(0, "-Xptxas=-v")
    with tempfile.TemporaryDirectory(dir=LIBDIR) as tmp:
        objs = [os.path.join(tmp, os.path.basename(f) + ".o") for f in srcs]
        cmds = [[*base, *opts, "-c", f, "-o", o] for f, o in zip(srcs, objs)]
        if verbose:
            print("\n".join(" ".join(c) for c in cmds))
        procs = [subprocess.Popen(c) for c in cmds]
        for c, p in zip(cmds, [p.wait() for p in procs]):
            if p:
                raise subprocess.CalledProcessError(p, c)
        subprocess.run([*base, "-shared", "-o", target, *objs], check=True)
    return target


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
