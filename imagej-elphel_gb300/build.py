"""Build recipe for libtp.so (the GB300 tile processor, C ABI in include/tp.h).

Compiles the CUDA translation units for sm_103a only, in parallel, and links a
shared library into imagej-elphel_gb300/_build/.  Host code is compiled with
-ffp-contract=off so the FP64 geometry set-up (rotation matrices, reverse
distortion table) is evaluated without fused multiply-adds on both x86_64 and
aarch64; the FP64 device geometry uses explicitly rounded intrinsics.
"""
import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "_build")
LIB = os.path.join(OUT_DIR, "libtp.so")
SOURCES = ["tp_plan.cu", "tp_kernels.cu", "tp_fused.cu", "tp_quad.cu", "tp_many.cu", "tp_texture.cu", "tp_adjoint.cu", "tp_adjoint_many.cu", "tp_adjoint_quad.cu", "tp_kernprep.cu", "tp_lma.cu",
           "tp_host.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]


def nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _deps():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files.append(os.path.join(REPO, "include", "tp.h"))
    files.append(os.path.abspath(__file__))
    return max(os.path.getmtime(f) for f in files)


def _compile(src, obj):
    cmd = [nvcc(), *ARCH, "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off",
           "-I", os.path.join(REPO, "include"), "-c", os.path.join(CSRC, src), "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, " ".join(cmd), r.stderr))
    return obj


def build(force=False, verbose=False):
    os.makedirs(OUT_DIR, exist_ok=True)
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= _deps():
        return LIB
    objs = [os.path.join(OUT_DIR, os.path.splitext(s)[0] + ".o") for s in SOURCES]
    with cf.ThreadPoolExecutor(len(SOURCES)) as ex:
        list(ex.map(_compile, SOURCES, objs))
    tmp = LIB + ".tmp.%d" % os.getpid()
    cmd = [nvcc(), *ARCH, "-shared", "-o", tmp, *objs, "-Xcompiler", "-fPIC"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s" % r.stderr)
    os.replace(tmp, LIB)
    if verbose:
        print(LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
