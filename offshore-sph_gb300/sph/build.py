"""Build libsph_gb300.so (the CUDA kernels + C ABI) in-tree with nvcc.

The translation units compile in parallel for sm_103a only; the library
links the CUDA runtime statically, so it needs nothing at run time but the
driver.  Output: offshore-sph_gb300/sph/_lib/libsph_gb300.so.
"""
import concurrent.futures as cf
import os
import shutil
import subprocess

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)                      # offshore-sph_gb300/
REPO = os.path.dirname(ROOT)
CSRC = os.path.join(ROOT, "csrc")
INCLUDE = os.path.join(REPO, "include")
LIBDIR = os.path.join(PKG, "_lib")
OBJDIR = os.path.join(ROOT, "_build")
LIB = os.path.join(LIBDIR, "libsph_gb300.so")

SOURCES = ["nn_build.cu", "pair.cu", "pair64.cu", "integrate.cu", "capi.cu", "static_ws.cu", "adjoint.cu", "batch.cu", "newmark.cu",
           "block.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
FLAGS = ["-O3", "-std=c++20", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
         "-I", INCLUDE, "-I", CSRC]
# the mixed-form pair arithmetic flushes FP32 denormals: its reciprocals and
# square roots then take the plain hardware approximations (the FP64 form is
# unaffected; every FP32 pair operand of a real scene is far from 1e-38)
# the per-block plugin equations sum without contraction, as the reference's
# loops do
SOURCE_FLAGS = {"pair.cu": ["-ftz=true"], "block.cu": ["-fmad=false"]}


def nvcc():
    p = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(p):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libsph_gb300")
    return p


def _deps():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "sph_gb300.h")]
    return max(os.path.getmtime(f) for f in files)


def up_to_date():
    return os.path.exists(LIB) and os.path.getmtime(LIB) >= _deps()


def build(force=False, verbose=False, extra_flags=()):
    """Compile the CUDA sources (in parallel) and link the shared library."""
    if not force and up_to_date():
        return LIB
    os.makedirs(LIBDIR, exist_ok=True)
    os.makedirs(OBJDIR, exist_ok=True)
    nv = nvcc()

    def compile_one(src):
        obj = os.path.join(OBJDIR, os.path.splitext(src)[0] + ".o")
        cmd = [nv, "-c", os.path.join(CSRC, src), "-o", obj] + ARCH + FLAGS + SOURCE_FLAGS.get(src, []) + \
            list(extra_flags)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed on %s:\n%s\n%s" % (src, " ".join(cmd), r.stderr))
        if verbose and r.stderr:
            print(r.stderr)
        return obj

    with cf.ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    tmp = LIB + ".tmp%d" % os.getpid()
    cmd = [nv, "-shared", "-o", tmp] + objs + ARCH
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc link failed:\n%s\n%s" % (" ".join(cmd), r.stderr))
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose=True,
                extra_flags=["-Xptxas", "-v"] if "--ptxas" in sys.argv else []))
