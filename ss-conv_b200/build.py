"""Build libssconv_b200.so (the C-ABI CUDA library, sm_100a, nvcc) and its Python bindings (g++) in-tree.

Usage: python ss-conv_b200/build.py [--force] [--verbose]
The shared library is written next to the Python package (ss_conv/libssconv_b200.so) so that
it travels with the source tree; no JIT cache is involved.
"""
import importlib.metadata
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "ss_conv", "libssconv_b200.so")
BINDINGS = os.path.join(HERE, "ss_conv", "_host.so")
MADE_FOR = os.path.join(HERE, "build", "_host.versions")
SOURCES = ["ssc_error.cu", "ssc_rulebook.cu", "ssc_conv.cu", "ssc_conv_tc.cu", "ssc_conv_stage.cu", "ssc_conv_pairs.cu", "ssc_backward.cu", "ssc_order.cu", "ssc_wgrad_tc.cu", "ssc_pool.cu", "ssc_layer.cu", "ssc_voxel.cu",
           "ssc_bnact.cu", "ssc_ceiling.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc():
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = os.path.join(home, "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _newest_input():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")] + [os.path.join(HERE, "..", "include", "ssconv_b200.h")]
    return max(os.path.getmtime(f) for f in files if os.path.exists(f))


def _versions():
    """What the bindings are bound to besides their sources."""
    return "python %s, torch %s" % (sys.version, importlib.metadata.version("torch"))


def bindings_current(inputs):
    """The bindings are newer than their sources and made for this Python and this torch."""
    if not (os.path.exists(BINDINGS) and os.path.exists(MADE_FOR)):
        return False
    with open(MADE_FOR) as f:
        return f.read() == _versions() and os.path.getmtime(BINDINGS) >= max(os.path.getmtime(i) for i in inputs)


def build_bindings(force=False):
    """ss_conv/_host.so: needs the headers of Python and torch, no GPU toolkit."""
    inputs = [os.path.join(CSRC, "ssc_host.cpp"), os.path.join(HERE, "..", "include", "ssconv_b200.h")]
    if not force and bindings_current(inputs):
        return BINDINGS
    import sysconfig
    import torch
    base = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", inputs[0], "-o", BINDINGS, "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
           "-I" + base, "-I" + os.path.join(base, "torch", "csrc", "api", "include"), "-I" + sysconfig.get_paths()["include"], "-I" + cuda,
           "-L" + os.path.dirname(LIB), "-lssconv_b200", "-Wl,-rpath,$ORIGIN",
           "-L" + os.path.join(os.path.dirname(torch.__file__), "lib"), "-ltorch_python", "-ltorch_cpu", "-ltorch", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed on ssc_host.cpp:\n" + r.stderr[-6000:])
    os.makedirs(os.path.dirname(MADE_FOR), exist_ok=True)
    with open(MADE_FOR, "w") as f:
        f.write(_versions())
    return BINDINGS


def build(force=False, verbose=False):
    lib = build_library(force, verbose)
    build_bindings(force)
    return lib


def build_library(force=False, verbose=False):
    sources = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    if os.path.exists(LIB) and not force and os.path.getmtime(LIB) >= _newest_input():
        return LIB
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    nvcc = _nvcc()
    flags = list(NVCC_FLAGS)

    def compile_one(src):
        obj = os.path.join(objdir, src + ".o")
        cmd = [nvcc, "-c", os.path.join(CSRC, src), "-o", obj] + flags + (["-Xptxas", "-v"] if verbose else [])
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed on %s:\n%s" % (src, r.stderr[-6000:]))
        if verbose:
            print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources))
    r = subprocess.run([nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"],
                       capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stderr[-4000:])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
