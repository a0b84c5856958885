"""Build the C-ABI CUDA library in-tree: csrc/*.cu -> mpsa/libmpsa.so (sm_100a only), and the Python module in front of its short
calls: csrc/native.cpp -> mpsa/_native.<Python tag>.torch-<version>.so.

    python mp-sparse-attn_b200/build.py [--force]

nvcc cross-compiles for sm_100a without a GPU.  The runtime is linked statically and the
driver API is reached through cudaGetDriverEntryPoint, so the library also loads on a
machine without a CUDA driver (used by the CPU-side symbol test).
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "mpsa", "libmpsa.so")
NATIVE_SRC = os.path.join(CSRC, "native.cpp")
SOURCES = ["api.cu", "quant.cu", "prep.cu", "gemm.cu", "attn.cu", "route.cu", "attention.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=default", "--use_fast_math=false"]


def _nvcc():
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def needs_build():
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    for f in os.listdir(CSRC):
        if f != "native.cpp" and os.path.getmtime(os.path.join(CSRC, f)) > t:
            return True
    return os.path.getmtime(__file__) > t


def build_lib(force=False, verbose=False):
    if not force and not needs_build():
        return OUT
    flags = [f for f in NVCC_FLAGS if not f.startswith("--use_fast_math")]
    objs = []
    bdir = os.path.join(HERE, "build")
    os.makedirs(bdir, exist_ok=True)
    procs = []
    for s in SOURCES:
        o = os.path.join(bdir, s.replace(".cu", ".o"))
        cmd = [_nvcc(), *flags, "-I", CSRC, "-c", os.path.join(CSRC, s), "-o", o]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(o)
    for s, pr in procs:
        out, _ = pr.communicate()
        if verbose and out:
            print(out)
        if pr.returncode != 0:
            raise RuntimeError(f"nvcc failed on {s}:\n{out}")
    cmd = [_nvcc(), "-shared", "-o", OUT, *objs, "-cudart", "static"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    return OUT


def native_out():
    """Where the module for this Python and this torch is: one made for another of either is never loaded."""
    import sysconfig

    import torch
    return os.path.join(HERE, "mpsa", f"_native.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so")


def build_native(force=False):
    """csrc/native.cpp -> native_out(), the module that takes torch tensors to the library (needs torch's headers)."""
    out = native_out()
    header = os.path.join(os.path.dirname(HERE), "include", "mpsa.h")
    if not force and os.path.exists(out) and os.path.getmtime(out) >= max(os.path.getmtime(f) for f in (NATIVE_SRC, header, __file__)):
        return out
    import sysconfig

    import torch
    base = os.path.dirname(torch.__file__)
    inc = [sysconfig.get_paths()["include"], os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    new = f"{out}.{os.getpid()}.new"                # (several ranks may get here at a time)
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *("-I" + i for i in inc), NATIVE_SRC, "-o", new,
           "-L" + os.path.join(base, "lib"), "-ltorch_python", "-ltorch_cpu", "-ltorch", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on native.cpp:\n{r.stdout}")
    os.replace(new, out)
    return out


if __name__ == "__main__":
    print(build_lib(force="--force" in sys.argv, verbose="-v" in sys.argv))
    try:
        print(build_native("--force" in sys.argv))
    except (ImportError, OSError, RuntimeError) as e:      # (no torch, no compiler, no headers: short calls go through ctypes)
        print(f"not built: the native module for short calls ({type(e).__name__}: {e})", file=sys.stderr)
