"""Compile the CUDA library for sm_100a, in tree.

    python p40-kernel_b200/build.py [--force] [--verbose]

Output: p40-kernel_b200/libbonsai_p40.so (same library name as the reference's build target, so a
program linked with -lbonsai_p40 picks it up unchanged), then bonsai_b200/_calls*.so (the Python package's native
calls into it; left out where there is no torch, which C and C++ programs do not need).  nvcc cross-compiles without a GPU.
No fast-math: the quantiser and the rotation must perform IEEE divisions and separate mul / add.
"""
import argparse
import glob
import importlib.metadata
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libbonsai_p40.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--fmad=false", "-prec-div=true", "-prec-sqrt=true", "-ftz=false",
    "-Xcompiler", "-fPIC", "-shared",
    "--expt-relaxed-constexpr", "--extended-lambda",
]


CALLS_SRC = os.path.join(CSRC, "python_calls.cpp")
CALLS = os.path.join(HERE, "bonsai_b200", "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
CALLS_STAMP = os.path.join(HERE, "build", "calls.stamp")      # what the present _calls file was built for


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")) +
                  glob.glob(os.path.join(HERE, "..", "include", "*.h")))


def stale(out=LIB, srcs=None):
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(s) > t for s in (srcs or sources()))


def compile_to(out, cmd):
    """Runs cmd with a temporary output that takes out's place when it is complete."""
    tmp = f"{out}.{os.getpid()}.tmp"
    try:
        subprocess.check_call([*cmd, "-o", tmp])
        os.replace(tmp, out)
    finally:
        if os.path.exists(tmp):
            os.remove(tmp)


def build_calls(force=False):
    """The native calls of the Python package (CPython extension, links against torch for tensors and streams): built again
    when the source, Python or torch has changed.  None where torch is not installed."""
    try:
        made_for = f"python {sys.version} torch {importlib.metadata.version('torch')}\n"
    except importlib.metadata.PackageNotFoundError:
        return None
    stamp = open(CALLS_STAMP).read() if os.path.exists(CALLS_STAMP) else ""
    if not (force or stamp != made_for or stale(CALLS, [CALLS_SRC])):
        return CALLS
    try:
        import torch
        from torch.utils import cpp_extension
    except ImportError as e:
        print(f"bonsai_b200: the Python calls are left out ({e})", file=sys.stderr)
        return None
    inc = [*cpp_extension.include_paths("cuda"), sysconfig.get_paths()["include"]]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    compile_to(CALLS, [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
                       f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                       *(f"-I{d}" for d in inc), CALLS_SRC,
                       f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"])
    os.makedirs(os.path.dirname(CALLS_STAMP), exist_ok=True)
    with open(CALLS_STAMP, "w") as f:
        f.write(made_for)
    return CALLS


def build(force=False, verbose=False, tuning=True):
    """tuning: compile the geometry knobs of bonsai_b200_set_option in (the parity tests force every tiling through
    them); a production build passes tuning=False (--no-tuning) and keeps only the documented options."""
    if force or stale():
        compile_to(LIB, [NVCC, *(["-Xptxas", "-v"] if verbose else []), *FLAGS, *(["-DBONSAI_B200_TUNING"] if tuning else []),
                         os.path.join(CSRC, "bonsai_b200.cu")])
    build_calls(force)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true", help="print ptxas register / shared-memory usage")
    ap.add_argument("--no-tuning", action="store_true", help="leave the test-only geometry knobs out of the library")
    a = ap.parse_args()
    print(build(a.force or a.no_tuning, a.verbose, not a.no_tuning))
    sys.exit(0)
