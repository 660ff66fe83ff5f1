"""Build step: libintfa.so (one nvcc invocation over csrc/*.cu for sm_100a) and _native.so, the Python binding over it
(one C++ file against PyTorch's headers).

Both are built IN-TREE (next to this file) so that they travel with the source tree; nothing is installed into
site-packages.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB = os.path.join(PKG_DIR, "libintfa.so")
SOURCES = ["intfa_api.cu", "intfa_quant.cu", "intfa_fwd.cu", "intfa_decode.cu"]
HEADERS = ["intfa_internal.h", "intfa_ptx.cuh", "intfa_fwd_pipe.cuh", "intfa_fwd_pipe_softmax.inc",
           "intfa_fwd_pipe_update.inc", os.path.join("..", "..", "include", "intfa.h")]
NATIVE = os.path.join(PKG_DIR, "_native.so")
NATIVE_SOURCES = ["intfa_torch.cpp", os.path.join("..", "..", "include", "intfa.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--threads", "4", "-shared", "-Xcompiler", "-fPIC"]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(CSRC, f) for f in deps]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _native_cmd():
    import torch
    from torch.utils import cpp_extension as ext
    cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
    inc = ext.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-w",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
    cmd += ["-isystem" + d for d in inc] + ["-o", NATIVE, "intfa_torch.cpp", LIB, "-Wl,-rpath,$ORIGIN"]
    for d in ext.library_paths():
        cmd += ["-L" + d, "-Wl,-rpath," + d]
    return cmd + ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]


def _run(cmd, target, verbose):
    res = subprocess.run(cmd, cwd=CSRC, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("%s failed building %s (exit %d)" % (os.path.basename(cmd[0]), os.path.basename(target), res.returncode))


def build(force=False, verbose=False):
    """Compile csrc/ into libintfa.so and _native.so where they are missing or older than their sources."""
    if force or _stale(LIB, SOURCES + HEADERS):
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        # (-soname: the binding finds the library next to itself, by name)
        _run([nvcc] + NVCC_FLAGS + ["-Xlinker", "-soname,libintfa.so"] + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + SOURCES, LIB, verbose)
    if force or _stale(NATIVE, NATIVE_SOURCES):
        _run(_native_cmd(), NATIVE, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
