"""Build libb200attn.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and the native
call path of the tensor-level entry points (against the installed torch and Python, whose versions
its file name carries: another torch looks for another file).

    python -m tritonops_b200.build [--force]
"""
import os
import subprocess
import sys
import sysconfig

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc")
LIB = os.path.join(CSRC, "libb200attn.so")
SOURCES = ["api.cu", "decode.cu", "prefill.cu", "prefill_bwd.cu", "kvcache.cu", "blocksel.cu", "rmsnorm.cu", "selftest.cu"]
HEADERS = ["common.cuh", os.path.join("..", "..", "include", "b200attn.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared"]


def host_path():
    """Where the native call path for this torch and this Python is built."""
    import torch
    return os.path.join(CSRC, f"_b200host.torch-{torch.__version__}.{sysconfig.get_config_var('SOABI')}.so")


def _stale():
    if not os.path.exists(LIB) or not os.path.exists(host_path()):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(host_path()))
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS]
    deps += [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".cu", ".cpp"))]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build_library(force=False, verbose=False):
    """Compile the CUDA sources into csrc/libb200attn.so; returns its path."""
    if not force and not _stale():
        return LIB
    for f in os.listdir(CSRC):      # none may stay beside a library it was not built with
        if f.startswith("_b200host.") and f.endswith(".so"):
            os.remove(os.path.join(CSRC, f))
    nvcc = os.environ.get("NVCC", "nvcc")
    cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + SOURCES
    res = subprocess.run(cmd, cwd=CSRC, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    build_host()
    return LIB


def build_host():
    """Compile csrc/host.cpp."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include",
           f"-I{sysconfig.get_paths()['include']}", "-o", host_path(), "host.cpp",
           f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", f"-Wl,-rpath,{root}/lib"]
    res = subprocess.run(cmd, cwd=CSRC, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("host build failed:\n" + res.stdout + res.stderr)


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
