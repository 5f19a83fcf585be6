"""Ahead-of-time build of the C-ABI CUDA library for sm_100a (no run-time compilation) and of the native host module.

    python -m nvfp4_training_b200.build

writes `libnvfp4_b200.so` and `_host.so` next to this file.  nvcc cross-compiles without a GPU; the host module is plain
C++ against the installed torch and Python headers and needs no CUDA compiler.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libnvfp4_b200.so")
HOST = os.path.join(HERE, "_host.so")
SOURCES = ["quant.cu", "quant_tile.cu", "quant_mma.cu", "quant_w2d.cu", "emit_ops.cu", "emit_rows_ring.cu", "emit_fused.cu", "gemm.cu", "noalloc.cu", "selftest.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc_path():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put the CUDA toolkit on PATH")


def _stale(target, sources):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(CSRC, f) for f in sources] + [os.path.join(HERE, "..", "include", "nvfp4_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _run(cmd, what, verbose):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("compiler failed building " + what)
    if verbose:
        print(res.stdout + res.stderr)


def host_tag():
    """What the host module is tied to: the C++ interfaces of the installed torch and of the interpreter."""
    import torch
    return f"torch {torch.__version__} python {sys.version_info.major}.{sys.version_info.minor}"


def host_is_stale():
    if _stale(HOST, ["host.cpp"]):
        return True
    with open(HOST, "rb") as f:
        return host_tag().encode() not in f.read()           # compiled in below


def build_host(force=False, verbose=False):
    """The host module (`csrc/host.cpp`): torch's C++ headers, the CUDA runtime's headers, no device code."""
    if not force and not host_is_stale():
        return HOST
    import torch
    from torch.utils.cpp_extension import include_paths
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc_path()))), "include")
    incs = [*include_paths(), cuda, sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f'-DNVFP4_HOST_TAG="{host_tag()}"', *[f"-I{d}" for d in incs],
           os.path.join(CSRC, "host.cpp"), "-o", HOST, f"-L{lib_dir}", f"-Wl,-rpath,{lib_dir}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    _run(cmd, HOST, verbose)
    return HOST


def build(force=False, verbose=False):
    build_host(force, verbose)
    if not force and not _stale(LIB, [f for f in os.listdir(CSRC) if f != "host.cpp"]):
        return LIB
    srcs = [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    cmd = [nvcc_path(), "-O3", "-std=c++17", "-lineinfo", "--fmad=false", "-shared", "-Xcompiler", "-fPIC", "--threads", "0",
           "-Xptxas", "-v" if verbose else "-O3", *ARCH, "-o", LIB, *srcs]
    _run(cmd, LIB, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
