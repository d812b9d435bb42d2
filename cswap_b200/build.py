"""Builds libcswap_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU) and the CPython extension
behind codec.py."""
from __future__ import annotations

import importlib.metadata
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libcswap_b200.so")
ROOT = os.path.dirname(HERE)
SOURCES = ["zfp_kernels.cu", "sparse_kernels.cu", "cswap_abi.cu", "swap_manager.cu", "cost_model.cu",
           "sparse_static.cu"]
HEADERS = ["pdl.cuh", "zfp_core.cuh", "zfp_field.cuh", "zfp_kernels.h", "sparse_kernels.h", "tile_counts.cuh", "internal.h",
           os.path.join("..", "..", "include", "cswap_b200.h"), os.path.join("..", "..", "include", "cswap_compat.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.exists(d) and os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """The CUDA library and, where torch is installed, the extension module; returns the library's path."""
    build_library(force, verbose)
    build_ext(force)
    return LIB


def build_library(force: bool = False, verbose: bool = False) -> str:
    """The CUDA library alone: needs nvcc, neither torch nor Python's headers."""
    if not force and not needs_build():
        return LIB
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    objs = []
    procs = []
    for s in SOURCES:
        o = os.path.join(objdir, s.replace(".cu", ".o"))
        cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + \
              ["-c", os.path.join(CSRC, s), "-o", o]
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(o)
    for s, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {s}")
    cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-Xcompiler", "-fPIC"]
    subprocess.check_call(cmd)
    return LIB


EXT_SOURCE = os.path.join(CSRC, "codec_ext.cpp")
EXT = os.path.join(HERE, "_codec_ext.so")
EXT_STAMP = os.path.join(HERE, "build", "_codec_ext.built_for")


def _built_for() -> str:
    """What an extension module is good for: the interpreter and the torch it was compiled against."""
    try:
        torch_version = importlib.metadata.version("torch")
    except importlib.metadata.PackageNotFoundError:
        torch_version = "none"
    return f"{sysconfig.get_config_var('SOABI')} torch {torch_version}"


def _ext_up_to_date() -> bool:
    deps = [EXT_SOURCE, os.path.join(ROOT, "include", "cswap_b200.h"), os.path.abspath(__file__)]
    if not os.path.exists(EXT) or not os.path.exists(EXT_STAMP):
        return False
    if any(os.path.getmtime(EXT) < os.path.getmtime(d) for d in deps):
        return False
    with open(EXT_STAMP) as f:
        return f.read() == _built_for()


def build_ext(force: bool = False) -> str | None:
    """Compile the CPython extension behind codec.py against the installed
    libtorch and the in-tree library (g++; needs no GPU).  Without torch there
    is nothing it could serve: None."""
    if not force and _ext_up_to_date():
        return EXT
    try:
        import torch
    except ImportError:
        sys.stderr.write("cswap_b200: torch is not installed, so the extension behind codec.py is not built\n")
        return None
    t = os.path.dirname(torch.__file__)
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    cmd = ["g++", "-std=c++17", "-O2", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(t, "include"),
           "-I", os.path.join(t, "include", "torch", "csrc", "api", "include"), "-I", cuda_inc,
           EXT_SOURCE, "-o", EXT, "-L", os.path.join(t, "lib"), "-L", HERE,
           f"-Wl,-rpath,{os.path.join(t, 'lib')}", "-Wl,-rpath,$ORIGIN",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-lcswap_b200"]
    subprocess.check_call(cmd)
    os.makedirs(os.path.dirname(EXT_STAMP), exist_ok=True)
    with open(EXT_STAMP, "w") as f:
        f.write(_built_for())
    return EXT


CPP_DRIVERS = ("execution_driver", "vgg16_step", "bert_step")


def build_cpp_driver(force: bool = False, name: str = "execution_driver") -> str:
    """Compile tests/cpp/<name>.cpp (drivers written against the C++ Execution
    class over stock libtorch, include/cswap_execution.hpp) against the in-tree
    library with g++."""
    import torch
    root = os.path.dirname(HERE)
    src = os.path.join(root, "tests", "cpp", name + ".cpp")
    hdrs = [os.path.join(root, "include", h) for h in ("cswap_execution.hpp", "cswap_b200.h")]
    exe = os.path.join(root, "tests", "cpp", name)
    if not force and os.path.exists(exe) and all(os.path.getmtime(exe) >= os.path.getmtime(f) for f in [src] + hdrs):
        return exe
    build()
    t = os.path.dirname(torch.__file__)
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    # the CUDA runtime libtorch itself is linked against (its wheel ships one), else the toolkit's
    import glob
    rt = sorted(glob.glob(os.path.join(os.path.dirname(t), "nvidia", "cuda_runtime", "lib", "libcudart.so.*")))
    rt = rt[0] if rt else os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "lib64", "libcudart.so")
    cmd = ["g++", "-std=c++17", "-O1", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", os.path.join(root, "include"), "-I", os.path.join(t, "include"),
           "-I", os.path.join(t, "include", "torch", "csrc", "api", "include"), "-I", cuda_inc, src, "-o", exe,
           "-L", os.path.join(t, "lib"), "-L", HERE, f"-Wl,-rpath,{os.path.join(t, 'lib')}",
           "-Wl,-rpath,$ORIGIN/../../cswap_b200", "-Wl,--no-as-needed",
           "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-lcswap_b200", rt,
           f"-Wl,-rpath,{os.path.dirname(rt)}", "-Wno-interference-size"]
    subprocess.check_call(cmd)
    return exe


def build_cpp_drivers(force: bool = False):
    return [build_cpp_driver(force, n) for n in CPP_DRIVERS]


if __name__ == "__main__":
    if "--cpp" in sys.argv:
        print(build_cpp_drivers(force="--force" in sys.argv))
        sys.exit(0)
    make = build_library if "--library" in sys.argv else build
    print(make(force="--force" in sys.argv, verbose="-v" in sys.argv))
