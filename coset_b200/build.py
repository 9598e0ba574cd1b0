"""Builds libcoset_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and _coset_torch.so
(the native PyTorch entry points on top of it) with g++.

    python -m coset_b200.build [--force] [--verbose]

The library is self-contained (static cudart, no torch symbols).  Codec translation units are
compiled with -fmad=false: the reference rounds after every float32 operation, so a contracted
multiply-add would change codes.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libcoset_b200.so")
TORCH_PATH = os.path.join(LIB_DIR, "_coset_torch.so")
TORCH_SOURCE = "torch_binding.cpp"
TORCH_STAMP = os.path.join(LIB_DIR, "_coset_torch.version")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

SOURCES = [
    "e8_codec.cu",
    "e8_layer.cu",
    "e8_host.cu",
    "e8_gradcomm.cu",
    "e8_vlut.cu",
    "e8_vlut_bytes.cu",
    "e8_stats.cu",
    "e8_ref.cu",
    "e8_dequant_gemm.cu",
    "e8_decode_gemm.cu",
    "e8_dense_gemm.cu",
    "f32_product.cu",
    "d4.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-fmad=false", "-prec-div=true", "-prec-sqrt=true", "-ftz=false",
    "-Xcompiler", "-fPIC",
]


def _nvcc():
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def _newer(target, deps):
    """True if `target` exists and is no older than any of `deps`."""
    return os.path.exists(target) and all(os.path.getmtime(d) <= os.path.getmtime(target) for d in deps)


def _run(cmd, verbose):
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.check_call(cmd)


def _torch_stamp():
    """What the PyTorch module is bound to besides its source: its ABI follows the version of torch and of Python."""
    import torch
    return f"torch {torch.__version__}, Python {sys.version.split()[0]}\n"


def _stamp_is(text):
    try:
        with open(TORCH_STAMP) as f:
            return f.read() == text
    except OSError:
        return False


def _build_torch_module(verbose):
    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    inc = [f for d in (*cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]) for f in ("-isystem", d)]
    libs = [f for d in cpp_extension.library_paths() for f in ("-L", d)]
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc,
          os.path.join(CSRC, TORCH_SOURCE), "-o", TORCH_PATH, "-L", LIB_DIR, "-lcoset_b200", "-Wl,-rpath,$ORIGIN", *libs,
          "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"], verbose)


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ that changed (or whose headers did) into lib/libcoset_b200.so, then the
    PyTorch module; returns the library's path."""
    os.makedirs(LIB_DIR, exist_ok=True)
    header = os.path.join(INCLUDE, "coset_b200.h")
    shared = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")] + [header, __file__]
    todo, objs = [], []
    for src in SOURCES:
        obj = os.path.join(LIB_DIR, src.replace(".cu", ".o"))
        objs.append(obj)
        if not force and _newer(obj, [os.path.join(CSRC, src), *shared]):
            continue
        verb = ["-Xptxas=-v"] if verbose else []
        todo.append([_nvcc(), *verb, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj])
    with ThreadPoolExecutor(max_workers=max(1, min(len(todo), os.cpu_count() or 1))) as pool:
        list(pool.map(lambda cmd: _run(cmd, verbose), todo))
    if force or not _newer(LIB_PATH, objs):
        _run([_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"], verbose)
    # the module finds the library's functions at load time: only its own source and the header matter to it
    stamp = _torch_stamp()
    if force or not _stamp_is(stamp) or not _newer(TORCH_PATH, [os.path.join(CSRC, TORCH_SOURCE), header, __file__]):
        _build_torch_module(verbose)
        with open(TORCH_STAMP, "w") as f:
            f.write(stamp)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
