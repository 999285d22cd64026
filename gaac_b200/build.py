"""Build in-tree the CUDA library, gaac_b200/libgaac_b200.so (sm_100a only), and the module that calls it with tensors, gaac_b200/_host.so.

    python -m gaac_b200.build            # build if sources are newer than the library
    python -m gaac_b200.build --force

nvcc cross-compiles without a GPU, so this also runs on a CPU-only box.
"""
from __future__ import annotations
import os, subprocess, sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libgaac_b200.so")
SOURCES = ["gaac_encode.cu", "gaac_attn.cu", "gaac_cache.cu", "gaac_noalloc.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--use_fast_math",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


HOST = os.path.join(HERE, "_host.so")


def _host_command():
    """The module is built against the torch that will load it."""
    import sysconfig
    import torch
    at = os.path.dirname(torch.__file__)
    include = [os.path.join(at, "include"), os.path.join(at, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *("-I" + d for d in include),
            os.path.join(CSRC, "gaac_host.cpp"), "-o", HOST, "-L" + os.path.join(at, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-ldl"]


def _sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(HOST):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(os.path.dirname(HERE), "include", "gaac_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = [("gaac_host.cpp", subprocess.Popen(_host_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True))]
    for src in _sources():
        obj = os.path.join("/tmp", "gaac_b200_" + os.path.basename(src) + ".o")
        objs.append(obj)
        procs.append((src, subprocess.Popen([nvcc, *NVCC_FLAGS, "-c", src, "-o", obj], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode:
            print(out)
        if pr.returncode:
            raise RuntimeError(f"the compiler failed on {src}")
    subprocess.check_call([nvcc, "-shared", "-o", LIB, *objs, "-lcudart"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
