"""Build in-tree the CUDA library, gaac_b200/libgaac_b200.so (sm_100a only), and the module that calls it with tensors, gaac_b200/_host.<interpreter>.so.

    python -m gaac_b200.build            # build if sources are newer than the library
    python -m gaac_b200.build --force

nvcc cross-compiles without a GPU, so this also runs on a CPU-only box.
"""
from __future__ import annotations
import os, re, subprocess, sys, sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libgaac_b200.so")
SOURCES = ["gaac_encode.cu", "gaac_attn.cu", "gaac_cache.cu", "gaac_noalloc.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--use_fast_math",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]
C_ABI = os.path.join(os.path.dirname(HERE), "include", "gaac_b200.h")
HOST = os.path.join(HERE, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))              # another interpreter does not take it for its own


def _host_command():
    """The module is built against the torch that will load it."""
    import torch
    at = os.path.dirname(torch.__file__)
    include = [os.path.join(at, "include"), os.path.join(at, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f"-DGAAC_TORCH_VERSION={torch.__version__}", *("-I" + d for d in include),
            os.path.join(CSRC, "gaac_host.cpp"), "-o", HOST, "-L" + os.path.join(at, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-ldl"]


def _sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _stale(made: str, sources) -> bool:
    return not os.path.exists(made) or any(os.path.getmtime(d) > os.path.getmtime(made) for d in sources)


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))] + [C_ABI]


def _start(name, command):
    return name, subprocess.Popen(command, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish(started, verbose: bool):
    failed = None
    for name, pr in started:
        out, _ = pr.communicate()
        if verbose or pr.returncode:
            print(out)
        if pr.returncode:
            failed = failed or name
    if failed:
        raise RuntimeError(f"the compiler failed on {failed}")


def _built_for() -> bytes:
    """What the module has in it: the header's ABI version and the torch that it was built against."""
    import torch
    with open(C_ABI) as f: abi = re.search(r"#define GAAC_ABI_VERSION (\d+)", f.read())[1]
    return f"ABI {abi}, torch {torch.__version__}".encode()


def _host_stale() -> bool:
    if _stale(HOST, [os.path.join(CSRC, "gaac_host.cpp"), C_ABI]):
        return True
    with open(HOST, "rb") as f: return _built_for() not in f.read()


def _start_host(force: bool):
    """The module's compiler at work, or nothing: up to date, or there is no torch or no C++ compiler here.  The library, which callers of the C ABI need alone, does without either."""
    try:
        if not force and not _host_stale():
            return []
        return [_start("gaac_host.cpp", _host_command())]
    except (ImportError, FileNotFoundError) as e:
        print(f"{os.path.basename(HOST)}, through which the Python package calls the library, is not built: {e}", file=sys.stderr)
        return []


def build(force: bool = False, verbose: bool = False) -> str:
    host = _start_host(force)
    if force or _stale(LIB, [*_sources(), *_headers()]):
        nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
        objs = [os.path.join("/tmp", "gaac_b200_" + os.path.basename(src) + ".o") for src in _sources()]
        _finish([_start(src, [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]) for src, obj in zip(_sources(), objs)], verbose)
        subprocess.check_call([nvcc, "-shared", "-o", LIB, *objs, "-lcudart"])
    _finish(host, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
