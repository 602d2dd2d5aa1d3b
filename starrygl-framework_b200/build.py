"""Build libsgl_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and _sgl_host.*.so (the Python side of its hot calls)
with g++ against the installed torch, whose version its name carries: another torch has another binary interface and gets a module of its own.

    python starrygl-framework_b200/build.py [--force] [--verbose]

The shared object lands in starrygl-framework_b200/lib/.  nvcc cross-compiles, so no GPU is needed.
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "lib")
OUT = os.path.join(OUT_DIR, "libsgl_b200.so")
SOURCES = ["api.cu", "sort.cu", "tcsr.cu", "sampler.cu", "relabel.cu", "gather.cu", "comm.cu", "p2p_route.cu", "plan.cu", "mail.cu", "slice.cu", "batch.cu", "launch.cu", "query.cu"]
FLAGS = ["-O3", "--threads", "0", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "--expt-relaxed-constexpr",
         "-Xcompiler", "-fPIC", "-shared", "-cudart", "shared"]


def host_path():
    import torch
    return os.path.join(OUT_DIR, f"_sgl_host.{torch.__version__}.{sys.implementation.cache_tag}.so")


def _stale(out, deps):
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in (*deps, os.path.join(HERE, "..", "include", "sgl_b200.h"), __file__))


def _run(cmd, what, verbose):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"building {what} failed")


def build(force=False, verbose=False):
    os.makedirs(OUT_DIR, exist_ok=True)
    kernels = [os.path.join(SRC, f) for f in os.listdir(SRC) if f.endswith((".cu", ".cuh"))]
    if force or _stale(OUT, kernels):
        nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
        _run([nvcc] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + [os.path.join(SRC, s) for s in SOURCES] + ["-ldl", "-o", OUT],
             "libsgl_b200.so", verbose)
    host, out = os.path.join(SRC, "host.cpp"), host_path()
    if force or _stale(out, [host]):
        import torch
        at = os.path.dirname(torch.__file__)
        inc = [os.path.join(at, "include"), os.path.join(at, "include", "torch", "csrc", "api", "include"), "/usr/local/cuda/include"]
        _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
              f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[x for i in inc for x in ("-isystem", i)],
              "-I", sysconfig.get_paths()["include"], host, "-o", out, "-L", OUT_DIR, "-lsgl_b200", "-L", os.path.join(at, "lib"),
              "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"], os.path.basename(out), verbose)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
