"""Builds libflamia_b200.so (the C-ABI shared library, nvcc for sm_100a) and _host.so (the native host path over it: torch ops and
autograd, g++) in-tree.

    python -m flamia_blackwell_attention_b200.build [--verbose]

nvcc cross-compiles without a GPU; the library itself only needs a device when an entry point is called.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libflamia_b200.so")
HOST = os.path.join(HERE, "_host.so")
SOURCES = ["abi.cu", "quant.cu", "selftest.cu", "fwd.cu", "bwd.cu", "side.cu", "noalloc.cu"]
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-O2", "--expt-relaxed-constexpr"]
# the attention kernels may flush denormals and use approximate division; the quantisers and the scalar / post kernels
# must not (their outputs are compared byte for byte)
FAST_MATH = {"fwd.cu", "bwd.cu"}


def _stale(obj, srcs):
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(s) > t for s in srcs)


def _host_flags():
    """Compile and link arguments of csrc/host.cpp against the installed torch and the C-ABI library beside it."""
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_path("include")]
    comp = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[x for i in inc for x in ("-isystem", i)]]
    link = ["-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
            "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-L" + HERE, "-l:libflamia_b200.so", "-Wl,-rpath,$ORIGIN"]
    return comp, link


def build(verbose=False, force=False):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "flamia_b200.h"))
    objs = []
    procs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        if not os.path.exists(s):
            continue
        o = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc, *FLAGS, "-c", s, "-o", o] + (["-Xptxas", "-v"] if verbose else [])
            if src in FAST_MATH:
                cmd.append("--use_fast_math")
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    # the system's compiler, not $CXX: PyTorch's C++ objects cross this module's boundary, so it must use the shared C++ runtime
    # that torch has loaded (a compiler that links its own one statically gives a module that crashes in the first stream)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    host_src, host_obj = os.path.join(CSRC, "host.cpp"), os.path.join(CSRC, "host.o")
    if force or _stale(host_obj, [host_src, headers[-1]]):
        procs.append(("host.cpp", subprocess.Popen([cxx, *_host_flags()[0], "-c", host_src, "-o", host_obj], stdout=subprocess.PIPE,
                                                   stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(f"---- {src}\n{out}")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc or g++ failed")
    if force or _stale(LIB, objs):
        subprocess.check_call([nvcc, "-shared", "-o", LIB, *objs, "-Xcompiler", "-fPIC",
                               "-gencode", "arch=compute_100a,code=sm_100a"])
    if force or _stale(HOST, [host_obj]):
        subprocess.check_call([cxx, "-shared", host_obj, "-o", HOST, *_host_flags()[1]])
    return LIB


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
