"""Build libgemq_b200.so from the CUDA sources in this directory with nvcc (sm_100a only), and the
host-side call module _host.so from host.cpp with g++ against torch's headers.

    python -m gemq_b200.csrc.build [--verbose]

Both land next to the Python package (gemq_b200/).  They are
rebuilt only when a source or header is newer than the library, _host.so also when torch is another one.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
ROOT = os.path.dirname(PKG)
LIB = os.path.join(PKG, "libgemq_b200.so")
HOST_LIB = os.path.join(PKG, "_host.so")
SOURCES = ["pack.cu", "tma.cu", "gemv.cu", "gemv_stream.cu", "route.cu", "layer.cu", "decode_fused.cu", "gemm_ts.cu", "prefill.cu", "expert_parallel.cu", "no_alloc.cu",
           "few_linear.cu", "few_moe.cu", "few_one.cu", "decoder.cu"]
HEADERS = ["common.cuh", "gemv.cuh", "few_rows.cuh", "few_table.cuh", "gemm_ts.cuh", "ptx.cuh", os.path.join(ROOT, "include", "gemq_b200.h")]
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; gemq_b200 has no CPU fallback and cannot be built without it")
    return nvcc


# the torch that _host.so was built against: its C++ interface changes with the version
HOST_STAMP = os.path.join(HERE, "build", "host.torch")


def torch_build() -> str:
    import torch
    return f"{torch.__version__} {torch.version.git_version} {sys.version_info[:2]}"


def host_stale() -> bool:
    if not os.path.exists(HOST_LIB) or not os.path.exists(HOST_STAMP):
        return True
    with open(HOST_STAMP) as f:
        if f.read() != torch_build():
            return True
    t = os.path.getmtime(HOST_LIB)
    return any(os.path.getmtime(d) > t for d in (os.path.join(HERE, "host.cpp"), HEADERS[-1], os.path.abspath(__file__)))


def build_host() -> None:
    """g++ host.cpp against the headers of the installed torch; its library is found next to it."""
    import sysconfig
    import torch
    from torch.utils.cpp_extension import include_paths
    inc = [f"-I{p}" for p in include_paths()] + [f"-I{sysconfig.get_paths()['include']}"]
    cuda = os.path.join(os.path.dirname(os.path.dirname(find_nvcc())), "include")
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                           *inc, f"-I{cuda}", os.path.join(HERE, "host.cpp"), "-o", HOST_LIB, f"-L{libs}", "-ltorch_python",
                           "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-L{PKG}", "-l:libgemq_b200.so", "-Wl,-rpath,$ORIGIN"])
    os.makedirs(os.path.dirname(HOST_STAMP), exist_ok=True)
    with open(HOST_STAMP, "w") as f:
        f.write(torch_build())


def is_stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(HERE, s) for s in SOURCES] + [h if os.path.isabs(h) else os.path.join(HERE, h) for h in HEADERS]
    deps.append(os.path.abspath(__file__))
    return any(os.path.getmtime(d) > t for d in deps)


def build(verbose: bool = False, force: bool = False) -> str:
    if not force and not is_stale():
        if host_stale():
            build_host()
        return LIB
    nvcc = find_nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    common = [nvcc, "-O3", "-std=c++17", "-lineinfo", *ARCH_FLAGS,
              "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include")]
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    objs = []
    for s in SOURCES:
        obj = os.path.join(objdir, s.replace(".cu", ".o"))
        objs.append(obj)
        procs.append((s, subprocess.Popen(common + ["-c", os.path.join(HERE, s), "-o", obj],
                                          stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for s, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {s} ---\n{out}\n")
        failed = failed or p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call([nvcc, "-shared", *ARCH_FLAGS, "-o", LIB, *objs, "-lcudart"])
    if force or host_stale():
        build_host()
    return LIB


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
