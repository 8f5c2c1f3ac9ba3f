"""Builds libsortnet_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _ops.so, the PyTorch
module of csrc/ops_ext.cpp, with the host compiler.

    python -m sortnet_b200.build [--force]

Every .cu under csrc/ is compiled to an object file (in parallel, skipped when newer than
its sources) and linked into sortnet_b200/libsortnet_b200.so with the CUDA runtime linked
statically, so the library depends on nothing but the driver.
"""
import concurrent.futures
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libsortnet_b200.so")
OPS = os.path.join(HERE, "_ops.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC", "-I", os.path.join(os.path.dirname(HERE), "include"),
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _newest_header():
    hs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(os.path.dirname(HERE), "include", "*.h"))
    return max([os.path.getmtime(h) for h in hs] + [0.0])


def _compile(src, obj, verbose):
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, r.stdout, r.stderr))
    return r.stderr


def build_ops(force: bool = False) -> str:
    """The native operator layer: one C++ file against PyTorch's headers, no CUDA code."""
    import sysconfig
    import torch
    src = os.path.join(CSRC, "ops_ext.cpp")
    newest = max(os.path.getmtime(src), _newest_header())
    stamp = os.path.join(OBJ, "ops_built_for")               # the module is bound to one PyTorch and one Python
    target = "%s %s %s" % (torch.__version__, sysconfig.get_config_var("SOABI"), torch._C._GLIBCXX_USE_CXX11_ABI)
    built_for = open(stamp).read() if os.path.exists(stamp) else ""
    if not force and os.path.exists(OPS) and os.path.getmtime(OPS) >= newest and built_for == target:
        return OPS
    base = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_ops", "-DTORCH_API_INCLUDE_EXTENSION_H",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
    for inc in (os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]):
        cmd += ["-isystem", inc]
    lib = os.path.join(base, "lib")
    cmd += [src, "-o", OPS, "-L" + lib, "-Wl,-rpath," + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for %s:\n%s" % (src, r.stderr))
    os.makedirs(OBJ, exist_ok=True)
    with open(stamp, "w") as f:
        f.write(target)
    return OPS


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    ops_job = concurrent.futures.ThreadPoolExecutor(max_workers=1).submit(build_ops, force)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdr = _newest_header()
    jobs, objs = [], []
    for s in srcs:
        o = os.path.join(OBJ, os.path.basename(s)[:-3] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr):
            jobs.append((s, o))
    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for log in ex.map(lambda so: _compile(so[0], so[1], verbose), jobs):
                if verbose:
                    sys.stderr.write(log)
    if jobs or not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(o) for o in objs):
        cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs
        subprocess.check_call(cmd)
    ops_job.result()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
