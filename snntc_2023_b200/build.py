"""Builds the CUDA libraries (sm_100a only) in-tree with nvcc.

    python -m snntc_2023_b200.build [--force] [-v]

Two shared libraries come out of the same sources:
    libsnntc_b200.so          the product: the C ABI declared in include/snntc_b200.h
    libsnntc_b200_measure.so  the same compiled with -DSNNTC_MEASURE: it adds the entry points that take the
                              kernel choice of a call explicitly (bench.py times the kernels of an operator
                              apart with them, the tests check kernel variants against each other)
Both are plain CUDA runtime code behind a C ABI and link the CUDA runtime statically, so the only requirement
at load time is an NVIDIA driver. A third, the CPython extension `_native` (csrc/snntc_torch.cpp), is the host path of
the Python operators: it links torch and the product library beside it.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libsnntc_b200.so")
LIB_MEASURE = os.path.join(HERE, "libsnntc_b200_measure.so")
SOURCES = ["snntc_forward.cu", "snntc_sort.cu", "snntc_walk_ring.cu", "snntc_walk_alone.cu", "snntc_walk_rows.cu",
           "snntc_lists.cu", "snntc_backward.cu", "snntc_bwd_dense.cu",
           "snntc_dw_skip.cu", "snntc_dw_tma.cu", "snntc_dx_sparse.cu", "snntc_dx_few.cu",
           "snntc_pool.cu",
           "snntc_noalloc.cu", "snntc_train.cu", "snntc_api.cu"]
NATIVE = os.path.join(HERE, "_native" + sysconfig.get_config_var("EXT_SUFFIX"))
NATIVE_SOURCE = os.path.join(CSRC, "snntc_torch.cpp")
API_SOURCE = "snntc_api.cu"   # the only file that reads SNNTC_MEASURE
HEADERS = [os.path.join(CSRC, "snntc_common.cuh"), os.path.join(CSRC, "snntc_bound.cuh"), os.path.join(CSRC, "snntc_merge.cuh"), os.path.join(CSRC, "snntc_walk.cuh"),
           os.path.join(CSRC, "snntc_launch.cuh"), os.path.join(CSRC, "snntc_ptx.cuh"),
           os.path.join(HERE, "..", "include", "snntc_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libsnntc_b200.so cannot be built")


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES]


def up_to_date():
    if not all(os.path.exists(p) for p in (LIB, LIB_MEASURE, NATIVE)):
        return False
    t = min(os.path.getmtime(p) for p in (LIB, LIB_MEASURE, NATIVE))
    return all(os.path.getmtime(p) <= t for p in sources() + HEADERS + [NATIVE_SOURCE])


def _native_compile(obj):
    from torch.utils import cpp_extension
    import torch
    include = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], "/usr/local/cuda/include"]
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wno-attributes",
             "-DTORCH_EXTENSION_NAME=_native", "-DTORCH_API_INCLUDE_EXTENSION_H",
             "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)] +
            ["-isystem" + p for p in include] + ["-c", NATIVE_SOURCE, "-o", obj])


def _native_link(obj):
    """The product library is found beside the extension; torch's libraries are in the process already (the package
    imports torch first)."""
    from torch.utils import cpp_extension
    return ["g++", "-shared", obj, "-o", NATIVE, "-L" + HERE, "-l:libsnntc_b200.so", "-Wl,-rpath,$ORIGIN",
            "-L" + cpp_extension.library_paths()[0], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch",
            "-ltorch_python"]


def build(force=False, verbose=False):
    if not force and up_to_date():
        return LIB
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    newest_header = max(os.path.getmtime(p) for p in HEADERS)
    procs = []

    def start(cmd, out, src):
        """Runs cmd beside the others unless `out` is newer than its source and the headers."""
        if force or not os.path.exists(out) or os.path.getmtime(out) < max(os.path.getmtime(src), newest_header):
            procs.append((cmd, subprocess.Popen(cmd)))

    objs = []
    extra = ["-Xptxas", "-v"] if verbose else []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        start([nvcc] + NVCC_FLAGS + extra + ["-c", src, "-o", obj], obj, src)
        objs.append(obj)
    api = os.path.join(CSRC, API_SOURCE)
    api_measure = os.path.join(objdir, "snntc_api_measure.o")
    start([nvcc] + NVCC_FLAGS + ["-DSNNTC_MEASURE", "-c", api, "-o", api_measure], api_measure, api)
    native_obj = os.path.join(objdir, "snntc_torch.o")
    start(_native_compile(native_obj), native_obj, NATIVE_SOURCE)
    for cmd, p in procs:
        if p.wait() != 0:
            raise RuntimeError("compiler failed: " + " ".join(cmd))
    subprocess.check_call([nvcc] + NVCC_FLAGS[:2] + ["-shared", "-o", LIB] + objs)
    api_obj = os.path.join(objdir, API_SOURCE[:-3] + ".o")
    subprocess.check_call([nvcc] + NVCC_FLAGS[:2] + ["-shared", "-o", LIB_MEASURE] +
                          [api_measure if o == api_obj else o for o in objs])
    subprocess.check_call(_native_link(native_obj))
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
