"""Builds libanode_routines_gpu.so in-tree with plain nvcc (sm_100a only), and _native.so, the Python side of the hot
entry points, with the host compiler.

The flags follow the reference's own recipe where they matter for numerics
(build.rs:47-48: -prec-div=true -prec-sqrt=true); the architecture list is replaced by the
single sm_100a target.  Usage: `python -m anode_b200.build [--force]`.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libanode_routines_gpu.so")
NATIVE = os.path.join(HERE, "_native.so")
NATIVE_SOURCE = os.path.join(CSRC, "bn_py.cpp")
SOURCES = ["bn_fused.cu", "bn_legacy.cu", "bn_compose.cu", "bn_sync.cu", "bn_static.cu", "bn_hoststep.cu", "bn_segres.cu", "bn_chan.cu", "bn_stream.cu", "bn_long.cu", "bn_band.cu", "bn_infer.cu", "bn_resident.cu", "bn_resident_diag.cpp"]
HEADERS = ["bn_plan.h", "bn_device.cuh", "bn_fused.cuh", "bn_ring.cuh", "bn_pipe.cuh", "bn_band.cuh", "bn_resident_plan.h", "bn_host.h", "bn_sync.h",
           os.path.join("..", "..", "include", "anode_routines_gpu.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-prec-div=true", "-prec-sqrt=true",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fno-strict-aliasing",
]


def _sources():
    return [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _nccl_include():
    """nccl.h is only needed for types; the library itself is resolved at run time."""
    try:
        import nvidia.nccl as n
        inc = os.path.join(list(n.__path__)[0], "include")
        if os.path.exists(os.path.join(inc, "nccl.h")):
            return inc
    except Exception:
        pass
    return "/usr/include"


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in _sources()] + [os.path.join(CSRC, h) for h in HEADERS]
    return any(os.path.exists(d) and os.path.getmtime(d) > t for d in deps)


def native_built_for():
    """What a build of the native module is bound to: this interpreter's ABI and this torch."""
    import sysconfig
    import torch
    return "built for %s, torch %s" % (sysconfig.get_config_var("SOABI"), torch.__version__)


def native_is_current(path, source, built_for):
    """Whether the module at `path` is newer than its source and this file, and was built for `built_for` (the text is
    compiled into it)."""
    if not os.path.exists(path) or any(os.path.getmtime(path) <= os.path.getmtime(f) for f in (source, os.path.abspath(__file__))):
        return False
    with open(path, "rb") as f:
        return built_for.encode() + b"\0" in f.read()


def build_native(force=False):
    """The CPython module anode_b200._native: compiled against this interpreter's and torch's headers, linked against
    torch only (the C ABI is handed to it as addresses at run time).  Built again after a change of either."""
    import sysconfig
    import torch
    built_for = native_built_for()
    if not force and native_is_current(NATIVE, NATIVE_SOURCE, built_for):
        return NATIVE
    root = os.path.dirname(torch.__file__)
    tmp = NATIVE + ".tmp%d" % os.getpid()
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI), '-DANODE_BUILT_FOR="%s"' % built_for,
           "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I", os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), "-I", sysconfig.get_paths()["include"],
           NATIVE_SOURCE, "-o", tmp, "-L", os.path.join(root, "lib"),
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    subprocess.check_call(cmd)
    os.replace(tmp, NATIVE)
    return NATIVE


def build_library(force=False, verbose=False):
    build_native(force)
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    objs = []
    procs = []
    for s in _sources():
        obj = os.path.join(CSRC, os.path.splitext(s)[0] + ".o")
        cmd = [nvcc] + NVCC_FLAGS + ["-I", _nccl_include(), "-c", os.path.join(CSRC, s), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for s, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError("nvcc failed on %s" % s)
    # the CUDA runtime is linked statically (nvcc's default); NCCL is looked up with dlopen
    # link to a temporary name and rename: a reader (or a copy of the tree) never sees a half-written library
    tmp = LIB + ".tmp%d" % os.getpid()
    link = [nvcc, "-shared", "-o", tmp] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-Xlinker", "-Bsymbolic", "-ldl"]
    subprocess.check_call(link)
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
