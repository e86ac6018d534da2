"""Builds libfmha_i8_sm100.so in-tree with nvcc for sm_100a (cross-compiles without a GPU) and the native Python
binding of its calls, _fmha_i8_py.so, with the host compiler.

    python build.py [--force] [--verbose]
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libfmha_i8_sm100.so")
BINDING = os.path.join(HERE, "_fmha_i8_py.so")
BINDING_SOURCE = os.path.join(CSRC, "py_binding.cpp")
SOURCES = ["fmha_api.cu"]
HEADERS = ["ptx.cuh", "fmha_fwd_sm100.cuh", "fmha_debug_sm100.cuh", "fmha_quant_sm100.cuh", "fmha_decode_sm100.cuh", "fmha_fwd64_sm100.cuh", "fmha_policy_sm100.cuh", "fmha_host_sm100.cuh",
           os.path.join("..", "..", "include", "fmha_i8_c.h"),
           os.path.join("..", "..", "include", "fmha_i8.h"),
           os.path.join("..", "..", "include", "fmha_param_i8.h")]


def nvcc_path():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def up_to_date(target=LIB, sources=None):
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    for p in sources or [os.path.join(CSRC, f) for f in SOURCES + HEADERS]:
        if os.path.exists(p) and os.path.getmtime(p) > t:
            return False
    return True


def build_binding(force=False):
    if not force and up_to_date(BINDING, [BINDING_SOURCE, os.path.join(CSRC, "..", "..", "include", "fmha_i8_c.h"), LIB]):
        return BINDING
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", "-Wall",
                           "-I" + sysconfig.get_paths()["include"], BINDING_SOURCE, "-o", BINDING,
                           "-L" + HERE, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN"])
    return BINDING


def build(force=False, verbose=False):
    if not force and up_to_date():
        build_binding()
        return LIB
    cmd = [nvcc_path(), "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
           "-Xcompiler", "-fPIC", "-shared", "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    subprocess.check_call(cmd)
    build_binding(force=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
