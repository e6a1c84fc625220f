"""Builds libfa_b200.so (the C-ABI library, nvcc for sm_100a) and _call.<ABI>.so (its call path on torch tensors) in-tree.

    python -m flash_attn_b200.build [--force] [--verbose]

The library is rebuilt only when a source is newer than the binary.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libfa_b200.so")
SOURCES = ["fa_api.cu", "fa_fwd_tiled.cu", "fa_decode.cu", "fa_aux.cu", "fa_static_scratch.cu", "fa_ring.cu"]
HEADERS = ["fa_internal.h", "sm100_ptx.cuh", "philox.cuh", os.path.join("..", "..", "include", "fa_b200.h")]
# units of compilation (source, object, flags), longest first: the tiled kernels once for each head dimension and number of query
# tiles a CTA (in one unit they take ptxas two minutes)
UNITS = [("fa_fwd_tiled.cu", f"fa_fwd_tiled_{d}_{nq}.o", [f"-DFA_TILED_D={d}", f"-DFA_TILED_NQ={nq}"])
         for d, nq in ((128, 2), (64, 2), (128, 1), (64, 1))]
UNITS += [(f, f.replace(".cu", ".o"), []) for f in SOURCES if f != "fa_fwd_tiled.cu"]


def nvcc_path():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA library cannot be built")


def needs_build(lib=LIB):
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in SOURCES + HEADERS)


def _compile(lib, build_dir, flags, verbose=False):
    os.makedirs(build_dir, exist_ok=True)
    common = [nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--compress-mode=size", "-Xcompiler", "-fPIC", "-Xptxas", "-v" if verbose else "-warn-spills"] + flags
    objs, procs = [], []
    for src, obj, defines in UNITS:
        objs.append(os.path.join(build_dir, obj))
        procs.append((src, subprocess.Popen(common + defines + ["-c", os.path.join(CSRC, src), "-o", objs[-1]],
                                            stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = []
    for src, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stderr.write(out)
        if pr.returncode != 0:
            failed.append(src)
    if failed:
        raise RuntimeError(f"nvcc failed on {', '.join(failed)}")
    subprocess.check_call([nvcc_path(), "-shared", "-o", lib + ".new"] + objs + ["-Xcompiler", "-fPIC", "-ldl"])
    os.replace(lib + ".new", lib)


# The call path is C++ against this Python and this torch: the file's name carries the one's ABI tag, and what it was built
# from (torch's version and the compiler's arguments) is kept beside the objects and in the module (_call.built_for).
CALL = os.path.join(PKG, "_call" + sysconfig.get_config_var("EXT_SUFFIX"))
CALL_SOURCE = os.path.join(CSRC, "fa_torch.cpp")


def _call_command():
    import torch
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc_path()))
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", f'-DFA_BUILT_FOR="{torch.__version__}"',
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-isystem", os.path.join(tdir, "include"), "-isystem", os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
            "-isystem", sysconfig.get_paths()["include"], "-isystem", os.path.join(cuda, "include"), CALL_SOURCE,
            "-L", os.path.join(tdir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]


def needs_build_call():
    stamp = os.path.join(PKG, "build", os.path.basename(CALL) + ".txt")
    if not os.path.exists(CALL) or not os.path.exists(stamp):
        return True
    newest = max(os.path.getmtime(CALL_SOURCE), os.path.getmtime(os.path.join(PKG, "..", "include", "fa_b200.h")))
    with open(stamp) as f:
        return os.path.getmtime(CALL) < newest or f.read() != "\n".join(_call_command())


def build_call(force=False):
    """Builds the module of csrc/fa_torch.cpp (flash_attn_forward on torch tensors) against the installed torch."""
    if force or needs_build_call():
        os.makedirs(os.path.join(PKG, "build"), exist_ok=True)
        command = _call_command()
        subprocess.check_call(command + ["-o", CALL + ".new"])
        os.replace(CALL + ".new", CALL)
        with open(os.path.join(PKG, "build", os.path.basename(CALL) + ".txt"), "w") as f:
            f.write("\n".join(command))
    return CALL


def build(force=False, verbose=False):
    """The library first: it and the C callers need neither torch nor Python."""
    if force or needs_build():
        _compile(LIB, os.path.join(PKG, "build"), [], verbose)
    build_call(force)
    return LIB


TEST_LIB = os.path.join(PKG, "libfa_b200_shortwait.so")


def build_test_variant(force=False):
    """Builds libfa_b200_shortwait.so, the library compiled with -DFA_TEST_SHORT_WAIT: bounded waits give
    up after about 2 ms and the producer of the tiled kernel can be told to leave KV tiles out
    (fa_test_skip_kv_tile).  Used only by the GPU test of the give-up path."""
    if force or needs_build(TEST_LIB):
        _compile(TEST_LIB, os.path.join(PKG, "build", "shortwait"), ["-DFA_TEST_SHORT_WAIT"])
    return TEST_LIB


BENCH = os.path.join(PKG, "fa_bench")


def build_driver(force=False):
    """Builds the C benchmark driver (csrc/fa_main.c) against the library with gcc."""
    src = os.path.join(CSRC, "fa_main.c")
    build()
    if not force and os.path.exists(BENCH) and os.path.getmtime(BENCH) > max(os.path.getmtime(src), os.path.getmtime(LIB)):
        return BENCH
    cuda = os.path.dirname(os.path.dirname(nvcc_path()))
    cc = "/usr/bin/gcc" if os.path.exists("/usr/bin/gcc") else "gcc"
    subprocess.check_call([cc, "-std=c99", "-O2", "-Wall", "-I", os.path.join(PKG, "..", "include"),
                           "-I", os.path.join(cuda, "include"), src, "-o", BENCH,
                           "-L", PKG, "-lfa_b200", "-L", os.path.join(cuda, "lib64"), "-lcudart", "-lm", "-lpthread",
                           "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + os.path.join(cuda, "lib64")])
    return BENCH


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(LIB)
    print(build_driver(force="--force" in sys.argv))
    print(build_test_variant(force="--force" in sys.argv))
