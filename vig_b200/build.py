"""Build ``libvig_b200.so`` (kernels, nvcc for sm_100a) and the package's C++ host module ``_host`` in-tree.
Run as ``python -m vig_b200.build``."""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libvig_b200.so")
HOST = os.path.join(HERE, "_host.so")
HOST_SOURCES = ["host_ops.cpp", "host_model.cpp"]
SOURCES = ["abi.cu", "bigla_simt.cu", "bigla_tc.cu", "bigla_wave.cu", "elementwise.cu", "noalloc.cu", "bigla_bwd_simt.cu", "bigla_bwd_mma.cu", "bigla_seg.cu", "block_tail.cu", "conv_proj.cu", "embed_conv.cu", "gemm_swiglu.cu", "gemm_pair.cu", "gemm_pair_norm.cu", "gemm_addnorm.cu", "dwconv_tma.cu", "gemm_bias.cu", "gemm_stem.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def needs_build():
    header = [os.path.join(HERE, "..", "include", "vig_b200.h")]
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    return (_stale(LIB, [f for f in files if f.endswith((".cu", ".cuh"))] + header),
            _stale(HOST, [f for f in files if f.endswith((".cpp", ".h"))] + header))


def _run_all(cmds, verbose):
    procs = [(cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for cmd in cmds]
    for cmd, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode:
            sys.stderr.write(out)
        if pr.returncode:
            raise RuntimeError(f"failed: {' '.join(cmd)}")


def build(force=False, verbose=False):
    lib, host = (True, True) if force else needs_build()
    out = os.path.join(HERE, "build")
    os.makedirs(out, exist_ok=True)
    cmds, obj = [], lambda src: os.path.join(out, os.path.splitext(src)[0] + ".o")
    if lib:
        cmds += [[_nvcc(), *(["-Xptxas=-v"] if verbose else []), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj(src)] for src in SOURCES]
    if host:
        import torch
        base = os.path.dirname(torch.__file__)
        inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], "/usr/local/cuda/include"]
        flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
                 f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
        cmds += [["g++", *flags, *[f"-I{i}" for i in inc], "-c", os.path.join(CSRC, src), "-o", obj(src)] for src in HOST_SOURCES]
    _run_all(cmds, verbose)
    if lib:
        subprocess.check_call([_nvcc(), "-shared", "-o", LIB, *[obj(s) for s in SOURCES], "-lcudart_static", "-ldl", "-lrt", "-lpthread"])
    if host:
        libs = os.path.join(base, "lib")
        subprocess.check_call(["g++", "-shared", "-o", HOST, *[obj(s) for s in HOST_SOURCES], f"-L{libs}", f"-Wl,-rpath,{libs}", "-ltorch_python",
                               "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ldl"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
