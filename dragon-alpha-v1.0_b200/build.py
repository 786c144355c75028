"""Builds libalpha_conv_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libalpha_conv_b200.so")
SOURCES = ["conv_api.cu", "native_api.cu", "matmul_api.cu", "pool_api.cu", "jni_shim.cpp"]
HEADERS = ["conv_kernels.cuh", "conv_halo.cuh", "conv_halo_pair.cuh", "conv_dw_halo.cuh", "winograd.cuh", "conv_tapstack.cuh", "sm100_ptx.cuh", "fast_div.cuh", "gemm_f32.cuh", "gemm_planes.cuh", "dependent_launch.cuh",
           "once_per_device.h", "host_common.h"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC"]


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    inc = os.path.join(HERE, "..", "include")
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS]
    deps += [os.path.join(inc, f) for f in os.listdir(inc)]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    """Compile the library if it is missing or older than its sources.  Returns its path."""
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    extra = os.environ.get("ALPHA_NVCC_EXTRA", "").split()   # e.g. -D switches for experiments
    cmd = [nvcc] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + SOURCES
    subprocess.check_call(cmd, cwd=CSRC)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))
