"""The library with launches and allocations that fail on request (cpp/launch_faults.cpp): the objects of
the build linked once more, with some CUDA calls wrapped."""
import contextlib
import ctypes as C
import os
import subprocess

from scdat_b200 import build, capi

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(build.BUILD, "libscdat_faults.so")


def faulty_library():
    build.build()
    src = os.path.join(HERE, "cpp", "launch_faults.cpp")
    objs = [os.path.join(build.BUILD, s + ".o") for s in build.SOURCES]
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(map(os.path.getmtime, objs + [src])):
        subprocess.run([build.NVCC, *build.ARCH, "-shared", "-Xcompiler", "-fPIC", src, *objs, "-o", LIB, "-Xlinker",
                        "--wrap=cudaLaunchCooperativeKernel,--wrap=cudaMalloc,--wrap=cudaFree,--wrap=cudaMemGetInfo"], check=True)
    return LIB


@contextlib.contextmanager
def faults():
    """capi on that library; gives the ctypes handle."""
    kept = capi.LIB_PATH, capi._LIB
    capi.LIB_PATH, capi._LIB = faulty_library(), None
    try:
        lib = capi.load()
        lib.fault_budget.argtypes = [C.c_size_t]
        lib.fault_used.restype = C.c_size_t
        try:
            yield lib
        finally:
            lib.fault_launches(0, 0)
            lib.fault_budget(0)
    finally:
        capi.LIB_PATH, capi._LIB = kept
