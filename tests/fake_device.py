"""The engine's host code on a fake CUDA runtime (tests/fake/fake_cudart.cpp): what it launches for a call,
without a GPU.  Test infrastructure only."""
import contextlib
import ctypes
import glob
import os
import subprocess

import build
import cuckoo_b200 as cb
import helpers as h

SRC = os.path.join(h.ROOT, "tests", "fake", "fake_cudart.cpp")


def link(folder):
    """The engine's objects linked with the fake runtime, with cuckoo_b200's declarations."""
    build.build()
    so = os.path.join(str(folder), "libfake.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + cuda, SRC, "-o", so] +
                   sorted(glob.glob(os.path.join(build.BUILD, "*.cu.o"))), check=True)
    return so


@contextlib.contextmanager
def on(so):
    """cuckoo_b200 on the fake runtime: yields its library."""
    kept = cb._lib, cb.LIB_PATH
    cb._lib, cb.LIB_PATH = None, so
    try:
        yield cb.lib()
    finally:
        cb._lib, cb.LIB_PATH = kept


def launches(L):
    """[(device, grid, block, dynamic shared memory)] since the last call."""
    out, v = [], (ctypes.c_int * 4)()
    for i in range(L.fake_launches()):
        L.fake_launch(i, v)
        out.append(tuple(v))
    L.fake_clear()
    return out
