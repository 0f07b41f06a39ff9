"""The library's host side on a CUDA runtime that lives on the host
(fake_cuda.cu): build() links it with the library's objects, lib() is a ctypes
handle with the binding's signatures, which a test puts in the place of
cgfd._lib.  Nothing runs on a GPU, and no kernel runs at all: the calls, their
arguments, work lists, errors and allocations are what such tests see."""
import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np

import cgfd

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(cgfd.LIB_PATH)
GEN_VEL, GEN_STR, LEAN = 0, 1, 2  # the paired kernels' launches


def build(out_dir):
    """Path of the linked library, or None without nvcc and g++."""
    if shutil.which("nvcc") is None or shutil.which("g++") is None:
        return None
    subprocess.run(["make", "-s", "-C", PKG, "-j8"], check=True)
    obj, lib = os.path.join(out_dir, "paired_work.o"), os.path.join(out_dir, "libcgfd_fake.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-c",
                    os.path.join(HERE, "paired_work.cu"), "-o", obj], check=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc"))), "include")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-g", "-std=c++17", "-I" + cuda,
                    "-Wl,-Bsymbolic", "-Wl,--no-undefined", os.path.join(HERE, "fake_cuda.cpp"),
                    obj, *glob.glob(os.path.join(PKG, "_build", "*.o")), "-lpthread", "-o", lib],
                   check=True)
    return lib


def lib(path):
    h = C.CDLL(path)
    for name, (res, args) in cgfd._SIGS.items():
        f = getattr(h, name)
        f.restype, f.argtypes = res, args
    h.fake_fail.argtypes = [C.c_char_p, C.c_int, C.c_int]
    return h


def items(h, q):
    """The items of launch q, rows of i0, j0, z0, z1, model, part."""
    v = np.zeros((h.fake_items(q), 6), np.int32)
    h.fake_get_items(q, v.ctypes.data_as(C.POINTER(C.c_int)))
    return v
