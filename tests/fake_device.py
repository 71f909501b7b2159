"""The library's host side without a device: its object files linked with the
runtime of fake_cudart.cpp, in which kernels do nothing."""
import ctypes
import glob
import os
import subprocess

import build as pkg_build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(where):
    """The fake library, built in the folder `where`."""
    pattern = os.path.join(pkg_build.OBJDIR, "*.o")
    pkg_build.build(force=not glob.glob(pattern))
    objs = sorted(glob.glob(pattern))
    out = os.path.join(str(where), "libmauve_fake.so")
    include = os.path.join(os.path.dirname(os.path.dirname(pkg_build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + include, "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-lpthread"], check=True)
    lib = ctypes.CDLL(out)
    for name in ("fake_refused", "fake_largest"):
        getattr(lib, name).restype = ctypes.c_size_t
    lib.fake_reset.argtypes = [ctypes.c_size_t]
    lib.fake_reply.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    lib.fake_fail_at.argtypes = [ctypes.c_long]
    lib.fake_no_memory_at.argtypes = [ctypes.c_long]
    for name in ("fake_launches", "fake_allocations"):
        getattr(lib, name).restype = ctypes.c_long
    lib.mvg_last_error.restype = ctypes.c_char_p
    lib.mvg_get_seed.restype = ctypes.c_uint64
    return lib
