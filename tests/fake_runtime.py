"""The library's host code on a CUDA runtime of host memory (native/fake_cudart.cpp): its objects
linked with that runtime, loaded through the package's own bindings."""
import contextlib
import ctypes as C
import glob
import os
import shutil
import subprocess

import pytest

from pxdock_gb300 import build, native

HERE = os.path.dirname(os.path.abspath(__file__))


class Fake:
    def __init__(self, lib):
        self.lib = lib
        for name in ("fake_peak", "fake_largest"):
            getattr(lib, name).restype = C.c_size_t
        lib.fake_mallocs.restype = C.c_long
        lib.fake_fail_at.argtypes = [C.c_long]
        lib.fake_violations.restype = lib.fake_launch.restype = C.c_char_p
        lib.fake_launch.argtypes = [C.c_int, C.POINTER(C.c_uint)]

    def reset(self):
        self.lib.fake_reset()

    @property
    def violations(self):
        return self.lib.fake_violations().decode()

    def launches(self):
        """[(kernel, (grid x, y, z))] since the last reset."""
        g, out = (C.c_uint * 3)(), []
        for k in range(self.lib.fake_n_launches()):
            name = self.lib.fake_launch(k, g).decode()
            out.append((name, tuple(g)))
        return out


@contextlib.contextmanager
def loaded(folder):
    """The package bound to the fake; the real binding is back afterwards."""
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    build.build()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc())))
    out = os.path.join(str(folder), "libfake.so")
    objs = sorted(glob.glob(os.path.join(build.OUT_DIR, "*.o")))
    objs = [o for o in objs if any(os.path.splitext(os.path.basename(s))[0] + ".o" == os.path.basename(o)
                                   for s in build.sources())]
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", "-O1", "-Wl,-Bsymbolic", "-I", os.path.join(cuda, "include"),
                    os.path.join(HERE, "native", "fake_cudart.cpp")] + objs + ["-o", out, "-ldl"], check=True)
    saved, path = native._lib, build.lib_path
    native._lib, build.lib_path = None, lambda: out
    try:
        yield Fake(native.load())
    finally:
        native._lib, build.lib_path = saved, path
