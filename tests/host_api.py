"""The library's host side without a GPU: its objects linked against
fake_cudart.cpp, where device memory is host memory and kernels are recorded
instead of run."""
import ctypes
import importlib.util
import os
import subprocess

from conftest import PKG_DIR

HERE = os.path.dirname(os.path.abspath(__file__))


def _module(name, path):
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


class HostApi:
    """`ib`: the binding over the fake runtime."""

    def __init__(self, workdir):
        bl = _module("host_api_build", os.path.join(PKG_DIR, "build_lib.py"))
        bl.build()
        objs = [os.path.join(bl.OBJ, u.replace(".cu", ".o")) for u in bl.UNITS]
        if not all(os.path.exists(o) for o in objs):
            bl.build(force=True)
        fake, path = os.path.join(workdir, "fake.o"), os.path.join(workdir, "libibgpu_host.so")
        include = os.path.join(os.path.dirname(os.path.dirname(bl.nvcc())), "include")
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-I", include, "-c",
                               os.path.join(HERE, "fake_cudart.cpp"), "-o", fake])
        subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", path, *objs, fake])
        self.ib = _module("host_api_ibgpu", os.path.join(PKG_DIR, "ibgpu.py"))
        self.L = self.ib.lib(path)
        self.L.fake_name.restype = ctypes.c_char_p

    def clear(self):
        self.L.fake_clear()

    def fail_malloc(self, nth):
        """The nth allocation from now fails (0: none)."""
        self.L.fake_fail_malloc(nth)

    def launches(self, part):
        """(kernel name, grid, words of the first argument) of every launch
        since clear() whose kernel's name contains `part`."""
        out = []
        for i in range(self.L.fake_launches()):
            name = self.L.fake_name(i).decode()
            if part in name:
                words = (ctypes.c_int64 * 20)()
                self.L.fake_arg(i, words)
                out.append((name, self.L.fake_grid(i), list(words)))
        return out

    def live(self, ptr):
        return bool(self.L.fake_live(ctypes.c_void_p(ptr)))


def words(ptr, n, at=0):
    """n 64-bit words of (fake) device memory."""
    return list((ctypes.c_int64 * n).from_address(ptr + at))
