"""The library's host code over tests/cpp/fake_cudart.cpp: no GPU, no kernel
runs, calls are logged. For what only the host decides (which kernel reads a
buffer, what happens when a call fails, what is freed)."""
import ctypes
import os
import subprocess

from gpusharesat_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
vp, i64 = ctypes.c_void_p, ctypes.c_int64


class Fake:
    def __init__(self, folder):
        build.build()
        objs = [obj for _, obj, _ in build.compile_commands()]
        fake, self.path = str(folder / "fake_cudart.o"), str(folder / "libfake.so")
        subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-I", build._cuda_include(), "-c",
                        os.path.join(HERE, "cpp", "fake_cudart.cpp"), "-o", fake], check=True)
        # (the library's own symbols first: a process may hold the real one too)
        subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", self.path, *objs, fake, "-lpthread"], check=True)
        self.lib = ctypes.CDLL(self.path)
        self.lib.fake_log.restype = self.lib.gss_last_error.restype = ctypes.c_char_p
        self.lib.gss_engine_graph_captures.restype = self.lib.gss_engine_filtered_passes.restype = i64
        self.lib.gss_sharer_add_clause.restype = i64

    def log(self):
        return self.lib.fake_log().decode().splitlines()

    def reset(self):
        self.lib.fake_reset()

    def fail(self, what, after=0):
        self.lib.fake_fail(what.encode(), after)

    def error(self):
        return self.lib.gss_last_error().decode()

    def engine(self):
        h = vp()
        rc = self.lib.gss_engine_create(0, ctypes.byref(h))
        return rc, h
