"""The library's host code on the CPU: its object files linked with a stand-in for the CUDA runtime
(tests/fake_cudart.cpp) that records launches instead of running them."""
import ctypes as C
import functools
import os
import shutil
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


@functools.lru_cache
def _linked():
    from beachslope_gb300 import build
    objs = [os.path.join(build.OUT, s.replace(".cu", ".o")) for s in build.SOURCES]
    build.build_library(force=not all(map(os.path.exists, objs)))
    tmp = tempfile.TemporaryDirectory()
    out = os.path.join(tmp.name, "libfake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", inc,
                           os.path.join(HERE, "fake_cudart.cpp"), *objs, "-o", out])
    return tmp, out


class FakeGpu:
    """api: the Python mirror, bound to the stand-in; calls(): the launches since the last clear()."""

    def __init__(self, monkeypatch, tmp):
        from beachslope_gb300 import api
        own = os.path.join(str(tmp), "libfake.so")   # a file of its own: a state of its own
        shutil.copy(_linked()[1], own)
        monkeypatch.setattr(api, "LIB_PATH", own)
        monkeypatch.setattr(api, "lib", api._load())
        self.api, self.lib = api, api.lib
        self.lib.fake_launch.restype = C.c_char_p
        self.lib.fake_pin.argtypes = [C.c_void_p, C.c_size_t]
        self.lib.fake_unpin.argtypes = [C.c_void_p]
        self.lib.fake_room.argtypes = [C.c_size_t]

    def clear(self):
        self.lib.fake_clear()

    def calls(self, name=""):
        g, b = C.c_uint(), C.c_uint()
        got = []
        for i in range(self.lib.fake_launches()):
            n = self.lib.fake_launch(i, C.byref(g), C.byref(b)).decode()
            if name in n:
                got.append((n, g.value, b.value))
        return got
