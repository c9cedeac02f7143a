"""The native library's host code on a fake CUDA runtime (fake_cuda.cpp), for
tests of what it asks of the runtime: no GPU needed."""
import ctypes
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor

import build as native_build
import rvsb

HERE = os.path.dirname(os.path.abspath(__file__))


class Launch(ctypes.Structure):
    """FakeLaunch: the current device and that of the output planes, what the
    launch's first slot holds, the colour decodes issued before the launch and
    before its resolve, and the workspace buffers of its slots that have no
    allocation of their size behind them."""

    _fields_ = [(n, ctypes.c_int) for n in ("device", "out_device", "slots", "variant", "small", "views",
                                            "decodes_before", "decodes_at_resolve")] + [("precision", ctypes.c_float),
                                                                                            ("unbacked", ctypes.c_int)]


def build(out_dir):
    """Compiles the library's host sources with the fake; its path."""
    flags = ["-O1", "-std=c++17", "-fPIC", "-ffp-contract=off", "-I", native_build.INCLUDE, "-I", native_build.CSRC,
             "-I", os.path.join(native_build.CUDA_HOME, "include")]
    sources = [os.path.join(native_build.CSRC, f) for f in native_build.CPP_SOURCES]
    sources.append(os.path.join(HERE, "fake_cuda.cpp"))
    objs = [os.path.join(out_dir, os.path.basename(s) + ".o") for s in sources]
    with ThreadPoolExecutor(len(sources)) as ex:
        list(ex.map(lambda so: subprocess.run(["g++"] + flags + ["-c", so[0], "-o", so[1]], check=True),
                    zip(sources, objs)))
    lib = os.path.join(out_dir, "librvsb_fake.so")
    # Symbolic: a CUDA runtime loaded by another module must not take the fake's place.
    subprocess.run(["g++", "-shared", "-o", lib] + objs + ["-ldl", "-lpthread", "-Wl,--no-undefined,-Bsymbolic"],
                   check=True)
    return lib


class Fake:
    """rvsb on the fake library; `lib` has the fake's own functions too."""

    def __init__(self, path, monkeypatch):
        monkeypatch.setattr(rvsb, "_lib", None)
        monkeypatch.setattr(rvsb, "LIB_PATH", path)
        self.lib = rvsb.load()
        self.lib.fake_reset()
        self.lib.fake_set_device(0)

    def launches(self):
        out = []
        for k in range(self.lib.fake_launches()):
            f = Launch()
            self.lib.fake_launch(k, ctypes.byref(f))
            out.append(f)
        return out

    def fail(self, call, after):
        """The call named `call` fails once, after `after` that succeed."""
        self.lib.fake_fail(call.encode(), after)
