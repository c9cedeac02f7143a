"""Device helpers of the native library compiled for the host (device_host.hpp
stands in for the intrinsics), for tests of their arithmetic and index logic
without a GPU."""
import ctypes
import os
import re
import subprocess

import build as native_build

HERE = os.path.dirname(os.path.abspath(__file__))

# asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); -> r = ptx_rcp_ftz(x);
_APPROX = re.compile(r'asm\("(rcp|rsqrt)\.approx(\.ftz)?\.f32 %0, %1;"\s*:\s*"=f"\((\w+)\)\s*:\s*"f"\((.*?)\)\);')
_WAIT = re.compile(r'asm volatile\("griddepcontrol\.wait;"[^;]*\);')


def _translate(text):
    text = _APPROX.sub(lambda m: f"{m[3]} = ptx_{m[1]}{'_ftz' if m[2] else ''}({m[4]});", text)
    return _WAIT.sub("", text)


def extract(source, start):
    """The definition in csrc/`source` that begins with the line `start` and
    ends with the first line that closes it in column 0."""
    text = open(os.path.join(native_build.CSRC, source)).read()
    begin = text.index(start)
    return text[begin:re.compile(r"^};?$", re.M).search(text, begin).end()] + "\n"


def build(out_dir, code):
    """Compiles `code` against the translated headers; the loaded library."""
    for f in os.listdir(native_build.CSRC):
        if f.endswith((".cuh", ".hpp")):
            with open(os.path.join(native_build.CSRC, f)) as i, open(os.path.join(out_dir, f), "w") as o:
                o.write(_translate(i.read()))
    src, lib = os.path.join(out_dir, "code.cpp"), os.path.join(out_dir, "code.so")
    with open(src, "w") as o:
        o.write('#include "device_host.hpp"\n' + code)
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-fPIC", "-shared", "-I", out_dir, "-I", HERE, "-I",
                    native_build.INCLUDE, "-I", os.path.join(native_build.CUDA_HOME, "include"), src, "-o", lib,
                    "-lpthread"], check=True)
    return ctypes.CDLL(lib)
