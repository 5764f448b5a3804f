"""The library's objects linked with a CUDA runtime that needs no GPU
(tests/host/fake_cudart.cpp) and with checks of internal host code
(tests/host/checks.cu)."""
import ctypes as C
import os
import subprocess

from nrpyelliptic_b200 import build

HOST = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host")


def load(tmp):
    """Builds the host library under `tmp` and loads it."""
    build.build()
    objs = [os.path.join(build.OBJDIR, os.path.basename(s) + ".o") for s in build.SOURCES]
    include = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    fake, checks, lib = (os.path.join(str(tmp), f) for f in ("fake.o", "checks.o", "libhost.so"))
    run = lambda *cmd: subprocess.run(cmd, check=True)
    run("g++", "-O1", "-std=c++17", "-fPIC", "-I", include, "-c", os.path.join(HOST, "fake_cudart.cpp"), "-o", fake)
    run(build.nvcc(), *build.ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.INCLUDE, "-I", build.CSRC,
        "-c", os.path.join(HOST, "checks.cu"), "-o", checks)
    run("g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", lib, *objs, fake, checks, "-lgomp")
    return C.CDLL(lib)
