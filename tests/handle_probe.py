"""Builds and loads handle_probe.cpp against the in-tree library."""
from __future__ import annotations

import ctypes
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def load(out_dir) -> ctypes.CDLL:
    from spherocyls_gb300 import build

    cuda = build.cuda_home()
    so = os.path.join(str(out_dir), "libhandle_probe.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "handle_probe.cpp"), f"-I{build.CSRC}",
                    f"-I{os.path.join(cuda, 'include')}", f"-L{build.LIB}", "-lspherocyl",
                    f"-Wl,-rpath,{build.LIB}", f"-L{os.path.join(cuda, 'lib64')}",
                    "-lcudart_static", "-ldl", "-lpthread", "-lrt"], check=True)
    lib = ctypes.CDLL(so)
    lib.probe_set_pass.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_double]
    lib.probe_or_status.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.probe_extras.argtypes = [ctypes.c_void_p]
    lib.probe_give_back.argtypes = [ctypes.c_void_p]
    lib.probe_fill.argtypes = [ctypes.c_size_t]
    lib.probe_fill.restype = ctypes.c_void_p
    lib.probe_free.argtypes = [ctypes.c_void_p]
    lib.probe_exhaust.argtypes = [ctypes.c_void_p]
    lib.probe_release.argtypes = [ctypes.c_void_p]
    return lib
