"""Builds kernel_entries.cu against the in-tree library and loads it."""
import ctypes as C
import os
import subprocess

from tracer_code_gb300 import build as tcbuild

_lib = None


def load():
    global _lib
    if _lib is None:
        so = tcbuild.build()
        here = os.path.dirname(os.path.abspath(__file__))
        out = os.path.join(tcbuild.BUILD, "libkernel_entries.so")
        src = os.path.join(here, "kernel_entries.cu")
        cmd = [tcbuild.nvcc_path(), "-shared", src, "-o", out] + tcbuild.common_flags() + [
            "-L", os.path.dirname(so), "-l:" + os.path.basename(so), "-Xlinker", "-rpath," + os.path.dirname(so)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        _lib = C.CDLL(out)
    return _lib


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)
