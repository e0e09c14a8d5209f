"""The library's own objects linked with a stand-in for the CUDA runtime
(fake_cudart.cpp), and the binding loaded over it: host code under test
without a GPU."""
import ctypes as C
import importlib.util
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "openqcd-2.4.2_b200")
_so = None


def _build():
    global _so
    if _so is None:
        if not shutil.which("nvcc") or not shutil.which("g++"):
            pytest.skip("no CUDA toolkit")
        spec = importlib.util.spec_from_file_location("b200_build", os.path.join(PKG, "build.py"))
        b = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(b)
        b.build()
        d = tempfile.mkdtemp(prefix="hostlib")
        inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc")))), "include")
        out = os.path.join(d, "libhost.so")
        subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", inc, "-Wl,-Bsymbolic", "-o", out,
                        os.path.join(HERE, "fake_cudart.cpp")]
                       + [os.path.join(b.OBJ, s[:-3] + ".o") for s in b.sources()], check=True)
        _so = out
    return _so


def load():
    """a binding of its own, over a library in its initial state"""
    so = _build()
    own = os.path.join(tempfile.mkdtemp(prefix="host", dir=os.path.dirname(so)), "libhost.so")
    shutil.copyfile(so, own)
    spec = importlib.util.spec_from_file_location("openqcd_b200_host", os.path.join(PKG, "openqcd_b200.py"))
    qb = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(qb)
    qb.LIB_PATH = own
    qb.lib().fake_watch.argtypes = [C.c_char_p, C.c_int, C.c_int]
    return qb
