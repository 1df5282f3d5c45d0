"""The binding over libeagb's host side without a GPU: the library's own
objects linked with fake_cudart.cpp in place of the CUDA runtime.  Kernels do
nothing, so results mean nothing; what the host side allocates, uploads,
launches and refuses is what it does on a GPU."""
import ctypes as C
import importlib.util
import os
import subprocess

from conftest import HERE, ROOT

PKG = os.path.join(ROOT, "ea-lcd-mc_gb300")


def _module(name, path):
    spec = importlib.util.spec_from_file_location(name, path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def load(folder):
    """(binding, fake) with the library built into `folder`."""
    bld = _module("eagb_build", os.path.join(PKG, "build.py"))
    bld.build()
    path = os.path.join(str(folder), "libeagb_fake.so")
    objs = [os.path.join(bld.BUILD, s + ".o") for s in bld.SOURCES]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    "-I" + os.path.join(bld.CUDA, "include"), os.path.join(HERE, "fake_cudart.cpp"), "-o", path] +
                   objs + ["-lpthread"], check=True)
    eagb = _module("eagb_fake", os.path.join(PKG, "eagb.py"))
    eagb.LIB_PATH = path
    fake = eagb.lib()
    for f in ("fake_live", "fake_calls"):
        getattr(fake, f).restype = C.c_long
    fake.fake_live_bytes.restype = C.c_ulonglong
    fake.fake_refused.restype = C.c_char_p
    fake.fake_fail_in.argtypes = [C.c_long]
    return eagb, fake
