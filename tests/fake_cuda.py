"""The library's own objects linked against a CUDA runtime in host memory (fake_cudart.cpp): its
host code runs without a GPU, with failures of allocations and launches made by the test."""
import ctypes
import glob
import os
import subprocess

import pytest

import vfs_b200 as vfs
from vfs_b200 import build, cases

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="session")
def fake_library(tmp_path_factory):
    objs = sorted(glob.glob(os.path.join(build.OBJ, "*.o")))
    if len(objs) != len(build.sources()):
        pytest.skip("the library's objects are not built here")
    out = str(tmp_path_factory.mktemp("fake") / "libvfs_fake.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-z,defs", "-Wl,-Bsymbolic",
                    "-I/usr/local/cuda/include", os.path.join(HERE, "fake_cudart.cpp")] + objs + ["-o", out], check=True)
    return out


@pytest.fixture
def fake(fake_library):
    """The fake library in the place of the real one: vfs.Context uses it, the returned handle
    controls it."""
    own = vfs._lib
    lib = vfs.load_library(fake_library)
    lib.fake_fail_kernel.argtypes = [ctypes.c_char_p]
    lib.fake_launches.argtypes = [ctypes.c_char_p]
    lib.fake_limit.argtypes = [ctypes.c_long]
    for f in ("launches", "mallocs", "allocated", "cleared_bytes", "captures", "graph_launches"):
        getattr(lib, "fake_" + f).restype = ctypes.c_long
    lib.fake_reset()
    yield lib
    lib.fake_reset()
    vfs._lib = own


def context(nx=16, ny=16, nz=16, immersed=0):
    case = cases.channel(nx, ny, nz)
    case.immersed = immersed
    ctx = vfs.Context(case.config())
    ctx.form_metrics(case.X, case.Y, case.Z)
    ctx.set_field(vfs.NVERT, case.nvert)
    return ctx
