"""The library linked against tests/fake_cuda.cpp, for tests of its host code on the CPU: failed
allocations and launches, copies that have not run when a call returns, device error bits."""
import ctypes as C
import os
import subprocess

import pytest

import lavaframe_gb300 as lf
from lavaframe_gb300 import build
from tests.conftest import ROOT

HOOK = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.POINTER(C.c_void_p)))
POOL, PINNED = 1, 2


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    """Links the library's objects with the fake runtime and loads the result."""
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    out = tmp_path_factory.mktemp("fake") / "liblf_fake.so"
    objs = sorted(build.BUILD.glob("*.o"))
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", cuda, "-o", str(out),
                    str(ROOT / "tests" / "fake_cuda.cpp"), *map(str, objs), "-lpthread"], check=True)
    L = C.CDLL(str(out))
    for name, (res, args) in lf._SIG.items():
        fn = getattr(L, name)
        fn.restype, fn.argtypes = res, args
    L.fake_block.restype = C.c_void_p
    L.fake_block.argtypes = [C.c_size_t, C.c_int]
    L.fake_hook.argtypes = [HOOK]
    return L


@pytest.fixture
def fake(fake_lib, monkeypatch):
    """The library on the fake runtime in the package's place."""
    monkeypatch.setattr(lf, "_lib", fake_lib)
    fake_lib.fake_reset()
    yield fake_lib
    fake_lib.fake_reset()
