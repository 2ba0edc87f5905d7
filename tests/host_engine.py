"""The engine's host code without a GPU: its own objects (komd_gb300/_build) linked
with tests/fake_cudart.cpp in place of the CUDA runtime.  No kernel runs."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="session")
def host_library(tmp_path_factory):
    from komd_gb300 import build
    build.build()
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    out = str(tmp_path_factory.mktemp("host") / "libkomd_host_only.so")
    objs = [os.path.join(build.OUT, s.replace(".cu", ".o")) for s in build.GPU_SOURCES]
    # -Bsymbolic: the fake's functions, whatever else of the runtime this process holds
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-O1", "-Wl,-Bsymbolic", "-I" + os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "fake_cudart.cpp")] + objs + ["-o", out, "-lpthread"], check=True)
    return out


@pytest.fixture
def host(host_library, monkeypatch):
    """komd_gb300.gpu bound to the host-only library; the fixture's value is that
    library (fake_* functions)."""
    from komd_gb300 import gpu
    monkeypatch.setattr(gpu, "LIB_GPU", host_library)
    monkeypatch.setattr(gpu, "_lib", None)
    lib = gpu.load()
    lib.fake_live.argtypes = [ctypes.c_size_t]
    lib.fake_count.argtypes = [ctypes.c_char_p]
    lib.fake_fail_malloc.argtypes = [ctypes.c_long]
    lib.fake_fail_malloc(-1)
    lib.fake_reset()
    return lib
