"""The library's host code on the CPU: its own objects linked with a CUDA
runtime whose kernels do nothing (tests/cpp/fake_cudart.cpp). Fixture `fake`:
the package's Simulation and Batch drive that library; `fake` sets how the
runtime answers and tells which kernels were launched."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


class Fake:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_log.restype = C.c_char_p
        lib.fake_cost.argtypes = [C.c_char_p, C.c_double]
        lib.fake_held.restype = C.c_longlong
        lib.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]

    def device(self, d):
        self.lib.cudaSetDevice(d)

    def sms(self, n):
        self.lib.fake_sms(n)

    def refuse(self, part):
        self.lib.fake_refuse(part.encode())

    def cost(self, part, ms):
        self.lib.fake_cost(part.encode(), ms)

    def raster_bad(self, bad):
        self.lib.fake_raster_bad(int(bad))

    def load(self, blocks):
        self.lib.fake_load(C.c_longlong(blocks))

    def held(self):
        return self.lib.fake_held()

    def malloc(self, n):
        p = C.c_void_p()
        self.lib.cudaMalloc(C.byref(p), n)
        return p.value

    def launches(self):
        """the kernels launched since the last call: mangled names, the solvers
        with their levels (levels_of in fake_cudart.cpp)"""
        names = self.lib.fake_log().decode().split()
        self.lib.fake_clear()
        return names


@pytest.fixture(scope="session")
def fake_path(tmp_path_factory):
    from dcgrid_gb300 import build
    cxx = shutil.which("g++")
    if not cxx or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("g++ or the CUDA headers missing")
    objs = [os.path.join(build.BUILD, os.path.splitext(s)[0] + ".o") for s in build.SOURCES]
    build.build(force=not all(os.path.exists(o) for o in objs))
    out = str(tmp_path_factory.mktemp("fake") / "libdcg_fake.so")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", os.path.join(CUDA, "include"),
                        os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp")] + objs + ["-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.fixture
def fake(fake_path, tmp_path, monkeypatch):
    """a fresh copy of the library and its runtime for every test"""
    from dcgrid_gb300 import sim
    path = str(tmp_path / "libdcg_fake.so")
    shutil.copyfile(fake_path, path)
    monkeypatch.setattr(sim, "LIB_PATH", path)
    monkeypatch.setattr(sim, "_lib", None)
    return Fake(sim.lib())
