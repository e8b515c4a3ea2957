"""Runs renderer code in a child process on a CUDA runtime that needs no GPU (fake_cudart.cpp, preloaded)."""
import os
import subprocess
import sys
import tempfile

TESTS = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
_lib = None

PRELUDE = """
import ctypes as C, sys
sys.path.insert(0, %r)
import numpy as np
from conftest import load_package
PKG = load_package()
fake = C.CDLL(None)
fake.fake_nulls.restype = fake.fake_kernels.restype = C.c_char_p
for f in (fake.fake_mallocs, fake.fake_launches):
    f.restype = C.c_long
fake.fake_fail_malloc.argtypes = [C.c_long]
fake.fake_pending.restype = fake.fake_live_bytes.restype = C.c_size_t


def nulls():
    return fake.fake_nulls().decode()


def scene(n, seed=1):
    rng = np.random.default_rng(seed)
    s = rng.random((n, 16), dtype=np.float32)
    s[:, 4:7] = -4.0
    return s


def raises(fn, *a):
    try:
        fn(*a)
    except PKG.GpsError as e:
        return e
    return None


CAM = PKG.OrbitCamera(distance=4.0).to_camera(64, 48)
P = PKG.RenderParams(spp_side=1)
""" % TESTS


def run(code):
    """The child's output; a failing assertion in it fails the test."""
    global _lib
    if _lib is None:
        _lib = os.path.join(tempfile.mkdtemp(prefix="fake_cudart"), "libfake_cudart.so")
        subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(CUDA, "include"),
                        os.path.join(TESTS, "fake_cudart.cpp"), "-o", _lib, "-ldl", "-pthread"], check=True)
    out = subprocess.run([sys.executable, "-c", PRELUDE + code], capture_output=True, text=True, timeout=300,
                         env={**os.environ, "LD_PRELOAD": _lib})
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout
