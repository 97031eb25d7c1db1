"""Kernel attributes belong to a device: every op that needs one has to launch on a second GPU of the same process too.
The library's own objects are linked against a stand-in of the CUDA runtime (``fake_cudart.cpp``) that checks launches."""
import ctypes
import glob
import os
import shutil
import subprocess

import pytest

from pippy_b200.csrc import build
from pippy_b200.ops import _lib

CUDA_INCLUDE = "/usr/local/cuda/include"
OBJECTS = sorted(glob.glob(os.path.join(build.OBJ_DIR, "*.o")))
pytestmark = pytest.mark.skipif(not (OBJECTS and shutil.which("g++") and os.path.isdir(CUDA_INCLUDE)),
                                reason="needs the library's objects, g++ and the CUDA headers")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake_cudart.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CUDA_INCLUDE, src, *OBJECTS, "-o", so,
                    "-lpthread"], check=True)
    handle = ctypes.CDLL(so)
    for name, types in _lib.SIGNATURES.items():
        getattr(handle, name).argtypes = [_lib._TYPES[t] for t in types]
    return handle


P = 1 << 20  # an aligned address; nothing reads it


def _xent(lib, classes):
    return lib.pb_xent(P, P, P, P, P, P, 64, classes, (classes + 7) // 8 * 8, -100, None)


def _gemm(lib, variant):
    return lib.pb_gemm_bf16_ws(P, P, P, 512, 512, 512, 512, 512, 512, 0, 0, None, None, 0, None, 0, 0, 0, variant, None, 0,
                               P, None)


def _attention(lib, tokens, heads, dim):
    w = heads * dim
    fwd = lib.pb_flash_fwd(P, P, P, P, P, 1, tokens, heads, heads, dim, w, w, w, w, 1.0, 1, P, None)
    bwd = lib.pb_flash_bwd(*[P] * 10, 1, tokens, heads, heads, dim, w, w, w, w, w, w, 1.0, 1, P, None)
    return fwd or bwd


@pytest.mark.parametrize("call,args", [
    (_xent, (1024,)), (_xent, (32000,)), (_xent, (56000,)), (_xent, (100000,)),
    (_gemm, (0,)), (_gemm, (1,)), (_gemm, (2,)), (_gemm, (3,)),
    (_attention, (512, 4, 64)), (_attention, (512, 4, 128)), (_attention, (4096, 32, 64)), (_attention, (4096, 32, 128)),
])
def test_ops_launch_on_every_device_of_a_process(fake, call, args):
    for device in (0, 1, 70, 0, 1):
        fake.fake_set_device(device)
        before = fake.fake_launches()
        assert call(fake, *args) == 0, (device, args)
        assert fake.fake_launches() > before
