"""What the host code does when a CUDA call fails, checked on the CPU: the
library's objects are linked against a fake CUDA runtime (fake_cuda.cpp) that
logs the calls and makes a chosen one return an error."""
import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest

from sift_wgpu_gb300 import _capi, build_ext

ERR_MEMORY = 2  # cudaErrorMemoryAllocation


class Fake:
    def __init__(self, path):
        self.lib = L = C.CDLL(str(path))
        L.fake_fail.argtypes = [C.c_char_p, C.c_int, C.c_int]
        L.fake_counter.argtypes = [C.c_uint32, C.c_uint32]
        L.fake_log.argtypes = [C.c_char_p, C.c_size_t]
        real = _capi.lib()
        for name in _capi.exported_symbols():
            fn, sig = getattr(L, name), getattr(real, name)
            fn.argtypes, fn.restype = sig.argtypes, sig.restype

    def fail(self, api, nth=1):
        self.lib.fake_fail(api.encode(), nth, ERR_MEMORY)

    def log(self):
        buf = C.create_string_buffer(1 << 22)
        self.lib.fake_log(buf, len(buf))
        return buf.value.decode().splitlines()

    def engine(self, params=None, **options):
        p = _capi.Params()
        self.lib.sift_cuda_params_default(C.byref(p))
        o = _capi.Options()
        self.lib.sift_cuda_options_default(C.byref(o))
        for k, v in options.items():
            setattr(o, k, v)
        h = C.c_void_p()
        assert self.lib.sift_cuda_create(C.byref(params or p), C.byref(o), C.byref(h)) == 0
        return h

    def detect(self, h, img):
        r = _capi.Result()
        rc = self.lib.sift_cuda_detect_and_compute(h, img.ctypes.data, img.shape[1], img.shape[0], img.strides[0],
                                                   C.byref(r))
        return rc, r


@pytest.fixture(scope="module")
def fake_lib(built_lib, tmp_path_factory):
    objs = [build_ext.BUILD / (s + ".o") for s in build_ext.CU_SOURCES + build_ext.CPP_SOURCES]
    if not all(o.exists() for o in objs):
        build_ext.build(force=True)
    out = tmp_path_factory.mktemp("fake") / "libsiftfake.so"
    include = build_ext.Path(build_ext._nvcc()).resolve().parents[1] / "include"
    subprocess.run([shutil.which("g++"), "-shared", "-fPIC", "-O1", "-std=c++17", "-I", str(include), "-o", str(out),
                    *map(str, objs), str(build_ext.PKG.parent / "tests" / "fake_cuda.cpp"), "-Wl,-Bsymbolic",
                    "-Wl,--no-undefined", "-lpthread"], check=True)
    return Fake(out)


@pytest.fixture
def fake(fake_lib):
    fake_lib.lib.fake_reset()
    return fake_lib


def aligned(shape, dtype=np.uint8, start=0):
    """An array whose memory starts `start` bytes after a 16-byte boundary."""
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    buf = np.zeros(n + 32, np.uint8)
    off = -buf.ctypes.data % 16 + start
    return buf[off:off + n].view(dtype).reshape(shape)


# ---- a call that failed does not make the next one fail ----------------------

@pytest.mark.parametrize("api", ["cudaHostAlloc", "cudaMalloc", "cudaStreamBeginCapture", "cudaGraphInstantiate",
                                 "cudaGraphLaunch", "cudaStreamSynchronize"])
def test_the_error_of_a_failed_call_is_not_the_next_ones(fake, api):
    """The runtime keeps a failed call's error until it is read; the launches look at it."""
    img = aligned((1024, 1040))
    h = fake.engine()
    fake.fail(api)
    assert fake.detect(h, img)[0] != 0
    assert fake.detect(h, img)[0] == 0
    fake.lib.sift_cuda_destroy(h)
    fake.lib.sift_cuda_destroy(fake.engine())
