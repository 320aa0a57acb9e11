"""What the host code does when a CUDA call fails, checked on the CPU: the
library's objects are linked against a fake CUDA runtime (fake_cuda.cpp) that
logs the calls and makes a chosen one return an error."""
import ctypes as C
import os
import shutil
import signal
import subprocess
import time

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

    def batch(self):
        p, o, h = _capi.Params(), _capi.Options(), C.c_void_p()
        self.lib.sift_cuda_params_default(C.byref(p))
        self.lib.sift_cuda_options_default(C.byref(o))
        assert self.lib.sift_cuda_batch_create(C.byref(p), C.byref(o), C.byref(h)) == 0
        return h

    def detect_batch(self, h, img):
        res = _capi.BatchResult()
        one = (_capi.BatchImage * 1)(_capi.BatchImage(img.ctypes.data, img.shape[1], img.shape[0], img.strides[0]))
        return self.lib.sift_cuda_batch_detect_and_compute(h, one, 1, C.byref(res))

    def server(self, **options):
        p, o, h = _capi.Params(), _capi.ServerOptions(), C.c_void_p()
        self.lib.sift_cuda_params_default(C.byref(p))
        self.lib.sift_cuda_server_options_default(C.byref(o))
        for k, v in options.items():
            setattr(o, k, v)
        assert self.lib.sift_cuda_server_create(C.byref(p), C.byref(o), C.byref(h)) == 0
        return h

    def request(self, h, img):
        """A borrowed image's request: its status, and the log from submit to poll."""
        ticket, served = C.c_uint64(), _capi.Served()
        self.log()
        assert self.lib.sift_cuda_server_submit(h, img.ctypes.data, img.shape[1], img.shape[0], img.strides[0], 7, 1,
                                                C.byref(ticket)) == 0
        assert self.lib.sift_cuda_server_poll(h, C.byref(served), 10_000_000) == 1
        log = self.log()
        assert self.lib.sift_cuda_server_release(h, ticket) == 0
        return served.status, log

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


@pytest.mark.parametrize("form", ["engine", "batch"])
def test_a_launch_that_fails_in_a_capture(fake, form):
    """The capture's end fails too (its other streams have not come back to it), and nobody reports that."""
    img = aligned(SMALL)

    def attempt(nth):
        fake.lib.fake_reset()
        h = fake.engine() if form == "engine" else fake.batch()
        run = (lambda: fake.detect(h, img)[0]) if form == "engine" else (lambda: fake.detect_batch(h, img))
        fake.fail("launch", nth)
        fake.fail("cudaStreamEndCapture")
        failed = run() != 0 and "failed launch" in fake.log()
        assert not failed or run() == 0
        close = fake.lib.sift_cuda_destroy if form == "engine" else fake.lib.sift_cuda_batch_destroy
        close(h)
        if failed:
            fake.lib.sift_cuda_destroy(fake.engine())
        return failed

    assert failures("launch", attempt) >= 20


READS_CALLER = ("k_fetch", "k_to_luma", "k_sq_norms", "cudaGraphLaunch")


def waited(log):
    """Whether a stream wait follows the last launch that may read the caller's memory; None without one."""
    for line in reversed(log):
        if line.startswith("cudaStreamSynchronize"):
            return True
        if any(k in line for k in READS_CALLER) and not line.startswith("failed"):
            return False
    return None


# ---- a call that fails leaves no kernel that reads the caller's memory ------

AFTER_UPLOAD = ["cudaHostAlloc", "cudaStreamBeginCapture", "cudaStreamEndCapture", "cudaGraphInstantiate",
                "cudaGraphLaunch"]


@pytest.mark.parametrize("api", AFTER_UPLOAD)
@pytest.mark.parametrize("shape,start", [((1024, 1040), 0), ((40, 50), 3)])
def test_failed_detection_has_let_go_of_the_image(fake, api, shape, start):
    h = fake.engine()
    fake.log()
    fake.fail(api)
    rc, _ = fake.detect(h, aligned(shape, start=start))
    log = fake.log()
    assert rc != 0 and any("k_fetch" in line for line in log)
    assert waited(log)
    rc, _ = fake.detect(h, aligned(shape, start=start))
    assert rc == 0
    fake.lib.sift_cuda_destroy(h)


@pytest.mark.parametrize("api", AFTER_UPLOAD)
def test_failed_colour_detection_has_let_go_of_the_pixels(fake, api):
    px = aligned((30, 40, 4))
    h, r = fake.engine(), _capi.Result()
    fake.log()
    fake.fail(api)
    rc = fake.lib.sift_cuda_detect_and_compute_pixels(h, px.ctypes.data, 40, 30, 160, _capi.PIXELS_RGBA8, C.byref(r))
    log = fake.log()
    assert rc != 0 and any("k_to_luma" in line for line in log)
    assert waited(log)
    fake.lib.sift_cuda_destroy(h)


def test_failed_match_has_let_go_of_the_rows(fake):
    rows, out = aligned((5, 128), np.float32), np.zeros(5, _capi.MATCH_DTYPE)
    h = fake.engine()
    for api in ("encode", "cudaFuncSetAttribute"):
        fake.log()
        fake.fail(api)
        rc = fake.lib.sift_cuda_match(h, rows.ctypes.data, 5, rows.ctypes.data, 5, out.ctypes.data)
        log = fake.log()
        assert rc != 0 and any("k_sq_norms" in line for line in log)
        assert waited(log), api
    fake.lib.sift_cuda_destroy(h)


@pytest.mark.parametrize("nth", [1, 2])
def test_failed_batch_has_let_go_of_the_images(fake, nth):
    """A batch reads its images in place from its graph; the event after it fails (the first is before it)."""
    h, img = fake.batch(), aligned((32, 64))
    for _ in range(2):
        fake.log()
        assert fake.detect_batch(h, img) == 0
    assert sum(line == "cudaEventRecord" for line in fake.log()) == 2
    fake.fail("cudaEventRecord", nth)
    assert fake.detect_batch(h, img) != 0
    assert waited(fake.log()) is not False
    fake.lib.sift_cuda_batch_destroy(h)


@pytest.mark.parametrize("api", ["cudaHostAlloc", "cudaGraphInstantiate", "cudaGraphLaunch", "done event"])
@pytest.mark.parametrize("autotune", [0, 1])
def test_failed_request_has_let_go_of_a_borrowed_image(fake, api, autotune):
    h, img = fake.server(autotune=autotune), aligned((40, 50), start=3)
    if api == "done event":
        status, log = fake.request(h, img)  # a slot, tuned and captured
        assert status == 0
        fake.fail("cudaEventRecord")
    elif api == "cudaHostAlloc":
        fake.fail(api, 3)  # (two are made with the slot: counters, cell)
    else:
        fake.fail(api)
    status, log = fake.request(h, img)
    assert status != 0 and any("k_fetch" in line for line in log)
    assert waited(log)
    fake.lib.sift_cuda_server_destroy(h)


# ---- a layout that failed half-way is laid out again -------------------------

SMALL, LARGE = (48, 64), (120, 160)
N_CAND = 8  # the word of octave 0's candidate count in a run's counters


def failures(api, attempt):
    """attempt(fail) with the 1st, 2nd, .. call of the api failing, until none is left; their number."""
    for nth in range(1, 200):
        if not attempt(nth):
            return nth - 1
    raise AssertionError(api)


@pytest.mark.parametrize("api", ["cudaMalloc", "cudaMemcpyAsync"])
@pytest.mark.parametrize("again", [SMALL, LARGE])
def test_engine_lays_out_again_after_a_failed_layout(fake, api, again):
    small, large = aligned(SMALL), aligned(LARGE)

    def attempt(nth):
        h = fake.engine()
        assert fake.detect(h, small)[0] == 0
        buffers = fake.lib.fake_live_device()
        fake.log()
        fake.fail(api, nth)
        failed = fake.detect(h, large)[0] != 0
        fake.lib.fake_reset()
        assert fake.detect(h, small if again == SMALL else large)[0] == 0
        # every buffer exists, and the tables are the small size's again
        assert fake.lib.fake_live_device() == buffers
        assert again == LARGE or "cudaMemcpyAsync" in fake.log()
        fake.lib.sift_cuda_destroy(h)
        return failed

    assert failures(api, attempt) >= 4


def test_engine_lays_out_again_after_lists_failed_to_grow(fake):
    img = aligned(SMALL)

    def attempt(nth):
        h = fake.engine()
        assert fake.detect(h, img)[0] == 0
        buffers = fake.lib.fake_live_device()
        fake.lib.fake_counter(N_CAND, 100_000)
        fake.fail("cudaMalloc", nth)
        failed = fake.detect(h, img)[0] != 0
        fake.lib.fake_reset()
        assert fake.detect(h, img)[0] == 0
        assert fake.lib.fake_live_device() == buffers
        fake.lib.sift_cuda_destroy(h)
        return failed

    assert failures("cudaMalloc", attempt) >= 4


def test_server_lays_out_again_after_lists_failed_to_grow(fake):
    img = aligned(SMALL)

    def attempt(nth):
        h = fake.server()
        assert fake.request(h, img)[0] == 0
        buffers = fake.lib.fake_live_device()
        fake.lib.fake_counter(N_CAND, 100_000)
        fake.fail("cudaMalloc", nth)
        failed = fake.request(h, img)[0] != 0
        fake.lib.fake_reset()
        assert fake.request(h, img)[0] == 0
        assert fake.lib.fake_live_device() == buffers
        fake.lib.sift_cuda_server_destroy(h)
        return failed

    assert failures("cudaMalloc", attempt) >= 4


@pytest.mark.parametrize("api", ["cudaMalloc", "cudaMemcpyAsync", "cudaHostAlloc", "cudaHostGetDevicePointer"])
@pytest.mark.parametrize("again", [SMALL, LARGE])
def test_batch_lays_out_again_after_a_failed_layout(fake, api, again):
    small, large = aligned(SMALL), aligned(LARGE)

    def attempt(nth):
        h = fake.batch()
        assert fake.detect_batch(h, small) == 0
        buffers = fake.lib.fake_live_device()
        fake.fail(api, nth)
        failed = fake.detect_batch(h, large) != 0
        fake.lib.fake_reset()
        assert fake.detect_batch(h, small if again == SMALL else large) == 0
        log = fake.log()
        assert fake.lib.fake_live_device() == buffers
        # the result buffer is this layout's: its parts depend on it, and none is left of one that failed
        if again == SMALL or (failed and api.startswith("cudaHost")):
            assert "cudaHostAlloc" in log
        fake.lib.sift_cuda_batch_destroy(h)
        return failed

    assert failures(api, attempt) >= 1


def test_batch_lays_out_again_after_lists_failed_to_grow(fake):
    img = aligned(SMALL)

    def attempt(nth):
        h = fake.batch()
        assert fake.detect_batch(h, img) == 0
        buffers = fake.lib.fake_live_device()
        fake.lib.fake_counter(N_CAND, 100_000)
        fake.fail("cudaMalloc", nth)
        failed = fake.detect_batch(h, img) != 0
        fake.lib.fake_reset()
        assert fake.detect_batch(h, img) == 0
        assert fake.lib.fake_live_device() == buffers
        fake.lib.sift_cuda_batch_destroy(h)
        return failed

    assert failures("cudaMalloc", attempt) >= 4


# ---- where a run read its image ----------------------------------------------

@pytest.mark.parametrize("shape,start,sigma,in_place", [
    ((40, 64), 0, 1.6, 1), ((1023, 1024), 0, 1.6, 1),
    ((1024, 1024), 0, 1.6, 0),  # brought in by a kernel of its own
    ((2048, 2064), 0, 1.6, 0),
    ((40, 64), 0, 0.5, 0),      # no base blur: the copy is read
    ((40, 64), 1, 1.6, 0), ((40, 50), 0, 1.6, 0)])
def test_in_place_says_where_the_run_read_the_image(fake, shape, start, sigma, in_place):
    p = _capi.Params()
    fake.lib.sift_cuda_params_new(C.byref(p), sigma, 1, 1, 0.5, 0.04, 10.0)
    h = fake.engine(p)
    assert fake.detect(h, aligned(shape, start=start))[0] == 0
    assert any("k_fetch" in line for line in fake.log()) != bool(in_place)
    assert fake.lib.sift_cuda_last_image_in_place(h) == in_place
    px, r = aligned((30, 40, 4)), _capi.Result()  # colour pixels become the engine's own plane
    assert fake.lib.sift_cuda_detect_and_compute_pixels(h, px.ctypes.data, 40, 30, 160, _capi.PIXELS_RGBA8,
                                                        C.byref(r)) == 0
    assert fake.lib.sift_cuda_last_image_in_place(h) == 0
    fake.lib.sift_cuda_destroy(h)


# ---- rows of the level kernel's tiles ----------------------------------------

@pytest.mark.parametrize("rows,small,large", [(0, 32, 64), (32, 32, 32), (64, 64, 64)])
@pytest.mark.parametrize("sigma,assumed", [(1.6, 0.5), (0.45, 0.3)])  # (the second's taps sum above 1)
def test_tile_rows_by_option(fake, rows, small, large, sigma, assumed):
    p = _capi.Params()
    fake.lib.sift_cuda_params_new(C.byref(p), sigma, 1, 3, assumed, 0.04, 10.0)
    h = fake.engine(p, level_tile_rows=rows)
    for shape, want in (((100, 64), small), ((1100, 1600), large)):
        fake.log()
        assert fake.detect(h, aligned(shape))[0] == 0
        # (kernels of taps that sum above 1 take 32-row tiles where nothing else is asked)
        levels = [line.split() for line in fake.log() if "k_blur_level" in line]
        grids = {line[2] for line in levels if not (want == 64 and rows == 0 and "Lb1E" in line[1])}
        assert grids == {f"{-(-shape[1] // 64)}x{-(-shape[0] // want)}"}
    fake.lib.sift_cuda_destroy(h)


# ---- lent results in a forked child ------------------------------------------

N_ORIENTED = 2  # the word of the keypoint count


@pytest.fixture
def lent(fake):
    """A lent result, on a device that writes plain memory."""
    fake.lib.fake_host_tables(1)
    h, img = fake.engine(), aligned(SMALL)
    fake.lib.fake_counter(N_ORIENTED, 1000)
    for _ in range(10):
        rc, r = fake.detect(h, img)
        assert rc == 0 and r.n == 1000
        fake.lib.sift_cuda_result_free(C.byref(r))
    fake.log()
    rc, r = fake.detect(h, img)
    yield r
    fake.lib.sift_cuda_result_free(C.byref(r))
    fake.lib.sift_cuda_destroy(h)
    fake.lib.fake_host_tables(0)


def ended(pid, seconds):
    end = time.time() + seconds
    while time.time() < end:
        if os.waitpid(pid, os.WNOHANG)[0]:
            return True
        time.sleep(0.0005)
    os.kill(pid, signal.SIGKILL)
    os.waitpid(pid, 0)
    return False


@pytest.mark.filterwarnings("ignore:This process .* is multi-threaded:DeprecationWarning")
def test_a_forked_child_frees_a_lent_result(fake, lent):
    """Forks while other threads free results: the child's own free comes back."""
    free = C.cast(fake.lib.sift_cuda_result_free, C.c_void_p)
    fake.lib.fake_free_results(free, 4)
    try:
        for _ in range(500):
            pid = os.fork()
            if pid == 0:
                fake.lib.sift_cuda_result_free(C.byref(lent))
                os._exit(0)
            assert ended(pid, 20)
    finally:
        fake.lib.fake_free_results(free, 0)
