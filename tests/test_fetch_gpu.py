"""How an image comes in: read in place by the base level (small, 16-byte
aligned), brought in by the fetch kernel (large, or starting or striding on
any byte), or copied by the copy engine (pinned). Every way gives the bytes of
the image: the pyramid equals that of a contiguous copy, whatever the start,
the stride and the width, and no byte before or after the image matters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb(built_lib):
    import sift_wgpu_gb300 as sg
    return sg


def pyramid(sgb, e, img):
    e.detect_and_compute(img)
    return e.debug_stage(sgb.STAGE_PYRAMID)


@pytest.mark.parametrize("w,h", [(1, 1), (15, 5), (16, 16), (17, 9), (33, 20), (257, 31), (1003, 40)])
def test_any_start_and_stride(sgb, w, h):
    rng = np.random.default_rng(w)
    img = rng.integers(0, 256, (h, w), dtype=np.uint8)
    with sgb.Engine(sgb.Sift.new(1.6, 1, 1, 0.5, 0.04, 10.0)) as e:
        want = pyramid(sgb, e, img)
        for start in (0, 1, 7, 8, 9, 15):
            for extra in (0, 1, 8, 13):
                buf = np.empty(64 + start + h * (w + extra), np.uint8)
                off = (-buf.ctypes.data) % 16 + start
                fill = rng.integers(0, 256, buf.shape, dtype=np.uint8)
                buf[:] = fill
                # the last row ends with its last pixel
                view = np.lib.stride_tricks.as_strided(buf[off:], (h, w), (w + extra, 1))
                view[:] = img
                assert np.array_equal(pyramid(sgb, e, view), want), (start, extra)


@pytest.mark.parametrize("w,stride,h", [(1040, 1040, 1024), (1025, 1040, 1040), (2047, 2048, 515)])
def test_large_images(sgb, w, stride, h):
    import torch
    img = np.random.default_rng(5).integers(0, 256, (h, stride), dtype=np.uint8)[:, :w]
    with sgb.Engine(sgb.Sift.new(1.6, 1, 1, 0.5, 0.04, 10.0)) as e:
        got = pyramid(sgb, e, img)
        assert np.array_equal(pyramid(sgb, e, torch.from_numpy(np.ascontiguousarray(img)).pin_memory().numpy()), got)
        # new bytes in the same buffer
        img[:] = 255 - img
        assert np.array_equal(pyramid(sgb, e, img), pyramid(sgb, e, torch.from_numpy(np.ascontiguousarray(img)).pin_memory().numpy()))


def test_rgba_in_place_and_copied(sgb):
    px = np.random.default_rng(6).integers(0, 256, (123, 164, 4), dtype=np.uint8)
    buf = np.zeros(px.size + 64, np.uint8)
    with sgb.Engine() as e:
        k, d = e.detect_and_compute(px)
        want = e.debug_stage(sgb.STAGE_PYRAMID)
        for start in (0, 4, 5):
            off = (-buf.ctypes.data) % 16 + start
            view = buf[off:off + px.size].reshape(px.shape)
            view[:] = px
            k1, d1 = e.detect_and_compute(view)
            assert np.array_equal(e.debug_stage(sgb.STAGE_PYRAMID), want)
            assert k1.tobytes() == k.tobytes() and d1.tobytes() == d.tobytes()


def test_device_run_then_host_call(sgb):
    """A host call right behind an asynchronous device run: neither sees the other's image or result buffer."""
    import torch
    rng = np.random.default_rng(8)
    a, b = (rng.integers(0, 256, (300, 400), dtype=np.uint8) for _ in range(2))
    with sgb.Engine() as e, sgb.Engine() as f:
        ka, kb = f.detect_and_compute(a)[0], f.detect_and_compute(b)[0]
        da = torch.from_numpy(a).cuda()
        torch.cuda.synchronize()
        for _ in range(5):
            e.run_device(da.data_ptr(), 400, 300, 400)
            k, _ = e.detect_and_compute(b)
            assert k.tobytes() == kb.tobytes()
            e.run_device(da.data_ptr(), 400, 300, 400)
            e.run_device(da.data_ptr(), 400, 300, 400)
            e.synchronize()
            assert e.debug_stage(sgb.STAGE_KEYPOINTS).tobytes() == ka.tobytes()
