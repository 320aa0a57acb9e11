"""Owned results that are lent result buffers: the arrays of
detect_and_compute, detect and the colour call stay the caller's while the
engine goes on, whatever is held, changed, freed elsewhere or outlives the
engine; a bounded number is lent, the rest are copies."""
import gc
import threading

import numpy as np
import pytest

from synthetic import synth_image

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb(built_lib):
    import sift_wgpu_gb300 as sg
    return sg


@pytest.fixture(scope="module")
def frames(sgb):
    """Images of one size and their results, each copied from a view."""
    imgs = [synth_image(900 + i, 400, 300) for i in range(6)]
    with sgb.Engine() as e:
        want = []
        for im in imgs:
            k, d = e.detect_and_compute_view(im)
            want.append((k.copy(), d.copy()))
    return imgs, want


def same(got, want):
    return got[0].tobytes() == want[0].tobytes() and got[1].tobytes() == want[1].tobytes()


def warmed(sgb, img):
    """An engine that has copied enough to lend (each result is freed at once)."""
    e = sgb.Engine()
    for _ in range(80):
        e.detect_and_compute(img)
    return e


def test_held_results_keep_their_values(sgb, frames):
    imgs, want = frames
    e = warmed(sgb, imgs[0])
    held = [e.detect_and_compute(im) for im in imgs]
    addresses = {r[0].ctypes.data for r in held}
    assert len(addresses) == len(held)
    for _ in range(3):
        for im in imgs:
            e.detect_and_compute(im)
            e.detect(im)
    assert all(same(r, w) for r, w in zip(held, want))
    assert all(r[0].flags.writeable and r[1].flags.writeable for r in held)
    e.close()
    gc.collect()
    assert all(same(r, w) for r, w in zip(held, want))


def test_a_changed_result_changes_nothing_else(sgb, frames):
    imgs, want = frames
    with warmed(sgb, imgs[0]) as e:
        for im, w in zip(imgs * 3, want * 3):
            k, d = e.detect_and_compute(im)
            assert same((k, d), w)
            k["x"] = -1.0
            d[:] = 7.0
            kv, dv = e.detect_and_compute_view(im)
            assert same((kv, dv), w)


def test_read_back_after_a_lent_result(sgb, frames):
    imgs, want = frames
    with warmed(sgb, imgs[0]) as e:
        r = e.detect_and_compute(imgs[1])
        del r
        assert e.debug_stage(sgb.STAGE_DESCRIPTORS).tobytes() == want[1][1].tobytes()


def test_results_freed_by_other_threads(sgb, frames):
    imgs, want = frames
    with warmed(sgb, imgs[0]) as e:
        bad = []

        def check(r, w):
            if not same(r, w):
                bad.append(1)

        threads = []
        for im, w in zip(imgs * 10, want * 10):
            threads.append(threading.Thread(target=check, args=(e.detect_and_compute(im), w)))
            threads[-1].start()
        for t in threads:
            t.join()
        assert not bad


def test_colour_and_keypoints_only(sgb, frames):
    imgs, want = frames
    with warmed(sgb, imgs[0]) as e:
        px = [np.repeat(im[:, :, None], 4, axis=2) for im in imgs]
        held = [e.detect_and_compute(p) for p in px]
        only = [e.detect(im) for im in imgs]
        ref = [e.detect_and_compute(p) for p in px]
        assert all(same(a, b) for a, b in zip(held, ref))
        assert all(k.tobytes() == w[0].tobytes() for k, w in zip(only, want))
