"""Lent result buffers and what goes on around them: the read-back does not
see what the caller writes into a result, and a result may be freed while a
stream is captured."""
import gc
import os
import select
import signal

import numpy as np
import pytest

from synthetic import synth_image

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb(built_lib):
    import sift_wgpu_gb300 as sg
    return sg


@pytest.mark.parametrize("octaves", [1, 4])
def test_read_back_of_a_result_that_the_caller_changed(sgb, octaves):
    img = synth_image(901, 400, 300)
    with sgb.Engine(sgb.Sift.new(1.6, octaves, 3, 0.5, 0.04, 10.0)) as e:
        want = e.detect_and_compute_view(img)[1].copy()
        for _ in range(120):
            k, d = e.detect_and_compute(img)
            d[:] = 7.0
            k["x"] = -1.0
        assert e.debug_stage(sgb.STAGE_DESCRIPTORS).tobytes() == want.tobytes()
        assert e.debug_stage(sgb.STAGE_DESCRIPTORS).tobytes() == want.tobytes()
        k, d = e.detect_and_compute(img)  # the run after it is its own
        assert d.tobytes() == want.tobytes()
        assert e.debug_stage(sgb.STAGE_KEYPOINTS).tobytes() == k.tobytes()


@pytest.fixture
def warmed(sgb):
    """An engine that lends (its results so far were copies that were freed at once)."""
    img = synth_image(900, 400, 300)
    e = sgb.Engine()
    for _ in range(80):
        e.detect_and_compute(img)
    yield e, img
    e.close()


def captured(during):
    """Runs `during` while this thread captures a graph in torch's mode, which forbids unsafe calls to every thread."""
    import torch
    a = torch.ones(8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    gc.disable()
    try:
        with torch.cuda.graph(graph):
            b = a * 2
            during()
    finally:
        gc.enable()
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(b.cpu().numpy(), np.full(8, 2.0, np.float32))


@pytest.mark.parametrize("closed", [False, True])
def test_results_freed_during_a_capture(warmed, closed):
    e, img = warmed
    held = [e.detect_and_compute(img) for _ in range(6)]
    if closed:
        e.close()
    captured(held.clear)


# ---- a result is ordinary memory ---------------------------------------------

def lending(sgb, img):
    """An engine with results to lend, and one that is lent."""
    e = sgb.Engine()
    for _ in range(80):
        e.detect_and_compute(img)
    return e, e.detect_and_compute(img)


@pytest.fixture(scope="module")
def two(sgb):
    imgs = [synth_image(910 + i, 400, 300) for i in range(2)]
    with sgb.Engine() as e:
        return imgs, [tuple(a.copy() for a in e.detect_and_compute_view(im)) for im in imgs]


def test_a_copy_to_the_device_outlives_the_result(sgb, two):
    """An enqueued copy of a result whose stream is busy (for some 25 ms) while the result goes and others come."""
    import torch
    imgs, want = two
    e, (k, d) = lending(sgb, imgs[0])
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(50_000_000)
        on_device = torch.from_numpy(d).to("cuda", non_blocking=True)
    del k, d
    for _ in range(8):
        e.detect_and_compute(imgs[1])
    torch.cuda.synchronize()
    e.close()
    assert on_device.cpu().numpy().tobytes() == want[0][1].tobytes()


@pytest.mark.filterwarnings("ignore:This process .* is multi-threaded:DeprecationWarning")
def test_a_forked_child_keeps_its_results(sgb, two):
    """A child that looks at a result, and writes to it, after the parent has dropped it and gone on."""
    imgs, want = two
    e, r = lending(sgb, imgs[0])
    go, answer = os.pipe(), os.pipe()
    pid = os.fork()
    if pid == 0:
        os.read(go[0], 1)
        ok = r[0].tobytes() == want[0][0].tobytes() and r[1].tobytes() == want[0][1].tobytes()
        r[1][:] = 7.0
        os.write(answer[1], b"1" if ok else b"0")
        os._exit(0)
    held = e.detect_and_compute(imgs[1])
    del r
    for _ in range(8):
        k, d = e.detect_and_compute(imgs[1])
        assert k.tobytes() == want[1][0].tobytes() and d.tobytes() == want[1][1].tobytes()
    os.write(go[1], b"x")
    answered = select.select([answer[0]], [], [], 60)[0]
    if not answered:
        os.kill(pid, signal.SIGKILL)
    os.waitpid(pid, 0)
    assert answered and os.read(answer[0], 1) == b"1"
    for fd in go + answer:
        os.close(fd)
    assert held[1].tobytes() == want[1][1].tobytes() and d.tobytes() == want[1][1].tobytes()
    e.close()
