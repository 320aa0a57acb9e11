"""Lent result buffers and what goes on around them: the read-back does not
see what the caller writes into a result, and a result may be freed while a
stream is captured."""
import gc

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
