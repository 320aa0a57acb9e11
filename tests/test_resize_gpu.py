"""The 2x resize at the edges of its 32 x 32 tiles, where each output has taps of
its own: planes of a few pixels (fewer taps than a whole window), 15 (the most
taps), odd sides (no uniform interior), one pixel around a multiple of a tile
and of its source window, against the oracle bit for bit."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(2, 2), (5, 3), (15, 15), (31, 62), (63, 64), (65, 66), (127, 30), (130, 131), (193, 257), (258, 95)])
def test_resize_at_tile_edges(built_lib, oracle_mod, w, h):
    import sift_wgpu_gb300 as sgb
    args = (1.6, 5, 1, 0.5, 0.04, 10.0)
    img = np.random.default_rng(w * 1000 + h).integers(0, 256, (h, w)).astype(np.uint8)
    want = oracle_mod.stages(img, oracle_mod.params(*args)).pyramid
    for storage in ("u8", "f32"):
        with sgb.Engine(sgb.Sift.new(*args), storage=storage) as e:
            kps, desc = e.detect_and_compute(img)
            assert np.array_equal(e.debug_stage(sgb.STAGE_PYRAMID), want)
    with sgb.Batch(sgb.Sift.new(*args)) as b:
        (bk, bd), _ = b.detect_and_compute([img, img[::-1].copy()])
        assert np.array_equal(bk, kps) and np.array_equal(bd, desc)
