"""64-row tiles of the level kernel by option, on planes that take 32-row tiles
by themselves and with taps that sum above 1: the oracle's pyramid, bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (65, 33), (63, 129), (257, 131)])
@pytest.mark.parametrize("params", [(1.6, 4, 3, 0.5), (0.45, 2, 3, 0.3), (2.3, 4, 2, 0.5)])
@pytest.mark.parametrize("storage", ["u8", "f16", "f32"])
def test_tall_tiles_on_small_planes(built_lib, oracle_mod, storage, params, w, h):
    import sift_wgpu_gb300 as sgb
    sigma, octaves, intervals, assumed = params
    img = np.random.default_rng(w).integers(0, 256, (h, w), dtype=np.uint8)
    want = oracle_mod.stages(img, oracle_mod.params(sigma, octaves, intervals, assumed, 0.04, 10.0)).pyramid
    s = sgb.Sift.new(sigma, octaves, intervals, assumed, 0.04, 10.0)
    with sgb.Engine(s, storage=storage, level_tile_rows=64) as e:
        e.detect_and_compute(img)
        assert np.array_equal(e.debug_stage(sgb.STAGE_PYRAMID), want)
