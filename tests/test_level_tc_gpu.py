"""The tensor-core level kernel against the oracle, bit for bit: every window
shape (blur radii 1 to 28 and the two-pass radii above), planes smaller than,
equal to and one pixel beyond its tiles, taps that sum above 1 (the clamped
form), and images whose sums lie on or next to an integer: constant areas of
every value, black, white, and full-range noise. The kernel may only take
another route to the same integers, so equality is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb(built_lib):
    import sift_wgpu_gb300 as sg
    return sg


def picture(kind, w, h):
    rng = np.random.default_rng(w * 8191 + h)
    if kind == "noise":
        return rng.integers(0, 256, (h, w), dtype=np.uint8)
    if kind == "black":
        return np.zeros((h, w), np.uint8)
    if kind == "white":
        return np.full((h, w), 255, np.uint8)
    if kind == "steps":  # areas of 0, 1, 254 and 255
        return rng.choice(np.array([0, 1, 254, 255], np.uint8), ((h + 36) // 37, (w + 40) // 41)).repeat(37, 0).repeat(41, 1)[:h, :w].copy()
    side = np.arange(256, dtype=np.uint8).reshape(16, 16)  # "flats": one area for each value
    return np.kron(side, np.ones((h // 16 + 1, w // 16 + 1), np.uint8))[:h, :w].copy()


# (sigma, octaves, intervals, assumed blur): level radii 3-7, 5-13, 10-25, 20-50 at the default; finer scales
# and small sigmas have radii 1-2 and taps that sum above 1
PARAMS = [(1.6, 4, 3, 0.5), (0.6, 3, 8, 0.5), (2.3, 4, 2, 0.5), (0.45, 2, 3, 0.3)]


@pytest.mark.parametrize("w,h", [(1, 1), (3, 70), (64, 32), (65, 33), (63, 129), (200, 31), (257, 131)])
@pytest.mark.parametrize("params", PARAMS)
def test_levels_at_tile_edges(sgb, oracle_mod, params, w, h):
    sigma, octaves, intervals, assumed = params
    for kind in ("noise", "steps"):
        img = picture(kind, w, h)
        want = oracle_mod.stages(img, oracle_mod.params(sigma, octaves, intervals, assumed, 0.04, 10.0)).pyramid
        for rows in (0, 32):
            s = sgb.Sift.new(sigma, octaves, intervals, assumed, 0.04, 10.0)
            with sgb.Engine(s, level_tile_rows=rows) as e:
                e.detect_and_compute(img)
                assert np.array_equal(e.debug_stage(sgb.STAGE_PYRAMID), want), (kind, rows)


@pytest.mark.parametrize("kind", ["flats", "black", "white", "noise"])
@pytest.mark.parametrize("storage", ["u8", "f16", "f32"])
def test_levels_next_to_integers(sgb, oracle_mod, kind, storage):
    """64-row tiles (a plane that fills the device) on constant areas of every value."""
    img = picture(kind, 1616, 1040)
    want = oracle_mod.stages(img).pyramid
    with sgb.Engine(sgb.Sift.default(), storage=storage) as e:
        e.detect_and_compute(img)
        assert np.array_equal(e.debug_stage(sgb.STAGE_PYRAMID), want)
        if storage == "u8":
            with sgb.Batch(sgb.Sift.default()) as b:
                k, d = b.detect_and_compute([img])[0]
                k1, d1 = e.detect_and_compute(img)
                assert k.tobytes() == k1.tobytes() and d.tobytes() == d1.tobytes()
