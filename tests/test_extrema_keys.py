"""The extrema mask compares 16-bit keys instead of f32 DoG values: over all
pairs of bytes the keys have the values' order, ties included (CPU); and the
candidates are the oracle's at the edges of the mask's 128 x 16 tiles, at every
alignment of a row's end, in dark images, whose values need the keys' rounded
form, and for every number of layers (GPU)."""
import numpy as np
import pytest

from synthetic import synth_image

LUT = np.arange(256, dtype=np.float32) / np.float32(255)
K255 = np.float32(0x808080)


def top_bit(v):
    """The highest power of two in v, as f32 (by its exponent field)."""
    return (v.astype(np.float32).view(np.int32) & 0x7F800000).view(np.float32)


def test_keys_have_the_order_of_the_values():
    a, b = np.meshgrid(np.arange(256), np.arange(256), indexing="ij")
    want = LUT[a] - LUT[b]
    fixed = (np.arange(256) * 0x808080 + top_bit(np.arange(256)).astype(np.int64)).astype(np.float32)
    assert np.array_equal(fixed * np.float32(2.0 ** -31), LUT)
    diff = fixed[a] - fixed[b]
    d = (a - b).astype(np.float32)
    e = (diff.astype(np.float64) - d.astype(np.float64) * K255).astype(np.float32)
    e = np.where(np.abs(e) == 128, np.copysign(np.float32(100), e), e)
    exact = (128 * (a - b) + e.astype(np.int64)).ravel()
    assert exact.min() > -0x8000 and exact.max() < 0x8000
    order = np.argsort(want.ravel(), kind="stable")
    steps, key_steps = np.diff(want.ravel()[order]), np.diff(exact[order])
    assert np.array_equal(steps == 0, key_steps == 0) and (key_steps >= 0).all()
    t = 128 * np.arange(256) + top_bit(np.arange(256)).astype(np.int64)
    safe = (a <= 2 * b) & (b <= 2 * a)
    assert np.array_equal((t[a] - t[b])[safe], exact.reshape(256, 256)[safe])


def dark(seed, w, h):
    """A scene of values 0..40 with a few bright spots."""
    img = (synth_image(seed, w, h).astype(int) // 7 - 8).clip(0, 255)
    rng = np.random.default_rng(seed)
    for _ in range(6):
        y, x = rng.integers(0, h), rng.integers(0, w)
        img[y:y + 5, x:x + 5] = 255
    return img.astype(np.uint8)


SIZES = [(1, 1), (3, 40), (61, 33), (64, 15), (97, 16), (127, 17), (128, 18), (129, 31), (131, 32), (190, 47),
         (256, 48), (257, 49), (323, 50), (386, 97)]


@pytest.mark.gpu
@pytest.mark.parametrize("intervals,border", [(3, 5), (4, 1), (2, 0), (1, 5), (7, 2)])
@pytest.mark.parametrize("scene", ["synth", "dark"])
def test_candidates_against_the_oracle(built_lib, oracle_mod, scene, intervals, border):
    import sift_wgpu_gb300 as sgb
    p = oracle_mod.params(1.6, 3, intervals, 0.5, 0.04, 10.0)
    p.image_border_width = border
    sift = sgb.Sift.new(1.6, 3, intervals, 0.5, 0.04, 10.0)
    sift.image_border_width = border
    eng = sgb.Engine(sift)
    found = 0
    for k, (w, h) in enumerate(SIZES):
        img = (synth_image if scene == "synth" else dark)(k, w, h)
        want = oracle_mod.stages(img, p).candidates
        eng.detect_and_compute(img)
        assert eng.debug_stage(sgb.STAGE_CANDIDATES).tobytes() == want.tobytes(), (w, h)
        found += len(want)
    assert found > 50
