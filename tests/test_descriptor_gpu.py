"""The descriptor kernel where its windows change form: windows of a few pixels
up to the grid's largest radius (31) and above it (samples straight from the
level), at every column offset of the grid fill's words, inside the level and
across its borders, against the oracle within the descriptor bar; and the same
bits in every storage mode."""
import numpy as np
import pytest

from parity import DESC_RTOL, match
from synthetic import synth_image

CASES = [
    # width, height, seed, sift_new args, (smallest, largest) radius that must occur
    (131, 97, 2, (0.8, 3, 3, 0.5, 0.02, 10.0), (10, 14)),
    (97, 203, 4, (1.6, 4, 3, 0.5, 0.02, 10.0), (18, 28)),
    (400, 301, 6, (1.7, 2, 2, 0.5, 0.02, 10.0), (20, 31)),
    (333, 250, 8, (2.2, 3, 3, 0.5, 0.01, 10.0), (27, 36)),
    (640, 64, 10, (1.6, 2, 5, 0.5, 0.01, 10.0), (17, 28)),
]
IDS = [f"{c[0]}x{c[1]}_sigma{c[3][0]}" for c in CASES]


def radii(kps):
    so = kps["size"].astype(np.float64) / 2.0 ** kps["octave"]
    return np.ceil(12 * so * np.sqrt(2) / 2).astype(int)


@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_cases_reach_their_windows(oracle_mod, case):
    w, h, seed, args, (lo, hi) = case
    kps, _ = oracle_mod.detect_and_compute(synth_image(seed, w, h), oracle_mod.params(*args))
    r = radii(kps)
    scale = 2.0 ** kps["octave"]
    x, y = kps["x"] / scale, kps["y"] / scale
    inner = (x > r + 1) & (y > r + 1) & (x + r + 2 < w // scale) & (y + r + 2 < h // scale)
    assert r.min() <= lo and r.max() >= hi
    assert (~inner).any() and (inner.any() or h == 64)
    if inner.any():
        assert set((np.floor(x[inner]).astype(int) - r[inner] - 1) & 3) == {0, 1, 2, 3}


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_windows_against_the_oracle(built_lib, oracle_mod, case):
    import sift_wgpu_gb300 as sgb
    w, h, seed, args, _ = case
    img = synth_image(seed, w, h)
    rk, rd = oracle_mod.detect_and_compute(img, oracle_mod.params(*args))
    got = [sgb.Engine(sgb.Sift.new(*args), storage=s).detect_and_compute(img) for s in ("u8", "f16", "f32")]
    m = match(rk, rd, *got[0])
    assert len(m.pairs) >= 0.98 * len(rk) > 0, m.summary()
    assert float(m.desc_err.max()) <= DESC_RTOL, m.summary()
    for kps, desc in got[1:]:
        assert np.array_equal(kps, got[0][0]) and np.array_equal(desc, got[0][1])
