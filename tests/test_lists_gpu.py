"""The ordered lists at the edges of their tiles: candidates over 512-word tiles
(one tile, a last one that is partial, tiles with more candidates than are
listed at a time, lists that outgrow their first capacity) and oriented
keypoints over 256-slot tiles, against the oracle's lists bit for bit; and the
offsets that a batch splits its result by."""
import numpy as np
import pytest

from parity import MATCH_RATE, match
from synthetic import synth_image


def args(sigma):
    return (sigma, 2, 3, 0.5, 0.02, 10.0)


def noise(w, h):
    return np.random.default_rng(w).integers(0, 256, (h, w)).astype(np.uint8)


CASES = [
    ("one_tile", 1.6, lambda: synth_image(3, 96, 50)),
    ("words_512", 1.6, lambda: synth_image(4, 64, 256)),  # 3 x 256 x 2 words: whole tiles
    ("words_513", 1.6, lambda: synth_image(5, 32, 171)),  # 3 x 171 words: one over
    ("narrow", 1.6, lambda: synth_image(6, 20, 900)),
    ("noise", 1.0, lambda: noise(512, 384)),
    ("dense", 0.55, lambda: noise(384, 260)),
    ("uneven", 0.55, lambda: np.concatenate([noise(700, 60), synth_image(7, 700, 200)])),
]


@pytest.mark.gpu
@pytest.mark.parametrize("name,sigma,make", CASES, ids=[c[0] for c in CASES])
def test_lists_against_the_oracle(built_lib, oracle_mod, name, sigma, make):
    import sift_wgpu_gb300 as sgb
    img = make()
    st = oracle_mod.stages(img, oracle_mod.params(*args(sigma)))
    eng = sgb.Engine(sgb.Sift.new(*args(sigma)))
    for _ in range(2):  # the second run finds the lists grown
        kps, desc = eng.detect_and_compute(img)
        assert eng.debug_stage(sgb.STAGE_CANDIDATES).tobytes() == st.candidates.tobytes()
        ref = eng.debug_stage(sgb.STAGE_REFINED)
        for f in ("x", "y", "response", "octave", "layer"):
            assert np.array_equal(ref[f], st.refined[f]), f
        m = match(st.keypoints, st.descriptors, kps, desc)
        assert len(m.pairs) >= MATCH_RATE * len(st.keypoints), m.summary()
    out = sgb.Batch(sgb.Sift.new(*args(sigma))).detect_and_compute([img, synth_image(8, 130, 90), img[:, ::-1].copy()])
    assert np.array_equal(out[0][0], kps) and np.array_equal(out[0][1], desc)
    one = eng.detect_and_compute(synth_image(8, 130, 90))
    assert np.array_equal(out[1][0], one[0]) and np.array_equal(out[1][1], one[1])


def test_dense_case_overfills_a_list(oracle_mod):
    st = oracle_mod.stages(noise(384, 260), oracle_mod.params(*args(0.55)))
    c = st.candidates[st.candidates["octave"] == 0]
    nw, h = 12, 260
    w = ((c["layer"] - 1) * h + c["y"].astype(int)) * nw + c["x"].astype(int) // 32
    per_tile = np.bincount(w // 512)
    assert per_tile.max() > 1024 and len(c) > max(1024, 3 * h * nw * 32 // 64)
