"""The table of orientation bins rests on two facts about byte differences,
checked here over all of them: off the axes no pair's angle is near a bin edge
(so no rounding of the reference's f32 sequence can move its bin), and on the
axes the f32 sequence gives the bins that the table holds."""
import numpy as np

PI2 = np.float32(2) * np.float32(np.pi)


def bin_positions(gx, gy):
    a = np.arctan2(gy, gx)
    return np.where(a < 0, a + 2 * np.pi, a) * 36 / (2 * np.pi)


def test_bins_are_sure_off_the_axes():
    lut = np.arange(256, dtype=np.float32) / np.float32(255)
    d = np.arange(256)[:, None] - np.arange(256)[None, :]
    diff = (lut[:, None] - lut[None, :]).astype(np.float64)
    # the smallest and largest f32 difference that each byte difference has
    lo, hi = np.full(511, np.inf), np.full(511, -np.inf)
    np.minimum.at(lo, d.ravel() + 255, diff.ravel())
    np.maximum.at(hi, d.ravel() + 255, diff.ravel())
    i = np.arange(-255, 256)
    off_axis = (i[:, None] != 0) & (i[None, :] != 0)
    want = np.floor(bin_positions(i[None, :] / 255.0, i[:, None] / 255.0))[off_axis]
    # atan2f to 4 ulp of pi, the wrap, the product and the quotient: below 2e-5 bins
    for x in (lo, hi):
        for y in (lo, hi):
            b = bin_positions(x[None, :], y[:, None])[off_axis]
            assert np.array_equal(np.floor(b), want)
            assert np.abs(b - np.rint(b)).min() > 6e-5


def test_axis_bins_by_the_f32_sequence():
    for a, want in ((0.0, 0), (np.pi / 2, 9), (np.pi, 18), (-np.pi / 2, 26)):
        an = np.float32(a)
        an = an + PI2 if an < 0 else an
        assert int(np.floor(an * np.float32(36) / PI2)) == want


def test_division_by_three():
    """v * fl(1/3) with one fused correction is the IEEE quotient (in rational arithmetic)."""
    from fractions import Fraction
    rng = np.random.default_rng(3)
    v = np.concatenate([rng.random(3000), 10.0 ** rng.uniform(-20, 6, 3000), np.arange(0, 2000)]).astype(np.float32)
    third = np.float32(1) / np.float32(3)
    for x in v:
        q = np.float32(x * third)
        r = np.float32(float(Fraction(float(x)) - 3 * Fraction(float(q))))  # exact: the fused residual is representable
        got = np.float32(float(Fraction(float(r)) * Fraction(float(third)) + Fraction(float(q))))
        assert got == np.float32(x) / np.float32(3)
