"""Descriptor matching where its split over CTAs, its queues and its candidate
lists can go wrong: one tile per CTA, one query tile over many CTAs, many
query tiles in one CTA, rows past the tiles, every row the same, descending
distances (every column a new best), other scales, rows that are not finite,
host rows on any address. Against the float64 oracle with the bound of the
other matching tests, scaled by the squared norms."""
import numpy as np
import pytest

from oracle.match import match

pytestmark = pytest.mark.gpu

GAP = 1e-5  # of squared distances of unit rows


@pytest.fixture(scope="module")
def eng(built_lib):
    import sift_wgpu_gb300 as sg
    with sg.Engine() as e:
        yield e


def rows(rng, n):
    x = np.abs(rng.standard_normal((n, 128))).astype(np.float32)
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def check(got, q, t, unit=1.0):
    gap = GAP * unit
    i1, _, i2, _, third, d2 = match(q, t)
    with np.errstate(invalid="ignore"):
        sure1 = d2[:, 1] - d2[:, 0] > gap
        sure2 = sure1 & (third - d2[:, 1] > gap)
    assert np.array_equal(got["train_idx"][sure1], i1[sure1])
    assert np.array_equal(got["second_idx"][sure2], i2[sure2])
    assert np.allclose(got["distance"].astype(np.float64) ** 2, d2[:, 0], atol=gap, rtol=0)
    if len(t) > 1:
        assert np.allclose(got["second_distance"].astype(np.float64) ** 2, d2[:, 1], atol=gap, rtol=0)


@pytest.mark.parametrize("nq,nt", [(128, 128), (129, 127), (1, 20000), (20000, 1), (3000, 130), (257, 3000), (5000, 128), (2500, 5000)])
def test_splits(eng, nq, nt):
    rng = np.random.default_rng(nq + nt)
    q, t = rows(rng, nq), rows(rng, nt)
    check(eng.match(q, t), q, t)


@pytest.mark.parametrize("scale", [512.0, 1e-3])
def test_other_scales(eng, scale):
    rng = np.random.default_rng(1)
    q, t = scale * rows(rng, 300), scale * rows(rng, 2000)
    check(eng.match(q, t), q, t, scale * scale)


def test_all_rows_the_same(eng):
    q = rows(np.random.default_rng(2), 1)
    got = eng.match(np.repeat(q, 200, 0), np.repeat(q, 5000, 0))
    assert np.all(got["train_idx"] == 0) and np.all(got["second_idx"] == 1)


def test_every_column_a_new_best(eng):
    rng = np.random.default_rng(3)
    a, b = rows(rng, 2)
    s = np.linspace(1, 0, 4000, dtype=np.float32)[:, None]
    t = (1 - s) * a + s * b  # nearer and nearer to a
    q = np.repeat(a[None], 140, 0)
    check(eng.match(q, t), q, t)
    check(eng.match(q, t[::-1].copy()), q, t[::-1])


def test_rows_that_are_not_finite(eng):
    rng = np.random.default_rng(4)
    q, t = rows(rng, 300), rows(rng, 1000)
    bad_t, bad_q = [0, 5, 127, 128, 999], [3, 130]
    t[bad_t[:3], 7] = np.nan
    t[bad_t[3:], 9] = np.inf
    q[bad_q[0], 0] = np.nan
    q[bad_q[1], 1] = np.inf
    got = eng.match(q, t)
    fine_q = np.setdiff1d(np.arange(300), bad_q)
    fine_t = np.setdiff1d(np.arange(1000), bad_t)
    want = eng.match(q[fine_q], t[fine_t])
    assert np.array_equal(got["train_idx"][fine_q], fine_t[want["train_idx"]])
    assert np.array_equal(got["second_idx"][fine_q], fine_t[want["second_idx"]])
    assert got["distance"][fine_q].tobytes() == want["distance"].tobytes()
    assert got["train_idx"][bad_q[0]] == -1 and np.isinf(got["distance"][bad_q[0]])


def test_host_rows_on_any_address(eng):
    rng = np.random.default_rng(5)
    q, t = rows(rng, 200), rows(rng, 700)
    want = eng.match(q, t)
    buf = np.zeros(t.size + q.size + 8, np.float32)
    for off in (0, 1, 2, 3):
        tv = buf[off:off + t.size].reshape(t.shape)
        tv[:] = t
        qv = buf[off + t.size:off + t.size + q.size].reshape(q.shape)
        qv[:] = q
        assert eng.match(qv, tv).tobytes() == want.tobytes()
