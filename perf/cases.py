"""The work that users of this framework have it do, as cases to be timed.

Single frames from a thumbnail to 4096 x 4096 through every host entry (owned
results, views, keypoints alone, colour), the three storage modes, other scale
counts and strided crops, batches of uneven images, the server on a mixed
queue, and descriptor matching. Frames are seeded scenes of blobs, rectangles
and noise at the density of the benchmark's images (200 blobs and 40
rectangles per 512 x 512). An engine is kept from frame to frame, as a program
that works through frames keeps it; every state has frames of its own.

`exact` follows the algorithm's definition: the levels are whole numbers by
definition (every blur pass and resize rounds to u8 from f32 sums in tap
order), and all that is computed from them is in 64 bits.
"""
import math

import numpy as np
import torch

import sift_wgpu_gb300 as sg
from sift_wgpu_gb300 import _capi

DENSITY = {2: 0.0019, 3: 0.0068, 4: 0.0100}  # oriented keypoints per pixel of these scenes, by intervals per octave
DESC = 128


def listed():
    one = dict(kind="frame", api="owned", storage="u8", octaves=4, intervals=3)
    return [
        # a thumbnail or a tracked patch: launches and latency
        dict(one, name="thumb_160x120", width=160, height=120),
        # a camera frame
        dict(one, name="vga_640x480", width=640, height=480),
        # keypoints alone (Sift.detect), 720p
        dict(one, name="detect_720p", api="detect", width=1280, height=720),
        # a crop of a larger frame (odd sides, rows not aligned), finer scales, f16 levels, results read in place
        dict(one, name="crop_1003x757_s4", api="crop", storage="f16", octaves=5, intervals=4, width=1003, height=757),
        # the headline workload: one 1080p frame, results owned by the caller
        dict(one, name="hd_1080p", width=1920, height=1080),
        # the same as a video loop runs it: pinned frames, results read in place, f32 levels
        dict(one, name="hd_pinned_f32", api="pinned", storage="f32", width=1920, height=1080),
        # an RGBA screenshot or decoded picture
        dict(one, name="rgba_1600x900", api="rgba", width=1600, height=900),
        # the large-image workload (aerial, scans): 4096 x 4096 with six octaves
        dict(one, name="large_4096", octaves=6, width=4096, height=4096),
        # a folder of uneven pictures in one run
        dict(name="batch_12", kind="batch", count=12, low=320, high=1600, pick=5, octaves=4),
        # a server's queue of mixed resolutions
        dict(name="serve_16", kind="serve", count=16, pick=4),
        # frame-to-frame matching of two 1080p descriptor sets
        dict(name="match_14k", kind="match", queries=14671, train=14747),
        # a small model against a frame
        dict(name="match_small", kind="match", queries=611, train=2203),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["frame"] * 7 + ["batch", "match", "match", "serve"])
    if kind == "match":
        return dict(kind=kind, queries=_spread(rng, 3, 14600), train=_spread(rng, 3, 14700))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), low=200, high=_spread(rng, 320, 1700), pick=rng.randint(0, 999), octaves=rng.randint(3, 6))
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(4, 16), pick=rng.randint(0, 999))
    return dict(kind=kind, api=rng.choice(["owned", "owned", "pinned", "detect", "crop", "rgba"]), storage=rng.choice(["u8", "u8", "f16", "f32"]),
                octaves=rng.randint(2, 6), intervals=rng.choice([3, 3, 2, 4]), width=_spread(rng, 96, 3600), height=_spread(rng, 96, 3600))


# ---- inputs -----------------------------------------------------------------


def _scene(width, height, seed):
    """A seeded u8 scene as a host array: blobs over a grey ground, rectangles over them, noise."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    area = width * height / (512.0 * 512.0)
    n, m = max(1, round(200 * area)), max(1, round(40 * area))
    b = u(n, 4)
    sigma = 2.0 + 18.0 * b[:, 2:3]
    ex = torch.exp(-((torch.arange(width, device="cuda") - b[:, 0:1] * width) ** 2) / (2 * sigma * sigma))
    ey = torch.exp(-((torch.arange(height, device="cuda") - b[:, 1:2] * height) ** 2) / (2 * sigma * sigma))
    img = 128.0 + (ey * (180.0 * b[:, 3:4] - 90.0)).T @ ex
    del ex, ey
    for x, y, w, h, v in u(m, 5).cpu().tolist():
        x, y = int(x * width), int(y * height)
        img[y:y + 8 + int(89 * h), x:x + 8 + int(89 * w)] = math.floor(256 * v)
    img += 3.0 * torch.randn(height, width, generator=g, device="cuda")
    return torch.floor(img.clamp_(0, 255) + 0.5).to(torch.uint8).cpu().numpy()


def _descriptors(n, seed):
    """Rows as a descriptor's: 4 x 4 x 8 sums of few strong directions, clipped at 0.2 and of unit length."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.rand(n, DESC, generator=g, device="cuda") ** 4
    for _ in range(2):
        v = (v / v.norm(dim=1, keepdim=True)).clamp_(max=0.2)
    return v / v.norm(dim=1, keepdim=True)


def _match_rows(case, seed):
    """Query and train rows; half of the queries are train rows seen again with noise."""
    t = _descriptors(case["train"], 2 * seed + 1)
    q = _descriptors(case["queries"], 2 * seed + 2)
    k = min(case["train"], case["queries"] // 2)
    q[:k] = (t[:k] + 0.02 * (q[:k] - q[:k].mean())).clamp_(min=0)
    q[:k] /= q[:k].norm(dim=1, keepdim=True)
    return q.cpu().numpy(), t.cpu().numpy()


def _sift(case):
    return sg.Sift(num_octaves=case.get("octaves", 4), num_intervals=case.get("intervals", 3))


def _sides(case):
    """(width, height) of every image of a batch or a queue."""
    r = np.random.default_rng(case["pick"])
    if case["kind"] == "serve":
        mix = [(640, 480)] * 4 + [(1280, 720)] * 3 + [(1920, 1080)] * 2 + [(3840, 2160)]
        return [mix[int(i)] for i in r.integers(0, len(mix), case["count"])]
    return [(int(w), int(h)) for w, h in r.integers(case["low"], case["high"] + 1, (case["count"], 2))]


_kept = {}  # the engines, batches and servers that a program keeps from frame to frame


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _pixels(case, seed):
    w, h = case["width"], case["height"]
    if case["api"] == "rgba":
        s = [_scene(w, h, 3 * seed + k) for k in range(3)]
        return np.ascontiguousarray(np.stack(s + [np.full_like(s[0], 255)], axis=2))
    if case["api"] == "crop":
        return _scene(w + 29, h + 13, seed)[7:7 + h, 11:11 + w]
    return _scene(w, h, seed)


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "match":
        s["query"], s["train"] = _match_rows(case, seed)
        s["engine"] = _keep("match", sg.Engine)
    elif case["kind"] == "frame":
        s["image"] = _pixels(case, seed)
        if case["api"] == "pinned":
            s["pinned"] = torch.from_numpy(s["image"]).pin_memory()
            s["image"] = s["pinned"].numpy()
        key = (case["octaves"], case["intervals"], case["storage"], case["width"], case["height"])
        s["engine"] = _keep(key, lambda: sg.Engine(_sift(case), storage=case["storage"]))
    else:
        s["images"] = [_scene(w, h, 1000 * seed + k) for k, (w, h) in enumerate(_sides(case))]
        if case["kind"] == "batch":
            s["batch"] = _keep(str(sorted(case.items())), lambda: sg.Batch(_sift(case)))
        else:
            s["server"] = _keep("server", sg.Server)
    return s


# ---- one pass ---------------------------------------------------------------


def _expected(case, width, height):
    """About how many keypoints a scene has (one of three blended scenes, with a lower noise, has more)."""
    return (1.3 if case.get("api") == "rgba" else 1.0) * DENSITY[case.get("intervals", 3)] * width * height


def _whole(rows, expected):
    """All of a result whose length depends on the image, as two views whose length does not: the first and the
    last rows, which overlap (padded with zeros where the image has far fewer than expected)."""
    m = int(0.72 * expected) + 12
    n = len(rows)
    if n < m:
        return [np.concatenate([rows, np.zeros((m - n,) + rows.shape[1:], rows.dtype)])] * 2
    if n > 2 * m:
        raise ValueError("%d keypoints where about %d are expected" % (n, expected))
    return [rows[:m], rows[n - m:]]


def _columns(kps, expected):
    return dict({f: _whole(kps[f], expected) for f in ("x", "y", "size", "angle", "response", "octave", "layer")}, count=len(kps))


def _result(case, kps, desc=None):
    expected = _expected(case, case["width"], case["height"])
    out = _columns(kps, expected)
    if desc is not None:
        out["descriptors"] = _whole(desc, expected)
    return out


def _results(case, results):
    sides = [_expected(case, w, h) for w, h in _sides(case)]
    out = _columns(np.concatenate([k for k, _ in results]), sum(sides))
    out["descriptors"] = [_whole(d, e) for (_, d), e in zip(results, sides)]
    out["counts"] = np.array([len(k) for k, _ in results], dtype=np.int32)
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "match":
        m = state["engine"].match(state["query"], state["train"])
        return {f: m[f] for f in ("train_idx", "distance", "second_idx", "second_distance")}
    if case["kind"] == "batch":
        return _results(case, state["batch"].detect_and_compute(state["images"], copy=False))
    if case["kind"] == "serve":
        return _results(case, state["server"].detect_batch(state["images"], copy=False))
    e, api = state["engine"], case["api"]
    if api == "detect":
        return _result(case, e.detect(state["image"]))
    if api in ("pinned", "crop"):
        return _result(case, *e.detect_and_compute_view(state["image"]))
    return _result(case, *e.detect_and_compute(state["image"]))


# ---- what a pass cannot do without --------------------------------------------


def _blur_sigmas(case):
    """(base blur, [[blur of level 1 ..] of each octave]) in f32."""
    f, s = np.float32, case.get("intervals", 3)
    sigma, assumed = f(1.6), f(0.5)
    k, target = np.power(f(2), f(1) / f(s)), []
    for i in range(s + 3):
        a, r, n = k, f(1), i
        while True:  # powers by repeated squaring
            if n & 1:
                r = f(r * a)
            n >>= 1
            if n == 0:
                break
            a = f(a * a)
        target.append(f(sigma * r))
    rows = []
    for o in range(case.get("octaves", 4)):
        scale = f(2.0 ** o)
        t = [f(x * scale) for x in target]
        rows.append([f(np.sqrt(f(f(b * b) - f(a * a)))) for a, b in zip(t, t[1:])])
    return f(np.sqrt(f(f(sigma * sigma) - f(assumed * assumed)))), rows


def _frame_work(case, w, h, desc, channels=1):
    base, rows = _blur_sigmas(case)
    n = _expected(case, w, h)
    flops, ow, oh = 4.0 * w * h * (2 * math.ceil(2 * base) + 1), w, h
    for row in rows:
        taps = sum(2 * math.ceil(2 * float(b)) + 1 for b in row)
        flops += ow * oh * (4.0 * taps + 54.0 * len(row) + 24.0)  # two passes, differences and 26 comparisons, resize
        ow, oh = ow // 2, oh // 2
    flops += n * (600 * 40.0 + (1500 * 80.0 if desc else 0.0))  # orientation and descriptor samples
    return w * h * channels + n * (28 + (4 * DESC if desc else 0)), flops


def work(case):
    if case["kind"] == "match":
        q, t = case["queries"], case["train"]
        return {"bytes": 4.0 * DESC * (q + t) + 16.0 * q, "flops": 2.0 * DESC * q * t}
    if case["kind"] == "frame":
        b, f = _frame_work(case, case["width"], case["height"], case["api"] != "detect", 4 if case["api"] == "rgba" else 1)
        return {"bytes": b, "flops": f}
    every = [_frame_work(case, w, h, True) for w, h in _sides(case)]
    return {"bytes": sum(b for b, _ in every), "flops": sum(f for _, f in every)}


# ---- the same in 64 bits -------------------------------------------------------


def _blur(img, sigma):
    """One level from another: two passes of f32 sums in tap order, each ending in a truncated u8."""
    f = np.float32
    r = int(math.ceil(f(2) * sigma))
    c = f(f(1) / f(np.sqrt(f(f(2) * f(math.pi))) * sigma))
    x = np.arange(r + 1, dtype=f)
    half = (c * np.exp((-(x * x) / f(f(2) * f(sigma * sigma))).astype(np.float64)).astype(f)).astype(f)
    k = np.concatenate([half[:0:-1], half])
    for axis in (1, 0):
        n = img.shape[axis]
        p = np.pad(img, [(r, r) if a == axis else (0, 0) for a in (0, 1)], mode="edge").astype(f)
        acc = np.zeros(img.shape, f)
        for i in range(2 * r + 1):
            acc += (p[:, i:i + n] if axis else p[i:i + n]) * k[i]
        img = np.clip(np.trunc(acc), 0, 255).astype(np.uint8)
    return img


def _taps(src, dst):
    """First source index, f32 weights (padded with 0) of each output of the Lanczos3 resize."""
    f = np.float32
    ratio = f(src) / f(dst)
    scale = max(ratio, f(1))
    support = f(f(3) * scale)
    rows = []
    for o in range(dst):
        at = f((f(o) + f(0.5)) * ratio)
        left = min(max(int(math.floor(f(at - support))), 0), src - 1)
        right = max(left + 1, min(int(math.ceil(f(at + support))), src))
        t = ((np.arange(left, right).astype(f) - f(at - f(0.5))) / scale).astype(f)

        def sinc(v):
            a = (v * f(math.pi)).astype(f)
            return np.where(v == 0, f(1), np.sin(a.astype(np.float64)).astype(f) / np.where(v == 0, f(1), a)).astype(f)

        w = np.where(np.abs(t) < 3, sinc(t) * sinc((t / f(3)).astype(f)), f(0)).astype(f)
        total = f(0)
        for v in w:
            total = f(total + v)
        rows.append((left, (w / total).astype(f)))
    most = max(len(w) for _, w in rows)
    return np.array([a for a, _ in rows]), np.stack([np.pad(w, (0, most - len(w))) for _, w in rows])


def _halve(img):
    h, w = img.shape
    left, wt = _taps(h, h // 2)
    t = np.zeros((h // 2, w), np.float32)
    for i in range(wt.shape[1]):
        t += img[np.minimum(left + i, h - 1)].astype(np.float32) * wt[:, i:i + 1]
    left, wt = _taps(w, w // 2)
    u = np.zeros((h // 2, w // 2), np.float32)
    for i in range(wt.shape[1]):
        u += t[:, np.minimum(left + i, w - 1)] * wt[:, i]
    return np.floor(np.clip(u, 0, 255) + np.float32(0.5)).astype(np.uint8)


def _offsets(c, dtype):
    """Gradient, Hessian and the solved offset of 3 x 3 x 3 neighbourhoods c[:, layer, y, x], by Cramer's rule."""
    c = c.astype(dtype)
    two, four = dtype(2), dtype(4)
    v = c[:, 1, 1, 1]
    g = np.stack([(c[:, 1, 1, 2] - c[:, 1, 1, 0]) / two, (c[:, 1, 2, 1] - c[:, 1, 0, 1]) / two, (c[:, 2, 1, 1] - c[:, 0, 1, 1]) / two])
    xx = c[:, 1, 1, 2] + c[:, 1, 1, 0] - two * v
    yy = c[:, 1, 2, 1] + c[:, 1, 0, 1] - two * v
    ss = c[:, 2, 1, 1] + c[:, 0, 1, 1] - two * v
    xy = (c[:, 1, 2, 2] - c[:, 1, 2, 0] - c[:, 1, 0, 2] + c[:, 1, 0, 0]) / four
    xs = (c[:, 2, 1, 2] - c[:, 2, 1, 0] - (c[:, 0, 1, 2] - c[:, 0, 1, 0])) / four
    ys = (c[:, 2, 2, 1] - c[:, 2, 0, 1] - (c[:, 0, 2, 1] - c[:, 0, 0, 1])) / four
    b = -g
    det = xx * (yy * ss - ys * ys) - xy * (xy * ss - ys * xs) + xs * (xy * ys - yy * xs)
    dx = b[0] * (yy * ss - ys * ys) - xy * (b[1] * ss - ys * b[2]) + xs * (b[1] * ys - yy * b[2])
    dy = xx * (b[1] * ss - ys * b[2]) - b[0] * (xy * ss - ys * xs) + xs * (xy * b[2] - b[1] * xs)
    ds = xx * (yy * b[2] - b[1] * ys) - xy * (xy * b[2] - b[1] * xs) + b[0] * (xy * ys - yy * xs)
    with np.errstate(all="ignore"):
        return v, g, (xx, yy, xy), np.abs(det) >= dtype(1e-10), np.stack([dx / det, dy / det, ds / det])


def _refined(dog, octave, case):
    """(x, y, size, response, layer) rows of one octave's extrema that pass, in (layer, y, x) order."""
    f, s, border = np.float32, case["intervals"], 5
    n, h, w = dog.shape
    if h <= 2 * border or w <= 2 * border:
        return np.zeros((0, 5))
    inside = lambda l, dy, dx: dog[l, border + dy:h - border + dy, border + dx:w - border + dx]  # noqa: E731
    at = []
    for l in range(1, s + 1):
        v = inside(l, 0, 0)
        high, low = np.ones(v.shape, bool), np.ones(v.shape, bool)
        for k in range(27):
            if k != 13:
                o = inside(l + k // 9 - 1, k // 3 % 3 - 1, k % 3 - 1)
                high &= v > o
                low &= v < o
        y, x = np.nonzero(high | low)
        at.append(np.stack([np.full(len(y), l), y + border, x + border]))
    at = np.concatenate(at, axis=1)
    out, alive = {}, np.arange(at.shape[1])
    cube = np.stack(np.meshgrid([-1, 0, 1], [-1, 0, 1], [-1, 0, 1], indexing="ij"))[:, None]
    for _ in range(5):
        l, y, x = at[:, alive]
        ok = (l >= 1) & (l < n - 1) & (x >= 1) & (x < w - 1) & (y >= 1) & (y < h - 1)
        alive = alive[ok]
        if not len(alive):
            break
        p = at[:, alive]
        c = dog[tuple(p[:, :, None, None, None] + cube)]
        v, g, (xx, yy, xy), ok, off = _offsets(c, f)
        near = ok & (np.abs(off) < f(0.5)).all(axis=0)
        with np.errstate(all="ignore"):
            val = v + f(0.5) * (g[0] * off[0] + g[1] * off[1] + g[2] * off[2])
            det = xx * yy - xy * xy
            keep = near & ~(np.abs(val) < f(f(0.04) / f(s))) & (det > 0) & ((xx + yy) * (xx + yy) / det < f(f(11) * f(11) / f(10)))
        if keep.any():
            v, g, _, _, o = _offsets(c[keep], np.float64)
            val = v + 0.5 * (g * o).sum(axis=0)
            lf = p[0, keep] + o[2]
            size = 1.6 * 2.0 ** (octave + lf / s)
            rows = np.stack([(p[2, keep] + o[0]) * 2.0 ** octave, (p[1, keep] + o[1]) * 2.0 ** octave, size, val, np.floor(lf + 0.5)], axis=1)
            out.update(zip(alive[keep].tolist(), rows))
        go = ok & ~near
        alive, off = alive[go], off[::-1, go]
        to = (at[:, alive].astype(f) + off).astype(np.float64)
        at[:, alive] = np.clip(np.sign(to) * np.floor(np.abs(to) + 0.5), -1e6, 1e6).astype(np.int64)  # half away from zero
        inside_layers = (at[0, alive] >= 0) & (at[0, alive] < n)
        alive = alive[inside_layers]
    return np.array([out[i] for i in sorted(out)]).reshape(-1, 5)


def _angles(g, x, y, so):
    """The orientation peaks of one keypoint, in bin order."""
    h, w = g.shape
    r = int(math.floor(4.5 * so + 0.5))
    d = np.arange(-r, r + 1)
    away = lambda v: (np.sign(v) * np.floor(np.abs(v) + 0.5)).astype(int)  # noqa: E731
    xi, yi = (away(np.float32(v) + d.astype(np.float32)) for v in (x, y))
    mx, my = (xi >= 1) & (xi < w - 1), (yi >= 1) & (yi < h - 1)
    xi, yi, dx, dy = xi[mx], yi[my], d[mx], d[my]
    if not len(xi) or not len(yi):
        return []
    gx = g[np.ix_(yi, xi + 1)] - g[np.ix_(yi, xi - 1)]
    gy = g[np.ix_(yi + 1, xi)] - g[np.ix_(yi - 1, xi)]
    wt = np.exp(-(dx[None, :] ** 2 + dy[:, None] ** 2) / (2 * (1.5 * so) ** 2))
    a, turn = np.arctan2(gy, gx).astype(np.float32), np.float32(2 * math.pi)  # the bin is by definition f32's: many angles lie on an edge
    b = np.floor(np.where(a < 0, a + turn, a) * np.float32(36) / turn).astype(int) % 36
    hist = np.bincount(b.ravel(), (np.hypot(gx, gy) * wt).ravel(), 36)
    for _ in range(2):
        hist = (np.roll(hist, 1) + hist + np.roll(hist, -1)) / 3
    prv, nxt = np.roll(hist, 1), np.roll(hist, -1)
    found = []
    for k in np.nonzero((hist >= 0.8 * hist.max()) & (hist > prv) & (hist > nxt))[0]:
        den = prv[k] - 2 * hist[k] + nxt[k]
        v = (k + 0.5 + (0.5 * (prv[k] - nxt[k]) / den if abs(den) > 1e-5 else 0.0)) * 2 * math.pi / 36
        v %= 2 * math.pi
        found.append(v - 2 * math.pi if v > math.pi else v)
    return found


def _descriptor(g, x, y, so, angle):
    h, w = g.shape
    bw = 3 * so
    rad = int(math.ceil(2 * bw * math.sqrt(2) - 1e-6))
    py, px = (v.ravel() for v in np.mgrid[-rad:rad + 1, -rad:rad + 1].astype(np.float64))
    ca, sa = math.cos(angle), math.sin(angle)
    xb, yb = (ca * px + sa * py) / bw + 1.5, (ca * py - sa * px) / bw + 1.5
    ok = (xb > -1) & (xb < 4) & (yb > -1) & (yb < 4) & (x + px >= 0) & (x + px < w - 1) & (y + py >= 0) & (y + py < h - 1)
    px, py, xb, yb = px[ok], py[ok], xb[ok], yb[ok]

    def at(xs, ys):
        x0, y0 = np.floor(xs).astype(int), np.floor(ys).astype(int)
        dx, dy = xs - x0, ys - y0
        x0, x1, y0, y1 = np.clip(x0, 0, w - 1), np.clip(x0 + 1, 0, w - 1), np.clip(y0, 0, h - 1), np.clip(y0 + 1, 0, h - 1)
        return (g[y0, x0] * (1 - dx) + g[y0, x1] * dx) * (1 - dy) + (g[y1, x0] * (1 - dx) + g[y1, x1] * dx) * dy

    xs, ys = x + px, y + py
    gx, gy = at(xs + 1, ys) - at(xs - 1, ys), at(xs, ys + 1) - at(xs, ys - 1)
    wm = np.hypot(gx, gy) * np.exp(-(px * px + py * py) / (2 * (2 * bw) ** 2))
    ab = (np.arctan2(gy, gx) - angle) % (2 * math.pi) * 8 / (2 * math.pi)
    x0, y0, a0 = np.floor(xb).astype(int), np.floor(yb).astype(int), np.floor(ab).astype(int)
    fx, fy, fa = xb - x0, yb - y0, ab - a0
    hist = np.zeros(6 * 6 * 8)
    for k in range(8):
        i, j, l = k & 1, k >> 1 & 1, k >> 2
        wt = wm * (fx if i else 1 - fx) * (fy if j else 1 - fy) * (fa if l else 1 - fa)
        hist += np.bincount(((y0 + 1 + j) * 6 + x0 + 1 + i) * 8 + (a0 + l) % 8, wt, 288)
    d = hist.reshape(6, 6, 8)[1:5, 1:5].ravel()
    if np.linalg.norm(d) >= 1e-8:
        d = np.minimum(d / np.linalg.norm(d), 0.2)
        d = d / np.linalg.norm(d)
    return d


def exact(case, seed):
    if case["kind"] == "match":
        q, t = (torch.from_numpy(v).cuda().double() for v in _match_rows(case, seed))
        i = torch.cat([((t * t).sum(1) - 2 * p @ t.T).topk(2, largest=False).indices for p in q.split(4096)])
        near = [(q - t[i[:, k]]).norm(dim=1).cpu().numpy() for k in range(2)]
        return {"train_idx": None, "distance": near[0], "second_idx": None, "second_distance": near[1]}
    if case["kind"] != "frame" or case["width"] * case["height"] > 1_000_000 or case["api"] == "rgba":
        return None
    with_desc = case["api"] != "detect"
    img, (base, rows) = _pixels(case, seed), _blur_sigmas(case)
    cur, kps, desc = _blur(img, base), [], []
    for o, row in enumerate(rows):
        if min(cur.shape) < 1:
            break
        levels = [cur]
        for b in row:
            levels.append(_blur(levels[-1], b))
        cur = _halve(levels[case["intervals"]]) if min(levels[0].shape) > 1 else levels[0][:0, :0]
        unit = [v.astype(np.float32) / np.float32(255) for v in levels]
        fine = [v.astype(np.float64) / 255 for v in levels]
        for x, y, size, val, layer in _refined(np.stack([b - a for a, b in zip(unit, unit[1:])]), o, case):
            g = fine[int(min(max(layer, 0), case["intervals"] + 2))]
            x0, y0, so = (float(np.float32(v)) / 2 ** o for v in (x, y, size))  # a keypoint's fields are f32: windows end by them
            for a in _angles(g, x0, y0, so):
                kps.append((x, y, size, a, val))
                if with_desc:
                    desc.append(_descriptor(g, x0, y0, so, a))
    k = np.array(kps).reshape(-1, 5)
    expected = _expected(case, case["width"], case["height"])
    out = {f: _whole(k[:, i], expected) for i, f in enumerate(("x", "y", "size", "angle", "response"))}
    out.update(octave=None, layer=None, count=None)
    if with_desc:
        out["descriptors"] = _whole(np.array(desc).reshape(-1, DESC), expected)
    return out
