"""Performance cases of the tracker: what users run, at the sizes they run it.

Each case is one call (or the two calls that belong together) through the public entry points:
the Python functions `autorift`, `track` and `submit`, and the C ABI's device-resident entry
points (`ar_prepare`, `ar_track_device`, `ar_track_device_rotated`, `ar_multichip_device`) as a
program that keeps its pairs and point sets on the GPU calls them. Scenes are seeded: filtered
noise as the reference image, and its bicubic warp by a smooth motion field plus noise (and
no-data blobs, given as a mask) as the secondary.

Kinds:
  track     one pass of `ar_track_device` over a grid with jittered centres and integer priors,
            on a pair of any element type: the correlator itself;
  plain     `track` from host points on a small Float32 pair, results on the host;
  rotated   `ar_track_device_rotated`: the per-chip rotation search;
  points    `ar_prepare` of a raw pair, then a pass over a few thousand scattered points (the
            filters and the quantiser carry the time);
  search    `ar_prepare` and `ar_multichip_device` of a raw UInt16 pair: the default pipeline;
  batch     `ar_multichip_device` on a prepared UInt8 pair with a radius and a prior per point
            and chip sizes 16 to 128;
  autorift  the one-line call on host arrays: upload, prepare, search, results on the host;
  serve     a burst of requests of mixed sizes through the request loop (`submit`, `wait`).
"""

import ctypes
import math

import numpy as np
import torch

import __graft_entry__

ar = __graft_entry__.load_package()
L = ar._lib
DEV = "cuda"
UP = 64


def listed():
    return [
        # A handful of points re-tracked while someone waits: chip 16, a small window.
        dict(name="track_u8_small", kind="track", dtype="uint8", rows=512, cols=512, chip=16,
             radius=8, spacing=18, up=16, measure="zncc", holes=False),
        # The fine pass of the default pipeline over a whole scene (chip 32, radius 25).
        dict(name="track_u8_c32r25", kind="track", dtype="uint8", rows=4096, cols=4096, chip=32,
             radius=25, spacing=8, up=64, measure="zncc", holes=True),
        # Fast-moving ice: windows wider than 64 px, a ragged scene.
        dict(name="track_u8_c32r44", kind="track", dtype="uint8", rows=2047, cols=3001, chip=32,
             radius=44, spacing=16, up=64, measure="zncc", holes=True),
        # Unquantised highpass imagery, direct FP32 correlation (the plain method).
        dict(name="track_f32_c32r25", kind="track", dtype="float32", rows=2048, cols=2048,
             chip=32, radius=25, spacing=12, up=64, measure="zncc", holes=True),
        # Large chips on raw UInt16 imagery: split-BF16 tensor cores.
        dict(name="track_u16_c64r32", kind="track", dtype="uint16", rows=2500, cols=1999, chip=64,
             radius=32, spacing=24, up=64, measure="zncc", holes=False),
        # The smallest published configuration: two 512^2 Float32 images, 841 points, from host
        # arrays of points to host results.
        dict(name="plain_f32_512", kind="plain", rows=512, cols=512, chip=32, radius=25,
             spacing=16, up=64),
        # Rotating features: three chip rotations a point on quantised imagery.
        dict(name="rotated_u8_c32r25", kind="rotated", dtype="uint8", rows=1536, cols=1536,
             chip=32, radius=25, spacing=12, up=64, angles=3),
        # Filter and quantise a UInt16 scene, then track a few thousand stations on it.
        dict(name="points_u16_highpass", kind="points", dtype="uint16", rows=6001, cols=5003,
             filter="highpass", width=5, quantize=True, points=3000, chip=32, radius=16, up=64),
        # The same with the Wallis filter on Float32 imagery, left unquantised.
        dict(name="points_f32_wallis", kind="points", dtype="float32", rows=3000, cols=3000,
             filter="wallis", width=21, quantize=False, points=1000, chip=32, radius=12, up=64),
        # The headline: the default pipeline on a Sentinel-2 tile.
        dict(name="search_u16_10980", kind="search", rows=10980, cols=10980, chip=32, radius=25,
             spacing=8, up=64),
        # Radii in [4, 48] and priors per point, chip sizes 16 to 128.
        dict(name="batch_u8_2745", kind="batch", rows=2745, cols=2745, spacing=8, up=64),
        # A burst of requests as a service receives them.
        dict(name="serve_u16_mixed", kind="serve", requests=7, side=512, seed=5, up=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds: sizes log-uniform over the ranges, odd ones included."""
    kind = rng.choice(["track", "track", "track", "plain", "rotated", "points", "search", "batch",
                       "autorift", "serve"])
    rows = _log(rng, 500, 4200)
    cols = max(480, min(4500, int(rows * rng.uniform(0.7, 1.4))))
    up = rng.choice([16, 64, 64, 128])
    if kind == "track":
        dtype = rng.choice(["uint8", "uint8", "uint8", "float32", "uint16", "int16"])
        chip = rng.choice([16, 24, 32, 32, 48, 64, 96, 128])
        radius = _log(rng, 5, 50 if chip <= 64 else 32)
        cap = 2e12 if dtype == "uint8" else 4e11
        c = dict(kind=kind, dtype=dtype, rows=rows, cols=cols, chip=chip, radius=radius,
                 spacing=rng.choice([8, 11, 16, 20, 32]), up=up,
                 measure=rng.choice(["zncc", "zncc", "ncc"]), holes=rng.random() < 0.5)
        return _within(c, cap)
    if kind == "plain":
        n = _log(rng, 300, 900)
        return dict(kind=kind, rows=n, cols=n + rng.randrange(64), chip=rng.choice([16, 32]),
                    radius=rng.randrange(8, 30), spacing=rng.randrange(12, 30), up=up)
    if kind == "rotated":
        c = dict(kind=kind, dtype=rng.choice(["uint8", "uint8", "float32"]), rows=rows, cols=cols,
                 chip=rng.choice([16, 32, 32, 64]), radius=_log(rng, 6, 32), spacing=16, up=up,
                 angles=rng.choice([3, 3, 5]))
        return _within(c, 3e11)
    if kind == "points":
        return dict(kind=kind, dtype=rng.choice(["uint16", "uint16", "int16", "uint8", "float32"]),
                    rows=rows, cols=cols, filter=rng.choice(["highpass", "highpass", "wallis"]),
                    width=rng.choice([3, 5, 5, 9, 15, 21, 31]), quantize=rng.random() < 0.7,
                    points=_log(rng, 50, 4000), chip=rng.choice([16, 32]),
                    radius=rng.randrange(6, 26), up=up)
    if kind == "search":
        return dict(kind=kind, rows=rows, cols=cols, chip=rng.choice([16, 32, 32]),
                    radius=_log(rng, 8, 40), spacing=rng.choice([8, 12, 16, 32]), up=up)
    if kind == "batch":
        return dict(kind=kind, rows=rows, cols=cols, spacing=rng.choice([8, 12, 16, 21]), up=up)
    if kind == "autorift":
        n = _log(rng, 500, 2100)
        return dict(kind=kind, rows=n, cols=n + rng.randrange(128), chip=rng.choice([16, 32, 32]),
                    radius=_log(rng, 8, 30), spacing=rng.choice([8, 16, 32]), up=up)
    return dict(kind=kind, requests=rng.randrange(3, 12), side=rng.choice([300, 400, 512, 600]),
                seed=rng.randrange(1 << 20), up=up)


def _within(c, cap):
    """`c` with its spacing widened until the pass is within `cap` operations."""
    while c["spacing"] < 200 and _flops(c) > cap:
        c["spacing"] += 3
    return c


# ---------------------------------------------------------------------------------------------
# Scenes (on the GPU, from the seed alone)


def _noise(shape, gen):
    return torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32)


def _blur(a, sigma):
    """Separable Gaussian filter with wrap-around, as sums of shifted copies."""
    r = int(3 * sigma + 0.5)
    w = [math.exp(-0.5 * (k / sigma) ** 2) for k in range(-r, r + 1)]
    t = sum(w)
    for d in (0, 1):
        acc = torch.zeros_like(a)
        for k, v in zip(range(-r, r + 1), w):
            acc.add_(torch.roll(a, k, d), alpha=v / t)
        a = acc
    return a


def _motion(cols, rows, amp, rs):
    """Smooth motion (fx, fy) as sums of Gaussian bumps, zero at the borders; [cols, rows]."""
    x = torch.arange(cols, device=DEV, dtype=torch.float32)[:, None]
    y = torch.arange(rows, device=DEV, dtype=torch.float32)[None, :]
    fx = torch.zeros((cols, rows), device=DEV)
    fy = torch.zeros((cols, rows), device=DEV)
    for _ in range(6):
        cx, cy = rs.uniform(0.25, 0.75) * cols, rs.uniform(0.25, 0.75) * rows
        w = rs.uniform(0.06, 0.15) * min(rows, cols)
        m, ang = rs.uniform(0.4, 1.0) * amp, rs.uniform(0, 2 * math.pi)
        g = torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * w * w))
        fx.add_(g, alpha=m * math.cos(ang))
        fy.add_(g, alpha=m * math.sin(ang))
    b = 0.1 * min(rows, cols)
    t = torch.minimum(torch.minimum(x, cols - 1 - x) / b, torch.minimum(y, rows - 1 - y) / b)
    t = t.clamp(0, 1)
    m = max(float(fx.abs().max()), float(fy.abs().max()), 1e-6)
    return fx * t * (amp / m), fy * t * (amp / m)


def _texture_pair(rows, cols, amp, seed):
    """(reference, secondary, fx, fy), zero mean and unit deviation, [cols, rows] (column-major)."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    a = _blur(_noise((cols, rows), gen), 1.7)
    a = (a - a.mean()) / a.std()
    fx, fy = _motion(cols, rows, amp, np.random.RandomState(seed & 0x7FFFFFFF))
    x = torch.arange(cols, device=DEV, dtype=torch.float32)[:, None] - fx
    y = torch.arange(rows, device=DEV, dtype=torch.float32)[None, :] - fy
    grid = torch.stack([2 * y / (rows - 1) - 1, 2 * x / (cols - 1) - 1], dim=-1)[None]
    del x, y
    b = torch.nn.functional.grid_sample(a[None, None], grid, mode="bicubic",
                                        padding_mode="border", align_corners=True)[0, 0]
    del grid
    b = b + 0.02 * _noise((cols, rows), gen)
    return a, b, fx, fy


def _holes(rows, cols, seed):
    """Validity of the secondary: about 3 % of it no-data blobs; [cols, rows] bool."""
    rs = np.random.RandomState((seed + 17) & 0x7FFFFFFF)
    ok = torch.ones((cols, rows), dtype=torch.bool, device=DEV)
    x = torch.arange(cols, device=DEV)[:, None]
    y = torch.arange(rows, device=DEV)[None, :]
    for _ in range(max(1, int(0.03 * rows * cols / 8500))):
        r, cx, cy = rs.uniform(20, 80), rs.uniform(0, cols), rs.uniform(0, rows)
        x0, x1 = int(max(cx - r, 0)), int(min(cx + r + 1, cols))
        y0, y1 = int(max(cy - r, 0)), int(min(cy + r + 1, rows))
        ok[x0:x1, y0:y1] &= (x[x0:x1] - cx) ** 2 + (y[:, y0:y1] - cy) ** 2 > r * r
    return ok


_TORCH = {"uint8": torch.uint8, "uint16": torch.uint16, "int16": torch.int16}


def _digitise(t, dtype, raw):
    """The values of a unit-deviation image as stored imagery: raw counts (mean 8000, deviation
    1500; 8 bits: three deviations over the range), or a filter's signed Float32 output."""
    if dtype == "float32":
        return 0.5 + 0.1 * t if raw else 1500 * t
    if dtype == "uint8":
        return torch.round(127.5 + 42.5 * t).clamp(0, 255)
    if dtype == "int16":
        return torch.round(1500 * t).clamp(-32768, 32767)
    return torch.round(8000 + 1500 * t).clamp(0, 65535)


def _images(rows, cols, dtype, seed, *, raw, holes, amp):
    """Device images [cols, rows] of `dtype`, the secondary's validity (or None), the motion."""
    a, b, fx, fy = _texture_pair(rows, cols, amp, seed)
    ok = _holes(rows, cols, seed) if holes else None
    a, b = _digitise(a, dtype, raw), _digitise(b, dtype, raw)
    if ok is not None:
        b = b * ok
    if dtype != "float32":
        a, b = (t.to(torch.int32).to(_TORCH[dtype]) for t in (a, b))
    return a, b, ok, fx, fy


def _host(t):
    """[cols, rows] on the device -> the column-major [rows, cols] host array."""
    return None if t is None else t.cpu().numpy().T


def _pair(a, b, ok, ctx):
    """The device pair (uploaded) of images and the secondary's validity."""
    return ar.ImagePair(_host(a), _host(b), None, _host(ok)).device(ctx)


# ---------------------------------------------------------------------------------------------
# Point sets


def _grid_axis(n, chip, radius, spacing):
    m = chip // 2 + radius + 6
    return np.arange(m, n - m, spacing, dtype=np.float64)


def _grid_counts(c):
    return (len(_grid_axis(c["rows"], c["chip"], c["radius"], c["spacing"])),
            len(_grid_axis(c["cols"], c["chip"], c["radius"], c["spacing"])))


def _grid_points(c, seed, fx=None, fy=None):
    """A grid with centres jittered by up to half a pixel, integer priors within 3 px."""
    rs = np.random.RandomState((seed + 29) & 0x7FFFFFFF)
    ys = _grid_axis(c["rows"], c["chip"], c["radius"], c["spacing"])
    xs = _grid_axis(c["cols"], c["chip"], c["radius"], c["spacing"])
    x, y = (v.ravel(order="F") for v in np.meshgrid(xs, ys))
    n = x.size
    x, y = x + rs.uniform(-0.5, 0.5, n), y + rs.uniform(-0.5, 0.5, n)
    dx0, dy0 = rs.randint(-3, 4, n).astype(np.float64), rs.randint(-3, 4, n).astype(np.float64)
    return _fields(x, y, np.full(n, c["radius"]), dx0, dy0, c["chip"])


def _scattered(c, seed):
    rs = np.random.RandomState((seed + 31) & 0x7FFFFFFF)
    m, n = c["chip"] // 2 + c["radius"] + 6, c["points"]
    x, y = rs.uniform(m, c["cols"] - m, n), rs.uniform(m, c["rows"] - m, n)
    return _fields(x, y, np.full(n, c["radius"]), np.zeros(n), np.zeros(n), c["chip"])


def _fields(x, y, r, dx0, dy0, chip):
    i = lambda v: np.ascontiguousarray(v, dtype=np.int64)
    return dict(x=x, y=y, radius_x=i(r), radius_y=i(r), dx_prior=dx0, dy_prior=dy0,
                chip_size_x=i(np.full(x.size, chip)), chip_size_y=i(np.full(x.size, chip)))


def _device_points(f):
    """The `ar_points` struct over device copies of the fields; (struct, tensors it points at)."""
    cols = [torch.from_numpy(np.ascontiguousarray(f[k])).to(DEV) for k in ar.points.FIELDS]
    return L.ArPoints(*(t.data_ptr() for t in cols), cols[0].numel()), cols


def _outputs(n, search):
    o = [torch.zeros(n, dtype=torch.float32, device=DEV) for _ in range(3)]
    if search:
        return o + [torch.zeros(n, dtype=torch.int16, device=DEV),
                    torch.zeros(n, dtype=torch.uint8, device=DEV)]
    return o + [torch.zeros(n, dtype=torch.uint8, device=DEV)]


_NAMES = ("dx", "dy", "correlation", "searched")
_SEARCH_NAMES = ("dx", "dy", "correlation", "chip_size", "interpolated")
_ANGLES = {3: (-3.0, 0.0, 3.0), 5: (-6.0, -3.0, 0.0, 3.0, 6.0)}


def _measure(c):
    return L.AR_NCC if c.get("measure") == "ncc" else L.AR_ZNCC


def _point_fields(c, seed):
    return _scattered(c, seed) if c["kind"] == "points" else _grid_points(c, seed)


def _track_images(c, seed):
    kind = c["kind"]
    return _images(c["rows"], c["cols"], c.get("dtype", "float32"), seed,
                   raw=kind in ("plain", "points") or c.get("dtype") == "uint16",
                   holes=c.get("holes", kind == "points"), amp=min(4.0, 0.4 * c["radius"]))


def _points_params(c):
    pre = ar.Wallis(c["width"]) if c["filter"] == "wallis" else ar.Highpass(c["width"])
    return ar.params(preprocess=pre, quantize="uint8" if c["quantize"] else "none")


def _requests(c, seed):
    """(rows, cols, keywords, scene seed) of a burst: sides in ratio 4:2:1 of one, two and four
    times the small side."""
    rs = np.random.RandomState(c["seed"])
    out = []
    for i in range(c["requests"]):
        side = c["side"] * (1, 2, 1, 4, 1, 2, 1)[i % 7]
        kw = dict(grid_spacing=int(rs.choice([8, 16, 32])), chip_size=int(rs.choice([16, 32, 64])),
                  search_radius=int(rs.randint(8, 49)), upsampling=c["up"])
        kw["chip_size_max"] = min(4 * kw["chip_size"], 64 if side < 400 else 128)
        out.append((side, side + int(rs.randint(0, 40)), kw, seed * 16 + i))
    return out


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    ctx = L.default_context()
    s = {"kind": kind, "ctx": ctx, "up": c["up"]}
    if kind == "serve":
        s["requests"] = []
        for rows, cols, kw, sd in _requests(c, seed):
            a, b, ok, _, _ = _images(rows, cols, "uint16", sd, raw=True, holes=True, amp=4.0)
            s["requests"].append((_host(a), _host(b), _host(ok), kw))
    elif kind == "autorift":
        a, b, ok, _, _ = _images(c["rows"], c["cols"], "uint16", seed, raw=True, holes=True,
                                 amp=min(8.0, 0.4 * c["radius"]))
        s["images"] = (_host(a), _host(b), _host(ok))
        s["kw"] = dict(grid_spacing=c["spacing"], chip_size=c["chip"], upsampling=c["up"],
                       search_radius=c["radius"], chip_size_max=min(4 * c["chip"], 128))
    elif kind == "plain":
        a, b, _, _, _ = _track_images(c, seed)
        s["pair"] = ar.ImagePair(_host(a), _host(b))
        s["pair"].device(ctx)
        f = _grid_points(c, seed)
        s["points"] = ar.PointSet(**f)
        s["params"] = ar.params(preprocess="none", quantize="none", upsampling=c["up"])
    elif kind in ("search", "batch"):
        dtype = "uint16" if kind == "search" else "uint8"
        a, b, ok, fx, fy = _images(c["rows"], c["cols"], dtype, seed, raw=kind == "search",
                                   holes=True, amp=15.0 if kind == "search" else 12.0)
        s["pair"] = _pair(a, b, ok, ctx)
        if kind == "search":
            p = ar.params(grid_spacing=c["spacing"], chip_size=c["chip"], upsampling=c["up"],
                          search_radius=c["radius"], chip_size_max=min(4 * c["chip"], 128))
            grid = ar.build_grid((c["rows"], c["cols"]), p)
            s["opts"] = ar.prepare_options(p)
        else:
            p = ar.params(chip_size=16, chip_size_max=128, upsampling=c["up"])
            grid = _batch_grid(c, seed, fx, fy)
        s["shape"], s["prm"] = grid.shape, ar.multichip_params(p)
        s["pts"], s["fields"] = _device_points({k: grid.flat(k) for k in ar.points.FIELDS})
        s["out"] = _outputs(len(grid), True)
    else:
        a, b, ok, _, _ = _track_images(c, seed)
        s["pair"] = _pair(a, b, ok, ctx)
        f = _point_fields(c, seed)
        s["pts"], s["fields"] = _device_points(f)
        s["out"] = _outputs(f["x"].size, False)
        s["measure"] = _measure(c)
        if kind == "points":
            s["opts"] = ar.prepare_options(_points_params(c))
        if kind == "rotated":
            s["angles"] = np.array(_ANGLES[c["angles"]], dtype=np.float64)
    torch.cuda.synchronize()
    return s


def _batch_grid(c, seed, fx, fy):
    """Fractional centres, a radius per point in [4, 48], priors within 3 px of the motion."""
    rs = np.random.RandomState((seed + 37) & 0x7FFFFFFF)
    ys, xs = (np.arange(24, n - 24, c["spacing"], dtype=np.float64)
              for n in (c["rows"], c["cols"]))
    X, Y = (np.asfortranarray(v) for v in np.meshgrid(xs, ys))
    iy, ix = np.clip(Y.astype(int) // 4 * 4, 0, c["rows"] - 1), np.clip(
        X.astype(int) // 4 * 4, 0, c["cols"] - 1)
    mx, my = fx.cpu().numpy()[ix, iy], fy.cpu().numpy()[ix, iy]
    r = rs.randint(4, 49, X.shape)
    return ar.pointset(X + rs.uniform(-0.5, 0.5, X.shape), Y + rs.uniform(-0.5, 0.5, X.shape),
                       search_radius_x=r, search_radius_y=r, chip_size=128,
                       dx_prior=np.round(-mx) + rs.randint(-3, 4, X.shape),
                       dy_prior=np.round(-my) + rs.randint(-3, 4, X.shape))


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "serve":
        tickets = [ar.submit(a, b, secondary_valid=ok, ctx=ctx, **kw)
                   for a, b, ok, kw in s["requests"]]
        return [_result(t.wait()) for t in tickets]
    if kind == "autorift":
        a, b, ok = s["images"]
        return _result(ar.autorift(a, b, secondary_valid=ok, ctx=ctx, **s["kw"]))
    if kind == "plain":
        r = ar.track(s["pair"], s["points"], s["params"], ctx=ctx)
        return dict(dx=r.dx, dy=r.dy, correlation=r.correlation, searched=r.searched)
    lib, h, pair, pts = ctx.lib, ctx.handle, s["pair"].handle, ctypes.byref(s["pts"])
    ptr = [t.data_ptr() for t in s["out"]]
    made = None
    if "opts" in s:
        made = ctypes.c_void_p()
        ctx.check(lib.ar_prepare(h, pair, ctypes.byref(s["opts"]), ctypes.byref(made)))
        pair = made
    if kind in ("search", "batch"):
        ctx.check(lib.ar_multichip_device(h, pair, pts, *s["shape"], ctypes.byref(s["prm"]), *ptr,
                                          None))
    elif kind == "rotated":
        ang = s["angles"]
        ctx.check(lib.ar_track_device_rotated(h, pair, pts, s["up"], s["measure"],
                                              ang.ctypes.data, ang.size, *ptr, None))
    else:
        ctx.check(lib.ar_track_device(h, pair, pts, s["up"], s["measure"], *ptr, None))
    if made is not None:
        ctx.check(lib.ar_pair_destroy(made))
    return dict(zip(_SEARCH_NAMES if kind in ("search", "batch") else _NAMES, s["out"]))


def _result(r):
    return dict(dx=r.dx, dy=r.dy, correlation=r.correlation, chip_size=r.chip_size.astype(np.int32),
                interpolated=r.interpolated)


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without


def _npoints(c):
    if c["kind"] == "points":
        return c["points"]
    if c["kind"] in ("track", "plain", "rotated"):
        gr, gc = _grid_counts(c)
        return gr * gc
    if c["kind"] == "batch":
        return len(range(24, c["rows"] - 24, c["spacing"])) * len(
            range(24, c["cols"] - 24, c["spacing"]))
    m = 2 * (min(4 * c["chip"], 128) // 2 + c["radius"] + 1)
    n = [max(0, -(-(v - m) // c["spacing"])) for v in (c["rows"], c["cols"])]
    return n[0] * n[1]


def _flops(c):
    """Products of every point's surface at its chip size (the finest one of a search)."""
    if c["kind"] == "batch":  # radii uniform in [4, 48]
        area = 16 * 16 * 4 * sum(r * r for r in range(4, 49)) / 45.0
        return 2.0 * _npoints(c) * area
    n = _npoints(c) * c.get("angles", 1)
    return 2.0 * n * c["chip"] ** 2 * (2 * c["radius"]) ** 2


def work(case):
    c = dict(case)
    if c["kind"] == "serve":
        b = f = 0.0
        for rows, cols, kw, _ in _requests(c, 0):
            w = work(dict(kind="autorift", rows=rows, cols=cols, chip=kw["chip_size"],
                          radius=kw["search_radius"], spacing=kw["grid_spacing"]))
            b, f = b + w["bytes"], f + w["flops"]
        return {"bytes": b, "flops": f}
    es = {"uint8": 1, "uint16": 2, "int16": 2, "float32": 4}
    dtype = c.get("dtype", {"plain": "float32", "batch": "uint8"}.get(c["kind"], "uint16"))
    px, n = c["rows"] * c["cols"], _npoints(c)
    masks = {"points": 2, "plain": 0}.get(c["kind"], 1)
    out = 15 if c["kind"] in ("search", "batch", "autorift") else 13
    return {"bytes": float(px * (2 * es[dtype] + masks) + n * (64 + out)), "flops": _flops(c)}


# ---------------------------------------------------------------------------------------------
# The same results in 64 bits (torch float64; correlation by FFT)


def exact(case, seed):
    """Outputs of the passes over one prepared pair, and of the filters before one. The searches
    (search, batch, autorift, serve) have none: their every later level depends on which points
    the earlier ones reject, so they have no value apart from the decisions themselves."""
    c = dict(case)
    if c["kind"] not in ("track", "plain", "rotated", "points") or _flops(c) > 4e12:
        return None
    a, b, ok, _, _ = _track_images(c, seed)
    a, b = (t.T.to(torch.float64) for t in (a, b))
    valid = torch.ones(a.shape, dtype=torch.bool, device=DEV) if ok is None else ok.T.clone()
    if c["kind"] == "points":
        a, va = _filter64(a, torch.ones_like(valid), c)
        b, vb = _filter64(b, valid, c)
        valid = va & vb
    angles = _ANGLES[c["angles"]] if c["kind"] == "rotated" else (0.0,)
    out = _track64(a, b, valid, _point_fields(c, seed), c["chip"], c["radius"], c["up"],
                   c.get("measure", "zncc"), angles)
    return dict(zip(_NAMES, out[:3] + (None,)))


def _box(t, w):
    """Sums over the w x w window clamped to the image."""
    for d in (0, 1):
        n = t.shape[d]
        w_ = min(w, n)
        lo, hi = w_ // 2, w_ - 1 - w_ // 2
        s = torch.cumsum(t, d)
        s = torch.cat([torch.zeros_like(s.narrow(d, 0, 1)), s], d)
        i = torch.arange(n, device=DEV)
        t = s.index_select(d, (i + hi + 1).clamp(max=n)) - s.index_select(d, (i - lo).clamp(min=0))
    return t


def _filter64(img, ok, c):
    w = c["width"]
    okd = ok.double()
    cnt = _box(okd, w)
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    mean = _box(torch.where(ok, img, zero), w) / cnt
    out = img - mean
    fine = ok & (cnt > 0)
    if c["filter"] == "wallis":
        sd = torch.sqrt(_box(torch.where(fine, out * out, zero), w) / _box(fine.double(), w))
        out = out / sd
        fine = fine & (sd > 0)
    eroded = _box((~ok).double(), w) < 0.5 if not bool(ok.all()) else ok
    vout = eroded & fine
    out = torch.where(fine, out, zero)
    if c["quantize"]:
        v = out[vout]
        m, sd = v.mean(), v.std()
        q = torch.round(((out - (m - 3 * sd)) * (255.0 / (6 * sd))).clamp(0, 255))
        out = torch.where(vout, q, zero)
    return out, vout


def _pyramid(up):
    """The cascade of pyrUp steps on 5 samples as one (5 up) x 5 matrix."""
    n, m = 5, np.eye(5)
    while n < 5 * up:
        ref = lambda p: -p if p < 0 else (2 * (2 * n - 1) - p if p > 2 * n - 1 else p)
        u = np.zeros((2 * n, n))
        for p in range(2 * n):
            if p % 2 == 0:
                u[p, p // 2] += 0.75
                u[p, ref(p - 2) // 2] += 0.125
                u[p, ref(p + 2) // 2] += 0.125
            else:
                u[p, ref(p - 1) // 2] += 0.5
                u[p, ref(p + 1) // 2] += 0.5
        m, n = u @ m, 2 * n
    return torch.from_numpy(m).to(DEV)


def _turned(chip, deg):
    """Each chip turned about its centre: bilinear, zero where a neighbour is outside it."""
    if deg == 0.0:
        return chip
    n = chip.shape[-1]
    s, co = math.sin(math.radians(deg)), math.cos(math.radians(deg))
    i = torch.arange(1, n + 1, device=DEV, dtype=torch.float64)
    d = i - (n + 1) / 2
    y = (n + 1) / 2 + co * d[:, None] + s * d[None, :]
    x = (n + 1) / 2 - s * d[:, None] + co * d[None, :]
    i0, j0 = torch.floor(y), torch.floor(x)
    ok = (i0 >= 1) & (j0 >= 1) & (i0 + 1 <= n) & (j0 + 1 <= n)
    fy, fx = y - i0, x - j0
    i0, j0 = (t.clamp(1, n - 1).long() - 1 for t in (i0, j0))
    v = (1 - fy) * ((1 - fx) * chip[:, i0, j0] + fx * chip[:, i0, j0 + 1]) + fy * (
        (1 - fx) * chip[:, i0 + 1, j0] + fx * chip[:, i0 + 1, j0 + 1])
    return torch.where(ok, v, torch.zeros((), dtype=torch.float64, device=DEV))


def _track64(ref, sec, valid, f, chip, radius, up, measure, angles):
    """dx, dy, correlation and searched of every point; every window lies inside the images."""
    n, h, nr = f["x"].size, chip // 2, 2 * radius
    wn = chip + nr - 1
    P = _pyramid(up)
    ii = torch.cumsum(torch.cumsum(valid.double(), 0), 1)
    ii = torch.nn.functional.pad(ii, (1, 0, 1, 0))
    col = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(DEV)
    x, y, dx0, dy0 = (col(f[k]) for k in ("x", "y", "dx_prior", "dy_prior"))
    wr, wc = (torch.floor(v + 0.5).long() - h - radius - 1 for v in (y, x))
    cr, cc = (torch.floor(v + 0.5 - p).long() - h - 1 for v, p in ((y, dy0), (x, dx0)))
    out = [torch.full((n,), math.nan, dtype=torch.float64, device=DEV) for _ in range(3)]
    searched = torch.zeros(n, dtype=torch.bool, device=DEV)
    step = max(1, int(6e8 / (wn * wn * 64 + 25 * up * up * 8)))
    ar_, br_ = torch.arange(wn, device=DEV), torch.arange(chip, device=DEV)
    for k in range(0, n, step):
        q = slice(k, min(k + step, n))
        win = ref[(wr[q, None] + ar_)[:, :, None], (wc[q, None] + ar_)[:, None, :]]
        ch0 = sec[(cr[q, None] + br_)[:, :, None], (cc[q, None] + br_)[:, None, :]]
        r0, c0 = cr[q], cc[q]
        any_ = (ii[r0 + chip, c0 + chip] - ii[r0, c0 + chip] - ii[r0 + chip, c0] + ii[r0, c0]) > 0.5
        box = lambda t: (lambda s: s[:, chip:, chip:] - s[:, :-chip, chip:] - s[:, chip:, :-chip]
                         + s[:, :-chip, :-chip])(torch.nn.functional.pad(
                             torch.cumsum(torch.cumsum(t, 1), 2), (1, 0, 1, 0)))
        if measure == "ncc":
            den = torch.sqrt(box(win * win).clamp(min=0))
        else:  # sums about the window's mean: the variance without cancellation
            wz = win - win.mean((1, 2), keepdim=True)
            den = torch.sqrt((box(wz * wz) - box(wz) ** 2 / chip ** 2).clamp(min=0))
        fw = torch.fft.rfft2(win - win.mean((1, 2), keepdim=True))
        best = peak = None
        for deg in angles:
            ch = _turned(ch0, deg)
            cz = ch - ch.mean((1, 2), keepdim=True)
            nrm = torch.sqrt((cz * cz).sum((1, 2), keepdim=True))
            fc = torch.fft.rfft2(cz, s=(wn, wn))
            num = torch.fft.irfft2(fw * fc.conj(), s=(wn, wn))[:, :nr, :nr]
            surf = torch.where((den > 0) & (nrm > 0), num / (den * nrm), torch.zeros_like(num))
            top = surf.flatten(1).max(1).values
            top = torch.where(nrm[:, 0, 0] ** 2 > 2.3e-16 * chip * chip, top, -math.inf)
            if best is None:
                best, peak = surf, top
            else:
                better = top > peak
                best = torch.where(better[:, None, None], surf, best)
                peak = torch.maximum(peak, top)
        at = best.flatten(1).argmax(1)
        pi, pj = at // nr, at % nr
        i0, j0 = (pi - 2).clamp(0, nr - 5), (pj - 2).clamp(0, nr - 5)
        b5 = torch.arange(5, device=DEV)
        m = torch.arange(best.shape[0], device=DEV)
        patch = best[m[:, None, None], (i0[:, None] + b5)[:, :, None], (j0[:, None] + b5)[:, None, :]]
        fine = (P @ patch @ P.T).flatten(1)
        v, e = fine.max(1)
        si, sj = e // (5 * up), e % (5 * up)
        good = any_ & torch.isfinite(peak)
        for o, t in zip(out, (sj / up + j0 - radius + dx0[q], si / up + i0 - radius + dy0[q], v)):
            o[q] = torch.where(good, t, math.nan)
        searched[q] = any_
    return out[0], out[1], out[2], searched
