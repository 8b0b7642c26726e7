"""The frames whose rendering time this repository is judged by.

A case is one frame as a renderer hands it to the hider: shaded grids (camera
or raster space), sample patterns and frame options in, the float channels and
the 8-bit r g b a image out.  Every pass goes through the public entry points
(``aqsis_gb300.aqh`` and the C functions of ``include/aqh.h`` it loads).

Three ways of feeding grids occur in use and in the cases:

* ``device``: the grids live in GPU memory and the frame stays open, as for a
  shading stage on the same GPU; a pass renders and reads the images back;
* ``host`` and ``host3``: packed host arrays of four-float or three-float
  entries (the latter is the reference's CqVector3D / CqColor layout); a pass
  opens the frame, hands over samples and grids, renders and reads back.

``exact`` renders the same frame in 64 bits with plain torch: hit tests, the
two Newton steps of the inverse bilinear, depth and opacity compositing,
pixel filter and exposure.
"""
import ctypes
import math

import numpy as np
import torch

from aqsis_gb300 import aqh
from aqsis_gb300 import scene as S

FLT_MAX = float(np.finfo(np.float32).max)
RGBA = np.array([0, 1, 2, 6], np.int32)
# `exact` leaves out frames with more hit tests than this (over ten seconds)
EXACT_TESTS = 9e9

BASE = dict(kind="opaque", width=640, height=480, xs=4, ys=4, grids=1000, side=16, filter="gaussian", fw=2.0,
            motion=0.0, dof=False, transparent=0.0, window=1.0, feed="device", batched=True, naov=0, spacing=1.0)


def _case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    return [
        # the smallest request a render server sees: latency of one whole call
        _case("opaque_320x240_host", width=320, height=240, xs=2, ys=2, grids=195, feed="host", batched=False),
        # a RIB scene of spheres diced at shading rate 1, camera-space grids of many sizes, constant shading
        _case("spheres_640x480_host", kind="spheres", grids=64, feed="host", batched=False),
        # an ordinary opaque frame from page-locked host arrays in the reference's own layout
        _case("opaque_1280x720_host3", width=1280, height=720, grids=31250, feed="host3"),
        # the largest opaque frame: 51.2M micropolygons, 25 layers deep, resident on the GPU
        _case("opaque_1920x1080", width=1920, height=1080, grids=200000),
        # layered transparency (smoke, foliage, glass) over half the image, 64 samples, a sharpening filter
        _case("transparent_1920x1080", kind="transparent", width=1920, height=1080, xs=8, ys=8, grids=16200,
              filter="catmull-rom", fw=3.0, transparent=1.0, window=0.5),
        # what most frames hold: opaque surfaces with some transparent ones among them
        _case("mixed_1280x720", kind="mixed", width=1280, height=720, grids=12000, transparent=0.25),
        # motion blur alone at preview size
        _case("motion_640x480", kind="motion", grids=3000, motion=20.0, batched=False),
        # depth of field alone, nothing moves
        _case("dof_1280x720", kind="motion", width=1280, height=720, grids=12000, dof=True),
        # the largest frame: motion blur and depth of field at 36 samples
        _case("motion_dof_1920x1080", kind="motion", width=1920, height=1080, xs=6, ys=6, grids=100000, motion=20.0,
              dof=True, filter="box", fw=1.0),
        # motion blur, depth of field and transparency together
        _case("motion_transparent_640x480", kind="motion", grids=1200, motion=12.0, dof=True, transparent=0.5),
        # odd everything: resolution, crop window, 5x3 samples, grids of many shapes, culled micropolygons,
        # output variables, a wide filter, exposure
        _case("ragged_1001x563_aov", kind="ragged", width=1001, height=563, xs=5, ys=3, grids=6000, filter="mitchell",
              fw=4.0, naov=3, feed="host", batched=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["opaque", "opaque", "spheres", "transparent", "mixed", "motion", "motion", "ragged"])
    w = int(_log(rng, 160, 2600))
    h = max(96, int(w * rng.uniform(0.45, 0.9)))
    n = rng.randint(2, 8)
    xs, ys = rng.choice([(n, n), (n, n), (n, max(1, n - 1))])
    side = rng.choice([16, 16, 16, 9, 7, 4])
    feed = rng.choice(["device", "device", "host", "host3"])
    c = dict(BASE, kind=kind, width=w, height=h, xs=xs, ys=ys, side=side, feed=feed, batched=rng.random() < 0.6,
             filter=rng.choice(["gaussian", "catmull-rom", "box", "triangle", "mitchell"]),
             fw=rng.choice([1.0, 2.0, 2.0, 3.0, 4.0]))
    if kind == "spheres":
        # the spheres' screen size follows the frame's
        w = c["width"] = min(w, 1400)
        c["height"] = min(h, 1000)
        c.update(grids=rng.randint(16, 96), feed=rng.choice(["host", "host3"]), side=16)
        return c
    # micropolygons by depth complexity: layers of one-pixel micropolygons over the window the grids lie in
    layers = {"opaque": _log(rng, 1.5, 26), "transparent": rng.uniform(1.5, 8.5), "mixed": _log(rng, 2, 6),
              "motion": _log(rng, 1.0, 8.0), "ragged": _log(rng, 1.5, 8)}[kind]
    c["spacing"] = rng.choice([1.0, 1.0, 0.7, 1.6])
    if kind == "transparent":
        c.update(transparent=1.0, window=rng.choice([0.5, 0.7, 1.0]))
        c["xs"], c["ys"] = min(xs, 6 if w > 1300 else 8), min(ys, 6 if w > 1300 else 8)
    elif kind == "mixed":
        c.update(transparent=rng.uniform(0.05, 0.5))
    elif kind == "motion":
        what = rng.choice(["motion", "dof", "both"])
        c["width"], c["height"] = w, h = min(w, 1300), min(h, 800)
        c["xs"], c["ys"] = min(xs, 6), min(ys, 6)
        c.update(motion=0.0 if what == "dof" else rng.uniform(4, 20), dof=what != "motion")
        if rng.random() < 0.25:
            layers = min(layers, 2.0)
            c.update(transparent=rng.uniform(0.2, 0.6))
    elif kind == "ragged":
        c.update(naov=rng.choice([0, 0, 1, 3, 5]), feed=rng.choice(["host", "host3"]))
        c["width"], c["height"] = w, h = min(w, 1600), min(h, 1000)
    area = w * h * c["window"] ** 2
    per_grid = (120.0 if kind == "ragged" else side * side) * c["spacing"] ** 2
    c["grids"] = max(8, int(layers * area / per_grid))
    return c


# ---------------------------------------------------------------------------
# inputs

def _camera(width, height, fov=40.0, near=0.1, far=1e4):
    """Perspective camera-to-raster matrix, row vectors, element [row * 4 + col]."""
    f = 1.0 / math.tan(math.radians(fov) / 2)
    a = width / height
    m = np.zeros((4, 4))
    m[0, 0] = f * width / (2 * a)
    m[2, 0] = 0.5 * width
    m[1, 1] = -f * height / 2
    m[2, 1] = 0.5 * height
    m[2, 2] = far / (far - near)
    m[3, 2] = -near * far / (far - near)
    m[2, 3] = 1.0
    return m.astype(np.float32)


def _frame(c):
    fr = dict(width=c["width"], height=c["height"], xsamples=c["xs"], ysamples=c["ys"], filter=c["filter"],
              xfilter=c["fw"], yfilter=c["fw"], q_dither=0.0)
    if c["motion"] > 0:
        fr["shutter"] = (0.0, 1.0)
    if c["dof"]:
        fr.update(fstop=2.8, focal_length=0.05, focal_distance=50.0, dof_scale=(c["height"] / 2, c["height"] / 2))
    if c["kind"] == "ragged":
        w, h = c["width"], c["height"]
        fr.update(crop=(w // 40, w - w // 25, h // 50, h - h // 30), gain=1.2, gamma=2.2, q_dither=0.5)
    if c["kind"] == "spheres":
        fr["camera_to_raster"] = tuple(float(v) for v in _camera(c["width"], c["height"]).reshape(16))
    return S.Frame(**fr)


def _patterns(c, fr, rng):
    """250 stratified, jittered patterns picked per pixel, as the reference's sampler does."""
    xs, ys, spp, n = c["xs"], c["ys"], c["xs"] * c["ys"], 250
    _, _, w, h = fr.sample_region
    ix, iy = np.tile(np.arange(xs), ys), np.repeat(np.arange(ys), xs)

    def cells():
        p = np.stack([(ix + rng.random((n, spp))) / xs, (iy + rng.random((n, spp))) / ys], -1).astype(np.float32)
        return np.minimum(p, np.nextafter(np.float32(1), np.float32(0)))

    def pick():
        return rng.integers(0, n, w * h, dtype=np.uint32)

    kw = {}
    if c["motion"] > 0:
        kw["time"] = ((np.arange(spp) + rng.random((n, 1))) / spp).astype(np.float32)
        kw["time_index"] = pick()
    if c["dof"]:
        kw.update(dof=cells(), dof_index=pick(), shuffle_index=pick(),
                  shuffle=np.argsort(rng.random((n, spp)), axis=1).astype(np.int32))
    if c["kind"] == "ragged":
        x0, x1, y0, y1 = fr.crop_window
        kw["dither"] = rng.random((x1 - x0) * (y1 - y0), dtype=np.float32)
    return S.Samples(npatterns=n, pos=cells(), pos_index=pick(), **kw)


def _table(cu, cv, nkeys, flags):
    """Grid table of the packed layouts: grids one after another."""
    cu, cv = np.asarray(cu, np.int64), np.asarray(cv, np.int64)
    nv = (cu + 1) * (cv + 1)
    G = len(cu)
    pb, cb = np.zeros(G, np.int64), np.zeros(G, np.int64)
    pb[1:], cb[1:] = np.cumsum(nv * nkeys)[:-1], np.cumsum(nv)[:-1]
    return dict(cu=cu.astype(np.int32), cv=cv.astype(np.int32), nkeys=np.full(G, nkeys, np.int32),
                flags=np.asarray(flags, np.int32), pbase=pb, cbase=cb,
                tbase=(np.arange(G) * nkeys if nkeys > 1 else np.zeros(G)).astype(np.int32),
                times=np.tile(np.array([0, 1], np.float32), G) if nkeys > 1 else np.zeros(1, np.float32))


def _raster_grids(c, seed):
    """Jittered raster-space grids: origins uniform over the window, one plane
    z = z0 + s (x - x0) each, random vertex colours; a second motion key moves
    a grid by one vector."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)

    def u(*shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo

    G, W, H, win = c["grids"], c["width"], c["height"], c["window"]
    if c["kind"] == "ragged":
        shapes = [(16, 16), (1, 1), (31, 9), (7, 13), (3, 2), (12, 5), (9, 16)]
        which = rng.integers(0, len(shapes), G)
        cu, cv = np.array([s[0] for s in shapes])[which], np.array([s[1] for s in shapes])[which]
    else:
        cu = cv = np.full(G, c["side"])
    nkeys = 2 if c["motion"] > 0 else 1
    transp = rng.random(G) < c["transparent"]
    flags = np.where(transp, S.GRID_SMOOTH, S.GRID_SMOOTH | S.GRID_OPAQUE)
    if c["kind"] == "ragged":
        flags = np.where(rng.random(G) < 0.4, S.GRID_OPAQUE, flags)
    t = _table(cu, cv, nkeys, flags)
    nv = torch.from_numpy((np.asarray(cu, np.int64) + 1) * (np.asarray(cv, np.int64) + 1)).cuda()
    gid = torch.repeat_interleave(torch.arange(G, device="cuda"), nv)          # grid of every vertex
    local = torch.arange(gid.numel(), device="cuda") - torch.from_numpy(t["cbase"]).cuda()[gid]
    stride = torch.from_numpy(np.asarray(cu, np.int64) + 1).cuda()[gid]
    jj, ii = local // stride, local % stride
    ox = u(G, lo=W * (1 - win) / 2, hi=W * (1 + win) / 2)
    oy = u(G, lo=H * (1 - win) / 2, hi=H * (1 + win) / 2)
    z0, sl = u(G, lo=1.0, hi=1000.0), u(G, lo=-0.01, hi=0.01)
    n, d = gid.numel(), c["spacing"]
    P = torch.zeros((n, 4), device="cuda")
    P[:, 0] = ox[gid] + d * (ii + u(n, lo=-0.3, hi=0.3))
    P[:, 1] = oy[gid] + d * (jj + u(n, lo=-0.3, hi=0.3))
    P[:, 2] = z0[gid] + sl[gid] * (P[:, 0] - ox[gid])
    if nkeys == 2:
        mag, ang = u(G, hi=c["motion"]), u(G, hi=2 * math.pi)
        Q = P.clone()
        Q[:, 0] += (mag * torch.cos(ang))[gid]
        Q[:, 1] += (mag * torch.sin(ang))[gid]
        # key 0 then key 1 of each grid
        at = torch.from_numpy(t["pbase"]).cuda()[gid] + local
        both = torch.empty((2 * n, 4), device="cuda")
        both[at] = P
        both[at + nv[gid]] = Q
        P = both
    Ci = torch.zeros((n, 4), device="cuda")
    Ci[:, :3] = u(n, 3)
    Oi = torch.ones((n, 4), device="cuda")
    Oi[:, 3] = 0
    tv = torch.from_numpy(transp).cuda()[gid]
    Oi[:, :3] = torch.where(tv[:, None], u(n, 3, lo=0.1, hi=0.9), Oi[:, :3])
    t.update(P=P, Ci=Ci, Oi=Oi)
    if c["kind"] == "ragged":
        t["culled"] = (rng.random(int((t["cu"].astype(np.int64) * t["cv"]).sum())) < 0.02).astype(np.uint8)
    if c["naov"]:
        t["aov"] = u(n, c["naov"], lo=-1.0)
    return t


def _sphere_grids(c, seed):
    """Spheres in the view frustum as camera-space grids of at most 16x16
    one-pixel micropolygons, matte shading, one constant colour each."""
    rng = np.random.default_rng(seed)
    W, H = c["width"], c["height"]
    m = _camera(W, H).astype(np.float64)
    f, aspect = 1.0 / math.tan(math.radians(20.0)), W / H
    cus, cvs, Ps, Cs = [], [], [], []
    for _ in range(c["grids"]):
        r, z = rng.uniform(0.2, 1.0), rng.uniform(5.0, 30.0)
        o = np.array([rng.uniform(-aspect, aspect) * z / f, rng.uniform(-1, 1) * z / f, z])
        tint = rng.uniform(0, 1, 3)
        px = r * f * H / 2 / (z - r)                      # raster radius
        nu, nv = max(1, math.ceil(2 * math.pi * px / 16)), max(1, math.ceil(math.pi * px / 16))
        cu, cv = max(1, math.ceil(2 * math.pi * px / nu)), max(1, math.ceil(math.pi * px / nv))
        th = np.linspace(0, 2 * math.pi, nu * cu + 1)
        ph = np.linspace(-math.pi / 2, math.pi / 2, nv * cv + 1)
        N = np.stack([np.cos(th)[None] * np.cos(ph)[:, None], np.sin(th)[None] * np.cos(ph)[:, None],
                      np.broadcast_to(np.sin(ph)[:, None], (len(ph), len(th)))], -1)
        P = o + r * N
        lit = np.abs((N * P).sum(-1)) / np.linalg.norm(P, axis=-1)
        C = tint * (0.5 * np.abs(N[..., 2:])) + 0.5 * lit[..., None] ** 10
        for b in range(nv):
            for a in range(nu):
                p = P[b * cv:(b + 1) * cv + 1, a * cu:(a + 1) * cu + 1].reshape(-1, 3)
                q = p @ m[:3, :3] + m[3, :3]
                q = q[:, :2] / (p @ m[:3, 3] + m[3, 3])[:, None]
                if q[:, 0].max() < -1 or q[:, 0].min() > W + 1 or q[:, 1].max() < -1 or q[:, 1].min() > H + 1:
                    continue
                cus.append(cu)
                cvs.append(cv)
                Ps.append(p)
                Cs.append(C[b * cv:(b + 1) * cv + 1, a * cu:(a + 1) * cu + 1].reshape(-1, 3))
    t = _table(cus, cvs, 1, np.full(len(cus), S.GRID_OPAQUE | S.GRID_CAMERA))
    n = sum(len(p) for p in Ps)
    P, Ci, Oi = (np.zeros((n, 4), np.float32) for _ in range(3))
    P[:, :3], Ci[:, :3], Oi[:, :3] = np.concatenate(Ps), np.concatenate(Cs), 1.0
    t.update(P=torch.from_numpy(P).cuda(), Ci=torch.from_numpy(Ci).cuda(), Oi=torch.from_numpy(Oi).cuda())
    return t


def _inputs(c, seed):
    c = dict(BASE, **c)
    fr = _frame(c)
    t = (_sphere_grids if c["kind"] == "spheres" else _raster_grids)(c, seed)
    return c, fr, t, _patterns(c, fr, np.random.default_rng(seed + 1))


def _pinned(a, keep):
    p = torch.empty(a.shape, dtype=a.dtype, pin_memory=True)
    p.copy_(a)
    keep.append(p)
    return p.numpy()


def prepare(case, seed):
    c, fr, t, smp = _inputs(case, seed)
    keep = []
    mps = int((t["cu"].astype(np.int64) * t["cv"]).sum())
    h = aqh.Hider(0)
    h.set_mode(c["batched"])
    x0, x1, y0, y1 = fr.crop_window
    st = dict(case=c, frame=fr, samples=smp, hider=h, keep=keep,
              channels=_pinned(torch.zeros((y1 - y0, x1 - x0, 9)), keep),
              rgba=_pinned(torch.zeros((y1 - y0, x1 - x0, 4), dtype=torch.uint8), keep),
              aov=_pinned(torch.zeros((y1 - y0, x1 - x0, c["naov"])), keep) if c["naov"] else None)
    if c["feed"] == "device":
        d = {k: (v if torch.is_tensor(v) else torch.from_numpy(v).cuda()) for k, v in t.items()}
        keep.append(d)
        torch.cuda.synchronize()
        h.frame_begin(fr)
        h.set_samples(smp)
        h.submit_grids_device(len(t["cu"]), *[d[k].data_ptr() for k in (
            "cu", "cv", "nkeys", "flags", "pbase", "cbase", "tbase", "times", "P", "Ci", "Oi")], mps)
    else:
        k = 3 if c["feed"] == "host3" else 4
        host = {n: _pinned(t[n][:, :k], keep) if n in ("P", "Ci", "Oi") else t[n] for n in (
            "cu", "cv", "nkeys", "flags", "pbase", "cbase", "tbase", "times", "P", "Ci", "Oi")}
        st["grids"] = S.Grids(culled=t.get("culled"), aov=t["aov"].cpu().numpy() if "aov" in t else None, **host)
    return st


def run(st):
    h, c = st["hider"], st["case"]
    if c["feed"] != "device":
        h.frame_begin(st["frame"])
        h.set_samples(st["samples"])
        h.submit_grids_host(st["grids"], packed3=c["feed"] == "host3")
    h.render(sync=False)
    ch, q = st["channels"], st["rgba"]
    h.synchronize()
    h._check(h.L.aqh_read_channels(h.ctx, ch.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), ch.size), "read")
    h._check(h.L.aqh_read_quantized_u8(h.ctx, RGBA.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), 4,
                                       q.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)), q.size), "read")
    out = {"rgba": q, "colour": ch[..., :7], "depth": ch[..., 7], "coverage": ch[..., 8]}
    if st["aov"] is not None:
        a = st["aov"]
        h._check(h.L.aqh_read_aov(h.ctx, a.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), a.size), "read")
        out["aov"] = a
    return out


def _mean_mps(c):
    if c["kind"] == "spheres":
        # one-pixel micropolygons over both sides of spheres of raster radius f r / (z - r): the mean of its square
        # over the radii and distances drawn, plus the rounding up of patch sizes
        f = c["height"] / 2 / math.tan(math.radians(20.0))
        return c["grids"] * 4 * math.pi * f * f * 0.0068
    return c["grids"] * (120.0 if c["kind"] == "ragged" else c["side"] ** 2)


def work(case):
    c = dict(BASE, **case)
    mps, spp = _mean_mps(c), c["xs"] * c["ys"]
    side = 9.0 if c["kind"] == "ragged" else c["side"]
    verts = mps * ((side + 1) / side) ** 2
    pix = c["width"] * c["height"]
    # points of every key, colours and opacities once; pattern choices; channels, bytes and output variables
    per_vertex = (32 if c["motion"] > 0 else 16) + 32
    nbytes = verts * per_vertex + pix * (4 + 40 + 4 * c["naov"])
    # a bound per micropolygon; a hit test, depth and colour per sample hit (every layer where all layers
    # show, one where the front one hides the rest); the filter's weighted sum per sample and window pixel
    layers = mps * c["spacing"] ** 2 / (pix * c["window"] ** 2)
    hits = pix * c["window"] ** 2 * spp * (layers if c["transparent"] >= 1 else min(layers, 1.0))
    taps = (2 * int(c["fw"] / 2) + 1) ** 2 if c["fw"] >= 2 else 1
    return {"bytes": float(nbytes), "flops": float(mps * 40 + hits * 150 + pix * spp * taps * 15)}


# ---------------------------------------------------------------------------
# the same frame in 64 bits

def _filter_weight(name, x, y, w):
    if name == "gaussian":
        return np.exp(-8.0 * ((x / w) ** 2 + (y / w) ** 2))
    if name == "box":
        return np.minimum(np.abs(x) <= w / 2, np.abs(y) <= w / 2).astype(np.float64)
    if name == "triangle":
        h = w / 2
        return np.minimum(np.maximum(0, (h - np.abs(x)) / h), np.maximum(0, (h - np.abs(y)) / h))
    if name == "catmull-rom":
        r = np.sqrt(x * x + y * y)
        return np.where(r >= 2, 0.0, np.where(r < 1, 3 * r ** 3 - 5 * r ** 2 + 2, -r ** 3 + 5 * r ** 2 - 8 * r + 4))

    def mitchell(t):
        t = np.abs(2 * t)
        b = c = 1 / 3.0
        return np.where(t > 1, (-b - 6 * c) * t ** 3 + (6 * b + 30 * c) * t ** 2 + (-12 * b - 48 * c) * t + 8 * b + 24 * c,
                        (12 - 9 * b - 6 * c) * t ** 3 + (-18 + 12 * b + 6 * c) * t ** 2 + 6 - 2 * b) / 6
    return mitchell(x / w) * mitchell(y / w)


class _Exact:
    """Vertices, samples and hit tests of one frame in 64 bits."""

    def __init__(self, c, fr, t, smp):
        self.c, self.fr = c, fr
        dev = "cuda"
        self.spp = c["xs"] * c["ys"]
        self.x0, self.y0, self.w, self.h = fr.sample_region
        i64 = lambda a: torch.from_numpy(np.asarray(a).astype(np.int64)).to(dev)  # noqa: E731
        f64 = lambda a: torch.from_numpy(np.asarray(a)).to(dev).double()  # noqa: E731
        self.cu, cv = i64(t["cu"]), i64(t["cv"])
        self.nv = (self.cu + 1) * (cv + 1)
        self.mpb = torch.cumsum(self.cu * cv, 0) - self.cu * cv
        self.n = int((self.cu * cv).sum())
        self.pb, self.cb, self.flags = i64(t["pbase"]), i64(t["cbase"]), i64(t["flags"])
        self.moving = c["motion"] > 0
        P = t["P"].double()
        if c["kind"] == "spheres":
            m = torch.from_numpy(_camera(c["width"], c["height"])).to(dev).double()
            q = P[:, :3] @ m[:3] + m[3]
            P = torch.cat([q[:, :2] / q[:, 3:], P[:, 2:3]], 1)
        self.P, self.Ci, self.Oi = P[:, :3].contiguous(), t["Ci"].double(), t["Oi"].double()
        self.culled = torch.from_numpy(t["culled"]).to(dev).bool() if "culled" in t else None
        self.pos, self.pi = f64(smp.pos).view(-1, self.spp, 2), i64(smp.pos_index)
        if self.moving:
            self.time, self.ti = f64(smp.time).view(-1, self.spp), i64(smp.time_index)
        if c["dof"]:
            d = f64(smp.dof).view(-1, self.spp, 2) * 2 - 1
            r = d.norm(dim=-1)
            self.lens = torch.where(r[..., None] == 0, torch.zeros_like(d),
                                    d * (d.abs().amax(-1) / r.clamp_min(1e-300))[..., None])
            self.di, self.si = i64(smp.dof_index), i64(smp.shuffle_index)
            self.strat = torch.argsort(i64(smp.shuffle).view(-1, self.spp), dim=1)  # stratum of each sample
            lens = np.float32(np.float32(0.05) / np.float32(2.8))
            self.mult = float(np.float32(0.5 * float(lens) * 50.0 / float(np.float32(50.0) + lens)))
            self.inv, self.dscale = float(np.float32(1 / 50.0)), c["height"] / 2

    def corners(self, m):
        """Grid, first vertex and row stride of micropolygons m."""
        g = torch.searchsorted(self.mpb, m, right=True) - 1
        k = m - self.mpb[g]
        cu = self.cu[g]
        return g, (k // cu) * (cu + 1) + k % cu, cu + 1

    def coc(self, z):
        return self.dscale * self.mult * (1 / z - self.inv).abs()

    def verts(self, g, i, s, key):
        b = self.pb[g] + key * self.nv[g] + i
        return [self.P[b], self.P[b + 1], self.P[b + s], self.P[b + s + 1]]

    def at(self, m, smp):
        """Corner points of micropolygons m as samples smp see them, key-0 corners, and the samples' positions."""
        pix, j = smp // self.spp, smp % self.spp
        x = (self.x0 + pix % self.w).double() + self.pos[self.pi[pix], j, 0]
        y = (self.y0 + pix // self.w).double() + self.pos[self.pi[pix], j, 1]
        g, i, s = self.corners(m)
        k0 = self.verts(g, i, s, 0)
        v = k0
        if self.moving:
            f = self.time[self.ti[pix], j][:, None]
            v = [(1 - f) * a + f * b for a, b in zip(k0, self.verts(g, i, s, 1))]
        if self.c["dof"]:
            d = self.lens[self.di[pix], self.strat[self.si[pix], j]]
            v = [torch.cat([a[:, :2] - self.coc(a[:, 2])[:, None] * d, a[:, 2:]], 1) for a in v]
        return v, k0, x, y

    def uv(self, v, x, y):
        """One Newton step of the inverse bilinear from the centre, a second unless nearly rectangular."""
        A, E, F = v[0][:, :2], v[1][:, :2] - v[0][:, :2], v[2][:, :2] - v[0][:, :2]
        G = v[3][:, :2] - v[2][:, :2] - E
        lin = G.abs().amax(1) < 1e-2 * torch.maximum(E.abs().amax(1), F.abs().amax(1))
        q = torch.stack([x, y], 1)
        u = w = torch.full_like(x, 0.5)
        for it in range(2):
            M1, M2 = E + G * w[:, None], F + G * u[:, None]
            b = A + E * u[:, None] + F * w[:, None] + G * (u * w)[:, None] - q
            det = M1[:, 0] * M2[:, 1] - M1[:, 1] * M2[:, 0]
            det = torch.where(det != 0, 1 / det, det)
            du = det * (b[:, 0] * M2[:, 1] - b[:, 1] * M2[:, 0])
            dw = -det * (b[:, 0] * M1[:, 1] - b[:, 1] * M1[:, 0])
            keep = lin if it else torch.zeros_like(lin)
            u, w = torch.where(keep, u, u - du), torch.where(keep, w, w - dw)
        return u, w

    def inside(self, v, k0, x, y):
        """Point in polygon: the corner order and degenerate edges follow key 0, the edges the moved corners."""
        near = lambda a, b: ((a - b) ** 2).sum(1) < 1e-8  # noqa: E731
        A, B, C, D = k0[0], k0[1], k0[3], k0[2]
        ab, bc, cd, da = near(A, B), near(B, C), near(C, D), near(D, A)
        shift, drop = ab | bc, ~(ab | bc) & cd
        deg = shift | drop | da
        pick = lambda P, Q, R, T: (P, torch.where(shift[:, None], R, Q),  # noqa: E731
                                   torch.where((shift | drop)[:, None], T, R), T)
        oA, oB, oC, _ = pick(A, B, C, D)
        flip = ((oA[:, 0] - oB[:, 0]) * (oB[:, 1] - oC[:, 1])) >= ((oA[:, 1] - oB[:, 1]) * (oB[:, 0] - oC[:, 0]))
        a, b, c, d = pick(v[0], v[1], v[3], v[2])
        fl, dg = flip[:, None], deg[:, None]
        first = torch.where(fl, b, torch.where(dg, c, d))
        second = torch.where(dg & ~fl, b, c)
        third = torch.where(fl, d, b)
        edges = [(a, first, True), (first, second, True), (torch.where(dg, second, second), torch.where(dg, a, third), False),
                 (torch.where(dg, second, third), a, False)]
        ok = torch.ones_like(x, dtype=torch.bool)
        for p, q, strict in edges:
            s = (y - p[:, 1]) * (q[:, 0] - p[:, 0]) - (x - p[:, 0]) * (q[:, 1] - p[:, 1])
            ok &= (s > 0) if strict else (s >= 0)
        return ok

    def boxes(self, m):
        """Pixel boxes that hold every position of micropolygons m over shutter and lens, clipped to the region."""
        g, i, s = self.corners(m)
        v = self.verts(g, i, s, 0) + (self.verts(g, i, s, 1) if self.moving else [])
        st = torch.stack(v)
        lo, hi = st.amin(0), st.amax(0)
        if self.c["dof"]:
            r = torch.maximum(self.coc(lo[:, 2]), self.coc(hi[:, 2]))[:, None]
            lo, hi = lo[:, :2] - r, hi[:, :2] + r
        x0 = lo[:, 0].floor().clamp(self.x0, self.x0 + self.w).long()
        x1 = hi[:, 0].ceil().clamp(self.x0, self.x0 + self.w).long()
        y0 = lo[:, 1].floor().clamp(self.y0, self.y0 + self.h).long()
        y1 = hi[:, 1].ceil().clamp(self.y0, self.y0 + self.h).long()
        nx, ny = (x1 - x0).clamp_min(0), (y1 - y0).clamp_min(0)
        if self.culled is not None:
            nx = torch.where(self.culled[m], torch.zeros_like(nx), nx)
        return x0 - self.x0, y0 - self.y0, nx, nx * ny

    def hits(self, keep):
        """(sample, depth, micropolygon) of every hit on the grids for which keep(grid) holds, in chunks."""
        step = 1 << 21
        for b in range(0, self.n, step):
            m = torch.arange(b, min(self.n, b + step), device="cuda")
            m = m[keep(self.corners(m)[0])]
            if not m.numel():
                continue
            x0, y0, nx, cnt = self.boxes(m)
            cum = torch.cumsum(cnt, 0)
            k0 = 0
            while k0 < m.numel():
                base = int(cum[k0 - 1]) if k0 else 0
                k1 = max(k0 + 1, int(torch.searchsorted(cum, base + (40_000_000 // self.spp), right=True)))
                k1 = min(k1, m.numel())
                c = cnt[k0:k1]
                at = torch.repeat_interleave(torch.arange(k0, k1, device="cuda"), c)
                o = torch.arange(at.numel(), device="cuda") - (cum[k0:k1] - c - base)[at - k0]
                k0 = k1
                if not at.numel():
                    continue
                pix = (y0[at] + o // nx[at]) * self.w + x0[at] + o % nx[at]
                s = (pix[:, None] * self.spp + torch.arange(self.spp, device="cuda")).view(-1)
                mm = m[at][:, None].expand(-1, self.spp).reshape(-1)
                v, k, x, y = self.at(mm, s)
                hit = self.inside(v, k, x, y).nonzero()[:, 0]
                v, x, y = [a[hit] for a in v], x[hit], y[hit]
                u, w = self.uv(v, x, y)
                D = (1 - w) * (1 - u) * v[0][:, 2] + (1 - w) * u * v[1][:, 2] + w * (1 - u) * v[2][:, 2] + w * u * v[3][:, 2]
                yield s[hit], D, mm[hit]

    def colour(self, m, s, step=20_000_000):
        """Colour and opacity of hits of samples s on micropolygons m."""
        out = torch.empty((m.numel(), 6), device="cuda", dtype=torch.float64)
        for b in range(0, m.numel(), step):
            mm, ss = m[b:b + step], s[b:b + step]
            v, _, x, y = self.at(mm, ss)
            u, w = self.uv(v, x, y)
            g, i, st = self.corners(mm)
            u, w = (torch.where((self.flags[g] & S.GRID_SMOOTH) != 0, a, torch.zeros_like(a))[:, None] for a in (u, w))
            a = self.cb[g] + i
            for k, src in ((0, self.Ci), (3, self.Oi)):
                out[b:b + step, k:k + 3] = ((1 - u) * (1 - w) * src[a, :3] + u * (1 - w) * src[a + 1, :3] +
                                            (1 - u) * w * src[a + st, :3] + u * w * src[a + st + 1, :3])
        return out


def exact(case, seed):
    c, fr, t, smp = _inputs(case, seed)
    e = _Exact(c, fr, t, smp)
    tests = 0
    for b in range(0, e.n, 1 << 22):
        tests += int(e.boxes(torch.arange(b, min(e.n, b + (1 << 22)), device="cuda"))[3].sum()) * e.spp
    if tests * (3 if e.moving or c["dof"] else 1) > EXACT_TESTS:
        return None
    N = e.w * e.h * e.spp
    opaque = lambda g: (e.flags[g] & S.GRID_OPAQUE) != 0  # noqa: E731
    z = torch.full((N,), FLT_MAX, device="cuda", dtype=torch.float64)
    win = torch.full((N,), -1, device="cuda", dtype=torch.int64)
    for s, D, m in e.hits(opaque):
        before = z[s]
        z.scatter_reduce_(0, s, D, "amin")
        better = (D == z[s]) & (D < before)
        s, m = s[better], m[better]
        win[s] = e.n
        win.scatter_reduce_(0, s, m, "amin")
    col = torch.zeros((N, 6), device="cuda", dtype=torch.float64)
    have = win >= 0
    at = have.nonzero()[:, 0]
    col[at] = e.colour(win[at], at)
    if c["transparent"] > 0:
        parts = [(s[k], D[k], m[k]) for s, D, m in e.hits(lambda g: ~opaque(g)) for k in [D < z[s]]]
        if parts:
            s, D, m = (torch.cat([p[k] for p in parts]) for k in range(3))
            del parts
            # far to near, equal depths later micropolygon first
            for key in (2, 1, 0):
                o = torch.argsort((s, -D, -m)[key], stable=True)
                s, D, m = s[o], D[o], m[o]
            del D, o
            first = torch.searchsorted(s, s)
            rank = torch.arange(s.numel(), device="cuda") - first
            have[s] = True
            for r in range(int(rank.max()) + 1 if rank.numel() else 0):
                k = (rank == r).nonzero()[:, 0]
                sk = s[k]
                d = e.colour(m[k], sk)
                old = col[sk]
                col[sk] = torch.cat([old[:, :3] * (1 - d[:, 3:].clamp(0, 1)) + d[:, :3],
                                     (1 - old[:, 3:]) * d[:, 3:] + old[:, 3:]], 1)
    # pixel filter: the window test by sample position, the weight by the sample's cell
    x0, x1, y0, y1 = fr.crop_window
    W, H, sx, sy = x1 - x0, y1 - y0, fr.shift[0], fr.shift[1]
    wide = math.ceil(c["fw"])
    have = have.view(e.h, e.w, e.spp).double()
    vals = [col[:, k].view(e.h, e.w, e.spp) for k in range(6)] + [z.view(e.h, e.w, e.spp)]
    naov = c["naov"]
    if naov:
        av = torch.zeros((N, naov), device="cuda", dtype=torch.float64)
        g, i, _ = e.corners(win[at])
        av[at] = t["aov"].double()[e.cb[g] + i]
        vals += [av[:, k].view(e.h, e.w, e.spp) for k in range(naov)]
    off = e.pos[e.pi].view(e.h, e.w, e.spp, 2)
    acc = torch.zeros((len(vals), H, W), device="cuda", dtype=torch.float64)
    tot, cnt = (torch.zeros((H, W), device="cuda", dtype=torch.float64) for _ in range(2))
    ci, cj = np.tile(np.arange(c["xs"]), c["ys"]), np.repeat(np.arange(c["ys"]), c["xs"])
    for fy in range(-sy, sy + 1):
        for fx in range(-sx, sx + 1):
            cx, cy = (ci + 0.5) / c["xs"] + fx - 0.5, (cj + 0.5) / c["ys"] + fy - 0.5
            wt = np.where((np.abs(cx) <= wide / 2) & (np.abs(cy) <= wide / 2), _filter_weight(c["filter"], cx, cy, wide), 0.0)
            sl = (slice(fy + sy, fy + sy + H), slice(fx + sx, fx + sx + W))
            o = off[sl]
            inw = ((o[..., 0] + fx - 0.5).abs() <= wide / 2) & ((o[..., 1] + fy - 0.5).abs() <= wide / 2)
            wt = inw * torch.from_numpy(wt).cuda()
            tot += wt.sum(-1)
            ok = have[sl]
            cnt += (inw * ok).sum(-1)
            wt = wt * ok
            for k, v in enumerate(vals):
                acc[k] += (v[sl] * wt).sum(-1)
    some = cnt > 0
    acc = torch.where(some, acc / tot, torch.zeros_like(acc))
    cov = (cnt / e.spp).clamp(max=1.0)
    rgb = (acc[:3] * fr.gain) ** (1.0 / fr.gamma) if fr.gamma != 1.0 else acc[:3] * fr.gain
    alpha = acc[3:6].mean(0) * cov
    out = {"rgba": None, "colour": torch.cat([rgb, acc[3:6], alpha[None]]).permute(1, 2, 0).contiguous().cpu().numpy(),
           # uncovered samples of transparent frames hold the largest float, whose sums overflow in 32 bits
           "depth": None if c["transparent"] > 0 else torch.where(some, acc[6], torch.full_like(cov, FLT_MAX)).cpu().numpy(),
           "coverage": cov.cpu().numpy()}
    if naov:
        out["aov"] = acc[7:].permute(1, 2, 0).contiguous().cpu().numpy()
    return out
