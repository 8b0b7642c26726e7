"""Frames rendered without waiting (aqh_render's sync = 0): when may the memory
their grids came from be used again?  A frame that keeps the device busy for
some milliseconds goes first, so the next frame's uploads are still queued when
its aqh_render returns.  (Its sample tables are below 64 KB: larger ones in
pageable memory make aqh_set_samples wait for the device.)"""
import ctypes as C
import time

import numpy as np
import pytest

from aqsis_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _scene(seed, w=96, h=64, grids=120, xs=3, transparent=False, aov=0, culled=False):
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=w, height=h, xsamples=xs, ysamples=xs, q_dither=0.0)
    g = S.regular_grids(grids, w, h, rng, n=8, zrange=(1.0, 50.0))
    if transparent:
        g.Oi[:, :3] = 0.5
        g.flags &= ~np.int32(S.GRID_OPAQUE)
    if aov:
        g.aov = rng.uniform(0.0, 1.0, (len(g.Ci), aov)).astype(np.float32)
    if culled:
        g.culled = (rng.random(g.micropolygons) < 0.3).astype(np.uint8)
    return S.Scene(fr, g, S.make_samples(fr, rng, 40))


def _busy(h, batched=False):
    """Starts a frame of 8x8 samples whose grids hide little of one another."""
    sc = _scene(99, w=640, h=480, grids=16000, xs=8)
    sc.grids.P[:, 2] = 60.0 - np.repeat(np.arange(16000), 81) * 1e-3   # farthest first
    h.set_mode(batched)
    h.frame_begin(sc.frame)
    h.set_samples(sc.samples)
    h.submit_grids_host(sc.grids)
    h.render(sync=False)
    return sc, h._packed_keep


class _Pinned:
    """Page-locked copies of a scene's grid arrays."""

    def __init__(self, L):
        L.aqh_host_alloc.restype, L.aqh_host_alloc.argtypes = C.c_void_p, [C.c_size_t]
        L.aqh_host_free.argtypes = [C.c_void_p]
        self.L, self.blocks = L, []

    def copy(self, a):
        a = np.ascontiguousarray(a)
        p = self.L.aqh_host_alloc(max(a.nbytes, 16))
        self.blocks.append(p)
        out = np.frombuffer((C.c_char * a.nbytes).from_address(p), a.dtype).reshape(a.shape)
        out[...] = a
        return out

    def free(self):
        for p in self.blocks:
            self.L.aqh_host_free(p)


def _result(aqh_lib, sc, packed3=False):
    h = aqh_lib.Hider(0)
    try:
        h.frame_begin(sc.frame)
        h.set_samples(sc.samples)
        h.submit_grids_host(sc.grids, packed3=packed3)
        h.render(sync=True)
        return h.read_channels(), h.read_aov() if h.naov else None
    finally:
        h.close()


def _same(a, b):
    return a is None and b is None or np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("kind", ["opaque", "culled", "aov", "transparent"])
@pytest.mark.parametrize("packed3,engines", [(False, False), (True, False), (True, True)],
                         ids=["host", "host3", "host3_engines"])
def test_arrays_are_free_when_a_plain_render_returns(aqh_lib, kind, packed3, engines):
    opts = dict(culled=kind == "culled", aov=3 if kind == "aov" else 0, transparent=kind == "transparent")
    a, b = _scene(1, **opts), _scene(2, **opts)
    want = _result(aqh_lib, a, packed3)
    assert not _same(want[0], _result(aqh_lib, b, packed3)[0])
    k = 3 if packed3 else 4
    pin = _Pinned(aqh_lib.load())
    h = aqh_lib.Hider(0)
    try:
        arrays = {f: pin.copy(getattr(a.grids, f)[:, :k]) for f in ("P", "Ci", "Oi")}
        for f in ("culled", "aov"):
            if getattr(a.grids, f, None) is not None:
                arrays[f] = pin.copy(getattr(a.grids, f))
        for f, x in arrays.items():
            setattr(a.grids, f, x)
        if engines:
            assert h.L.aqh_set_host_copy(h.ctx, 1) == 0
        h.frame_begin(a.frame)
        h.set_samples(a.samples)   # (waits: before the busy frame)
        keep = _busy(h)
        h.frame_begin(a.frame)
        h.submit_grids_host(a.grids, packed3=packed3)
        _set_samples(h, a.samples)
        h.render(sync=False)
        for f, x in arrays.items():
            x[...] = getattr(b.grids, f)[:, :k] if f in ("P", "Ci", "Oi") else getattr(b.grids, f)
        h.synchronize()
        assert _same(h.read_channels(), want[0])
        if h.naov:
            assert _same(h.read_aov(), want[1])
        del keep
    finally:
        h.close()
        pin.free()


def _set_samples(h, s):
    """set_samples without its wait."""
    L, real = h.L, h.L.aqh_synchronize
    try:
        L.aqh_synchronize = lambda ctx: 0
        h.set_samples(s)
    finally:
        L.aqh_synchronize = real


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
def test_next_frame_of_single_grids_leaves_the_last_one_alone(aqh_lib, batched):
    """aqh_submit_grid copies into the context's own memory, which the frame
    before may still be uploading."""
    a, b = _scene(3), _scene(4)
    want = _result(aqh_lib, a)
    h = aqh_lib.Hider(0)
    try:
        for sc in (a, b):   # the staging memory has its size
            h.set_mode(batched)
            h.frame_begin(sc.frame)
            h.submit_scene_grids(sc.grids)
            h.set_samples(sc.samples)
            h.render(sync=True)
        keep = _busy(h, batched)
        h.frame_begin(a.frame)
        h.submit_scene_grids(a.grids)
        _set_samples(h, a.samples)
        h.render(sync=False)
        h.frame_begin(b.frame)
        h.submit_scene_grids(b.grids)
        h.synchronize()
        assert _same(h.read_channels(), want[0])
        del keep
    finally:
        h.close()


def test_stats_do_not_wait_for_the_frame(aqh_lib):
    """The list entries are known after binning, long before the frame is done."""
    h = aqh_lib.Hider(0)
    try:
        sc, keep = _busy(h)
        h.synchronize()
        want = h.stats()["tile_grid_pairs"]
        for _ in range(5):
            h.render(sync=False)
            t0 = time.perf_counter()
            got = h.stats()["tile_grid_pairs"]
            t1 = time.perf_counter()
            h.synchronize()
            t2 = time.perf_counter()
            assert got == want
        assert t1 - t0 < t2 - t1, (t1 - t0, t2 - t1)
        del keep
    finally:
        h.close()


def test_refused_frame_has_read_its_arrays(aqh_lib):
    """Camera-space grids without a matrix are refused after their upload was
    queued: aqh_render returns once that is done, with its own message."""
    a = _scene(5)
    a.grids.flags = a.grids.flags | np.int32(S.GRID_CAMERA)
    pin = _Pinned(aqh_lib.load())
    h = aqh_lib.Hider(0)
    try:
        a.grids.P = pin.copy(a.grids.P)
        sc, keep = _busy(h)
        h.frame_begin(a.frame)
        h.submit_grids_host(a.grids)
        _set_samples(h, a.samples)
        with pytest.raises(aqh_lib.AqhError, match="camera-to-raster"):
            h.render(sync=False)
        t0 = time.perf_counter()
        h.synchronize()
        assert time.perf_counter() - t0 < 1e-3   # the busy frame, and so the upload behind it, was done
        del keep, sc
    finally:
        h.close()
        pin.free()
