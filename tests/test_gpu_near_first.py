"""Opaque static frames deep enough to be sampled near to far, against the
oracle, whose micropolygons go in insertion order: exact.  The cases aim at
what that rests on: depths below their bound's min z (rounding, Newton steps on
folded and sliver quads), ties and near ties between layers, zero and NaN
depths, grids of more micropolygons than are analysed, tile edges."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _scene(w=62, h=41, xs=4, ys=4, layers=7.0, n=(4, 14), jitter=0.3, spacing=1.0, slope=0.02, z=(1.0, 60.0), levels=0,
           stretch=1.0, crop=None, smooth=True, seed=0):
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=w, height=h, xsamples=xs, ysamples=ys, q_dither=0.0, crop=crop)
    parts, have = [], 0
    # `layers` micropolygons per pixel, so that the frame qualifies whatever their size
    while have < layers * (w + 2) * (h + 2):
        k = int(rng.integers(n[0], n[1] + 1))
        g = S.regular_grids(1, w, h, rng, n=k, jitter=jitter, zrange=z, slope=slope, origin_margin=k * spacing,
                            smooth=smooth)
        o = g.P[0, :2].copy()
        g.P[:, :2] = o + (g.P[:, :2] - o) * np.array([spacing, spacing * stretch], np.float32)
        if levels:
            g.P[:, 2] = float(rng.integers(1, levels + 1))
        if rng.random() < 0.2:
            g.P[:] = g.P.reshape(k + 1, k + 1, 4)[:, ::-1].reshape(-1, 4)   # clockwise
        parts.append(g)
        have += k * k
    return S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 60))


CASES = {
    "layers": dict(), "steep": dict(slope=3.0), "folded": dict(jitter=0.9), "regular": dict(jitter=0.0),
    "slivers": dict(stretch=0.02), "tiny": dict(spacing=0.05, n=(10, 31)), "big": dict(spacing=6.0, n=(1, 4)),
    "one_level": dict(levels=1, slope=0.0, jitter=0.3), "levels": dict(levels=4, slope=0.0),
    "near_levels": dict(z=(10.0, 10.00001), slope=1e-7), "depth_crosses_zero": dict(z=(-0.4, 0.4)),
    "behind": dict(z=(-50.0, -1.0)), "large_grids": dict(n=(33, 40), layers=9.0), "unit_grids": dict(n=(1, 1), layers=5.0),
    "samples_1x1": dict(xs=1, ys=1), "samples_16x16": dict(xs=16, ys=16, w=20, h=14), "samples_5x3": dict(xs=5, ys=3),
    "crop": dict(crop=(11, 53, 2, 40)), "constant": dict(smooth=False), "far": dict(z=(1e6, 1e7), slope=100.0),
}


def _both(aqh_lib, scene, batched, packed):
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        if not packed:
            return h.render_scene(scene)
        h.frame_begin(scene.frame)
        h.set_samples(scene.samples)
        h.submit_grids_host(scene.grids)
        h.render(sync=True)
        res = {"channels": h.read_channels(), "quantized": h.read_quantized()}
        res.update(h.read_samples())
        return res
    finally:
        h.close()


@pytest.mark.parametrize("batched,packed", [(False, False), (True, False), (True, True)],
                         ids=["plain", "batched", "packed"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_deep_frame_matches_oracle(aqh_lib, oracle, name, batched, packed):
    sc = _scene(seed=sorted(CASES).index(name), **CASES[name])
    compare(_both(aqh_lib, sc, batched, packed), oracle.render(sc), exact_pixels=True)


@pytest.mark.parametrize("seed", range(12))
def test_deep_frame_with_options(aqh_lib, oracle, seed):
    """Detail levels, trim curves, culled micropolygons, camera space."""
    sc = _scene(seed=100 + seed, jitter=(0.0, 0.3, 0.6)[seed % 3])
    rng = np.random.default_rng(seed)
    if seed % 4 == 0:
        sc = S.with_lod(sc, seed=seed)
    elif seed % 4 == 1:
        sc = S.with_trim(sc, seed=seed)
    elif seed % 4 == 2:
        sc.grids.culled = (rng.random(sc.grids.micropolygons) < 0.2).astype(np.uint8)
    else:
        sc = S.to_camera_space(sc, every=2)
    compare(_both(aqh_lib, sc, seed % 2 == 1, False), oracle.render(sc), exact_pixels=True)


def test_deep_frame_with_nan_depths(aqh_lib):
    """A NaN depth sends its tile to the ordered kernel: both forms agree, and
    nothing but the tiles the NaN corners lie in changes."""
    sc = _scene(seed=5)
    clean = _both(aqh_lib, sc, False, False)
    g = sc.grids
    P = g.P.copy()
    P[len(P) // 2, 2] = np.nan
    sc = S.Scene(sc.frame, dataclasses.replace(g, P=P), sc.samples)
    a, b = _both(aqh_lib, sc, False, False), _both(aqh_lib, sc, True, True)
    assert np.array_equal(a["winner"], b["winner"])
    assert np.array_equal(a["occlz"].view(np.uint32), b["occlz"].view(np.uint32))
    assert (a["winner"] != clean["winner"]).mean() < 0.01


def test_list_entries_are_reported(aqh_lib):
    """A plain frame that did not wait for binning reports its list entries on
    request, as the batched form does; each of two frames its own."""
    a, b = _scene(seed=1), _scene(seed=2, w=300, h=200, layers=1.0)
    want, got = [], []
    for batched, out in ((True, want), (False, got)):
        h = aqh_lib.Hider(0)
        try:
            h.set_mode(batched)
            for sc in (a, b):
                h.frame_begin(sc.frame)
                h.set_samples(sc.samples)
                h.submit_grids_host(sc.grids)
                h.render(sync=batched)
                out.append(h.stats()["tile_grid_pairs"])
                h.synchronize()
        finally:
            h.close()
    assert want == got and min(want) > 0 and want[0] != want[1]
