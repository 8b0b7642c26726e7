"""Which frames are sampled near to far depends on their size (number of samples,
micropolygons per pixel): frames on both sides of each line, in both execution
forms, against the oracle: exact."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _static(w, h, xs, mps, seed):
    """About `mps` micropolygons over w x h pixels, some of their depths tied."""
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=w, height=h, xsamples=xs, ysamples=xs, q_dither=0.0)
    g = S.regular_grids(max(1, round(mps / 49)), w, h, rng, n=7, jitter=0.3, zrange=(1.0, 40.0), slope=0.05)
    P = g.P.reshape(g.ngrids, 64, 4)
    P[::5, :, 2] = np.float32(11.3)
    g.P = P.reshape(-1, 4)
    return S.Scene(fr, g, S.make_samples(fr, rng, 50))


def _moving(mps, dof, seed):
    """Exactly `mps` micropolygons: grids of 4x4 and single ones."""
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=48, height=36, xsamples=4, ysamples=4, q_dither=0.0)
    if dof:
        fr.fstop, fr.focal_length, fr.focal_distance, fr.dof_scale = 2.8, 0.4, 20.0, (12.0, 12.0)
    parts = [S.regular_grids(mps // 16, 48, 36, rng, n=4, zrange=(1.0, 40.0), motion=5.0)]
    if mps % 16:
        parts.append(S.regular_grids(mps % 16, 48, 36, rng, n=1, zrange=(1.0, 40.0), motion=5.0))
    g = S.concat_grids(parts)
    assert g.micropolygons == mps
    return S.Scene(fr, g, S.make_samples(fr, rng, 50))


def _check(aqh_lib, oracle, sc, batched):
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        res = h.render_scene(sc)
    finally:
        h.close()
    compare(res, oracle.render(sc), exact_pixels=True)


# micropolygons times samples a pixel, per pixel: 24 is the line below 16,384 micropolygons, 12 above
@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("w,h,xs,per_pixel", [
    (24, 18, 1, 20.0), (24, 18, 1, 32.0), (40, 30, 2, 20.0), (40, 30, 2, 32.0), (60, 45, 4, 20.0), (60, 45, 4, 30.0),
    (180, 140, 1, 10.0), (180, 140, 1, 14.0), (180, 140, 2, 10.0), (180, 140, 2, 14.0), (240, 180, 4, 10.0),
    (240, 180, 4, 14.0)])
def test_static_frames_around_the_line(aqh_lib, oracle, w, h, xs, per_pixel, batched):
    _check(aqh_lib, oracle, _static(w, h, xs, per_pixel * w * h / (xs * xs), int(per_pixel) + xs), batched)


@pytest.mark.parametrize("w", [358, 366])
def test_static_frames_around_the_sample_count(aqh_lib, oracle, w):
    """16 samples: 360x360 pixels of the sample region are just below 2^21, 368x360 just above."""
    _check(aqh_lib, oracle, _static(w, 358, 4, 0.2 * w * 358, w), True)


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("dof", [False, True], ids=["motion", "both"])
@pytest.mark.parametrize("mps", [1023, 1024])
def test_moving_frames_around_the_line(aqh_lib, oracle, mps, dof, batched):
    _check(aqh_lib, oracle, _moving(mps, dof, mps), batched)


@pytest.mark.parametrize("nkeys", [1, 3])
def test_small_moving_frames_of_other_key_counts(aqh_lib, oracle, nkeys):
    """Depth of field alone, and more keys than the two-key records hold."""
    sc = _moving(512, True, nkeys)
    g = sc.grids
    P = g.P.reshape(g.ngrids, 2, 25, 4)
    P = P[:, :1] if nkeys == 1 else np.stack([P[:, 0], 0.4 * P[:, 0] + 0.6 * P[:, 1], P[:, 1]], 1)
    n = g.ngrids
    sc = dataclasses.replace(sc, grids=dataclasses.replace(
        g, P=np.ascontiguousarray(P).reshape(-1, 4).astype(np.float32), nkeys=np.full(n, nkeys, np.int32),
        pbase=np.arange(n, dtype=np.int64) * 25 * nkeys, tbase=np.zeros(n, np.int32),
        times=np.linspace(0.0, 1.0, nkeys).astype(np.float32)))
    _check(aqh_lib, oracle, sc, True)
