"""Transparent hits between occluding hits that differ by single roundings, against
the oracle: exact.  Opaque quads lie in one plane, so their hits round to the
plane's depth or just below it; transparent ones lie within a few roundings of
it; and here and there a nearer quad follows.  Whether a transparent hit is a
fragment then hangs on which of the opaque hits before it the reference skips by
early-z."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _scene(seed, xs=4, moving=False, dof=False, grids=420):
    rng = np.random.default_rng(seed)
    w, h = 48, 40
    fr = S.Frame(width=w, height=h, xsamples=xs, ysamples=xs, q_dither=0.0)
    if dof:
        fr.fstop, fr.focal_length, fr.focal_distance, fr.dof_scale = 2.8, 0.4, 20.0, (10.0, 10.0)
    level = np.float32(rng.uniform(30.0, 60.0))
    ulp = np.spacing(level)
    parts = []
    for i in range(grids + 1):
        n = 13 if i == 0 else int(rng.integers(1, 4))
        g = S.regular_grids(1, w, h, rng, n=n, jitter=0.3, zrange=(1.0, 2.0), slope=0.0, origin_margin=10.0)
        origin = np.array([-3.0, -3.0], np.float32) if i == 0 else g.P[0, :2].copy()
        g.P[:, :2] = origin + 5.0 * (g.P[:, :2] - g.P[0, :2])
        kind = 0 if i == 0 else rng.choice(3, p=[0.48, 0.48, 0.04])
        flags = g.flags
        if kind == 0:
            g.P[:, 2] = level
        elif kind == 1:
            g.P[:, 2] = level - ulp * rng.integers(0, 6, len(g.P)).astype(np.float32)
            g.Oi[:, :3] = 0.4
            flags = flags & ~np.int32(S.GRID_OPAQUE)
        else:
            g.P[:, 2] = level * rng.uniform(0.4, 0.8, len(g.P)).astype(np.float32)
        g = dataclasses.replace(g, flags=flags)
        if moving:
            shift = np.zeros_like(g.P)
            shift[:, :2] = rng.uniform(-4.0, 4.0, 2)
            g = dataclasses.replace(g, P=np.concatenate([g.P, g.P + shift]), nkeys=np.full(1, 2, np.int32),
                                    times=np.array([0.0, 1.0], np.float32), tbase=np.zeros(1, np.int32))
        parts.append(g)
    return S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 50))


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
def test_static_frame_matches_oracle(aqh_lib, oracle, seed, batched):
    _check(aqh_lib, oracle, _scene(seed, xs=(4, 4, 2, 1, 5, 8)[seed]), batched)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("kind", ["motion", "dof", "both"])
def test_moving_frame_matches_oracle(aqh_lib, oracle, seed, kind):
    sc = _scene(20 + seed, xs=(4, 4, 2, 1, 5, 4)[seed], moving=kind != "dof", dof=kind != "motion")
    _check(aqh_lib, oracle, sc, False)


def _check(aqh_lib, oracle, sc, batched):
    ref = oracle.render(sc)
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        res = h.render_scene(sc)
    finally:
        h.close()
    assert (ref["nfrag"] > 0).mean() > 0.2
    compare(res, ref)
