"""The motion sampler's pruning of tiles and time slices by a micropolygon's
path, its replay of flagged samples, and its fragments of transparent frames
against the oracle (exact: the first only leaves out tests that cannot hit,
the others follow the reference's order).  Frames are several tiles wide, so
paths start, end, cross and graze tiles; each case moves its grids
differently."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _scene(shutter=(0.0, 1.0), times=(0.0, 1.0), move=(30.0, 4.0), dof=False, z=(1.0, 50.0), shear=0.0, static=0.3,
           xs=4, ys=4, flat=False, crop=None, transparent=0.0, keys=2, grids=160, jitter=0.3,
           turn=0.0, levels=4, seed=0):
    """Two-key grids over a 72x56 frame, each displaced along `move` turned by a
    random angle, key 1 sheared by `shear`; a share `static` has one key, a share
    `transparent` lets what lies behind it through."""
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=72, height=56, xsamples=xs, ysamples=ys, q_dither=0.0, shutter=shutter, crop=crop)
    if dof:
        fr.fstop, fr.focal_length, fr.focal_distance, fr.dof_scale = 2.8, 0.4, 20.0, (40.0, 40.0)
    parts = []
    for i in range(grids):
        n = int(rng.integers(1, 9))
        g = S.regular_grids(1, 72, 56, rng, n=n, zrange=z, slope=0.0 if flat else 0.02, motion=1.0, jitter=jitter,
                            origin_margin=10.0)
        P = g.P.reshape(2, -1, 4)
        a = rng.uniform(0, 2 * np.pi)
        d = np.array([np.cos(a) * move[0] - np.sin(a) * move[1], np.sin(a) * move[0] + np.cos(a) * move[1]])
        P[1, :, :2] = P[0, :, :2] + d + shear * (P[0, :, :2] - P[0, 0, :2])[:, ::-1]
        if turn:
            c, sn = np.cos(turn), np.sin(turn)
            P[1, :, :2] = P[1, 0, :2] + (P[1, :, :2] - P[1, 0, :2]) @ np.array([[c, -sn], [sn, c]], np.float32)
        if flat:
            P[:, :, 2] = float(rng.integers(2, 1 + levels))   # coplanar layers: depths tie and round below their bounds
        if rng.random() < transparent:
            g.Oi[:, :3] = rng.uniform(0.1, 1.05, (len(g.Oi), 3))   # some corners opaque
            g.flags &= ~np.int32(S.GRID_OPAQUE)
        if rng.random() < static:
            g = dataclasses.replace(g, P=P[0].copy(), nkeys=np.ones(1, np.int32), times=np.zeros(1, np.float32),
                                    tbase=np.zeros(1, np.int32))
        else:
            # further keys on the way, off the straight line
            k = np.linspace(0.0, 1.0, keys)[:, None, None]
            way = P[:1] + k * (P[1:] - P[:1])
            way[1:-1, :, :2] += rng.uniform(-2.0, 2.0, (keys - 2, 1, 2))
            g = dataclasses.replace(g, P=way.reshape(-1, 4).astype(np.float32), nkeys=np.full(1, keys, np.int32),
                                    times=np.linspace(times[0], times[1], keys).astype(np.float32))
        parts.append(g)
    return S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 50))


CASES = {
    "long": dict(), "short": dict(move=(0.3, 0.0)), "rest": dict(move=(0.0, 0.0)), "huge": dict(move=(4000.0, 0.0)),
    "beyond_int16": dict(move=(90000.0, 3.0)), "shear": dict(shear=0.8, move=(9.0, 2.0)),
    "keys_inside_shutter": dict(times=(0.3, 0.6)), "keys_around_shutter": dict(times=(-1.0, 3.0)),
    "late_shutter": dict(shutter=(100.0, 100.5), times=(100.0, 100.5)), "reversed_keys": dict(times=(1.0, 0.0)),
    "dof": dict(dof=True, move=(12.0, 1.0)), "dof_depth_reaches_zero": dict(dof=True, z=(-0.05, 0.05), move=(8.0, 0.0)),
    "samples_1x1": dict(xs=1, ys=1), "samples_16x16": dict(xs=16, ys=16, move=(10.0, 0.0)), "samples_5x3": dict(xs=5, ys=3),
    "crop": dict(crop=(13, 61, 9, 40)), "flat": dict(flat=True), "flat_dof": dict(flat=True, dof=True, move=(6.0, 0.0)),
    "deep": dict(grids=900, move=(5.0, 1.0)), "deep_dof": dict(grids=900, dof=True, move=(4.0, 0.0)),
    "deep_static_dof": dict(grids=900, dof=True, static=1.0), "deep_folded": dict(grids=700, jitter=0.9, move=(3.0, 0.0)),
    "deep_turning": dict(grids=700, turn=1.2, move=(6.0, 0.0)), "deep_4_keys": dict(grids=700, keys=4, move=(8.0, 0.0)),
    "deep_flat": dict(grids=700, flat=True, levels=60, move=(3.0, 0.0)),
    "deep_near_eye": dict(grids=700, dof=True, z=(0.05, 2.0), move=(2.0, 0.0)),
    "deep_beyond_keys": dict(grids=700, times=(0.4, 0.5), move=(4.0, 0.0)),
    "transparent": dict(transparent=0.5, move=(12.0, 2.0)), "transparent_all": dict(transparent=1.0, move=(6.0, 0.0)),
    "transparent_dof": dict(transparent=0.5, dof=True, move=(12.0, 2.0)),
    "transparent_flat": dict(transparent=0.5, flat=True, move=(9.0, 0.0)),
    "transparent_4_keys": dict(transparent=0.4, keys=4, move=(14.0, 3.0)), "4_keys": dict(keys=4, move=(14.0, 3.0)),
    "transparent_16x16": dict(transparent=0.5, xs=16, ys=16, move=(8.0, 0.0)),
    "transparent_1x1": dict(transparent=0.6, xs=1, ys=1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_moving_frame_matches_oracle(hider, oracle, name):
    sc = _scene(seed=sorted(CASES).index(name), **CASES[name])
    compare(hider.render_scene(sc), oracle.render(sc), exact_pixels=True)
