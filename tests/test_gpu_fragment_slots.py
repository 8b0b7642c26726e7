"""Pool slots of transparent frames: the reported number is that of the fragments
stored, not of the slots the samplers reserved, and slots left empty do not make
a frame of few samples per pixel outgrow the pool."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests import test_gpu_mixed as MX
from tests import test_gpu_motion_paths as MP

pytestmark = pytest.mark.gpu


def _render(aqh_lib, sc, batched):
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        return h.render_scene(sc)
    finally:
        h.close()


def _transparent(sc, share, seed=0):
    """Makes that share of the grids transparent."""
    g = sc.grids
    rng = np.random.default_rng(seed)
    pick = rng.random(g.ngrids) < share
    nv = (g.cu + 1) * (g.cv + 1)
    for i in np.flatnonzero(pick):
        g.Oi[g.cbase[i]:g.cbase[i] + nv[i], :3] = 0.5
    flags = np.where(pick, g.flags & ~np.int32(S.GRID_OPAQUE), g.flags).astype(np.int32)
    return dataclasses.replace(sc, grids=dataclasses.replace(g, flags=flags))


CASES = {
    "mixed": lambda: MX._scene(seed=5), "mixed_1x1": lambda: MX._scene(seed=6, xs=1, ys=1),
    "mixed_16x16": lambda: MX._scene(seed=7, xs=16, ys=16, grids=40), "mixed_flat": lambda: MX._scene(seed=8, levels=3),
    "motion": lambda: _transparent(MP._scene(seed=5), 0.5), "motion_1x1": lambda: _transparent(MP._scene(seed=6, xs=1, ys=1), 0.7),
    "motion_dof": lambda: _transparent(MP._scene(seed=7, dof=True, move=(6.0, 1.0)), 0.5),
}


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fragments_are_counted_not_slots(aqh_lib, name, batched):
    res = _render(aqh_lib, CASES[name](), batched)
    assert res["nfrag"].sum() > 0
    assert res["stats"]["fragments"] == res["nfrag"].sum()


@pytest.mark.parametrize("moving", [False, True], ids=["static", "motion"])
def test_one_sample_per_pixel_fits_the_pool(aqh_lib, moving):
    """1.5 fragments per sample, where the pool holds two, are stored at the first attempt."""
    rng = np.random.default_rng(1)
    w, h, n = 1100, 800, 20
    fr = S.Frame(width=w, height=h, xsamples=1, ysamples=1, q_dither=0.0)
    parts = []
    for layer in range(2):
        for y in range(-2, h // n + 1):
            for x in range(-2, w // n + 1):
                opaque = layer == 1 and (x + y) % 2 == 0
                g = S.regular_grids(1, w, h, rng, n=n, jitter=0.0, zrange=(1.0, 2.0), slope=0.0)
                g.P[:, :2] = g.P[:, :2] - g.P[0, :2] + np.array([x * n, y * n], np.float32)
                g.P[:, 2] = 9.0 if opaque else 3.0 + layer
                if not opaque:
                    g.Oi[:, :3] = 0.5
                    g = dataclasses.replace(g, flags=g.flags & ~np.int32(S.GRID_OPAQUE))
                if moving:
                    P1 = g.P.copy()
                    P1[:, 0] += 0.5
                    g = dataclasses.replace(g, P=np.concatenate([g.P, P1]), nkeys=np.full(1, 2, np.int32),
                                            times=np.array([0.0, 1.0], np.float32), tbase=np.zeros(1, np.int32))
                parts.append(g)
    res = _render(aqh_lib, S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 60)), True)
    assert 1.4 < res["nfrag"].mean() < 1.6
    assert res["stats"]["fragments"] == res["nfrag"].sum()
    assert res["stats"]["rerenders"] == 0
