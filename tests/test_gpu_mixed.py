"""Static frames that mix opaque and transparent micropolygons (the mixed
sampler) against the oracle, in both execution forms: exact, since it keeps the
reference's order of early-z, stores and fragments.  Grids overlap many deep,
in interleaved order, so transparent hits land before, between and behind
occluding ones of the same round of candidates."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _scene(transparent=0.4, grids=220, xs=4, ys=4, z=(1.0, 40.0), levels=0, big=False, matte=False, lod=False,
           triangular=False, crop=None, seed=0):
    """`levels`: depths from that many flat planes, so depths tie and round below their bounds."""
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=70, height=45, xsamples=xs, ysamples=ys, q_dither=0.0, crop=crop)
    parts = []
    for _ in range(grids):
        g = S.regular_grids(1, 70, 45, rng, n=int(rng.integers(1, 12)), zrange=z, slope=0.0 if levels else 0.05,
                            origin_margin=8.0)
        if big:
            g.P[:, :2] = g.P[0, :2] + 4.0 * (g.P[:, :2] - g.P[0, :2])
        if levels:
            g.P[:, 2] = float(rng.integers(-1, levels))
        flags = g.flags
        if rng.random() < transparent:
            g.Oi[:, :3] = rng.uniform(0.1, 1.05, (len(g.Oi), 3))   # some corners opaque
            flags = flags & ~np.int32(S.GRID_OPAQUE)
        if matte:
            flags = flags | np.int32(rng.choice([0, S.GRID_MATTE, S.GRID_MATTEALPHA]))
        if triangular and rng.random() < 0.4:
            flags = flags | np.int32(S.GRID_TRIANGULAR)
        parts.append(dataclasses.replace(g, flags=flags))
    sc = S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 60))
    return S.with_lod(sc, seed=seed) if lod else sc


CASES = {
    "interleaved": dict(), "few_transparent": dict(transparent=0.05), "mostly_transparent": dict(transparent=0.9),
    "flat_levels": dict(levels=4), "one_level": dict(levels=2), "big": dict(big=True, grids=60), "matte": dict(matte=True),
    "lod": dict(lod=True), "triangular": dict(triangular=True), "samples_1x1": dict(xs=1, ys=1),
    "samples_16x16": dict(xs=16, ys=16, grids=60), "samples_5x3": dict(xs=5, ys=3), "crop": dict(crop=(17, 62, 3, 40)),
    "depth_crosses_zero": dict(z=(-0.3, 0.3)),
}


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_mixed_frame_matches_oracle(aqh_lib, oracle, name, batched):
    sc = _scene(seed=sorted(CASES).index(name), **CASES[name])
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        res = h.render_scene(sc)
    finally:
        h.close()
    compare(res, oracle.render(sc))


def test_nan_depths_combine_in_insertion_order(aqh_lib, oracle):
    """A list holding a NaN depth has no sorted order; what it composites to
    must not depend on the order its fragments were appended in."""
    sc = _scene(transparent=0.8, seed=3)
    sc.grids.P[::37, 2] = np.nan
    out = []
    for batched in (False, True):
        h = aqh_lib.Hider(0)
        try:
            h.set_mode(batched)
            out.append(h.render_scene(sc))
        finally:
            h.close()
    a, b = out
    for k in ("winner", "nfrag", "valid"):
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(a["sdata"].view(np.uint32), b["sdata"].view(np.uint32))
