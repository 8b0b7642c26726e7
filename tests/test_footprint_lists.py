"""The grid lists and the redo list in the serving path's HBM footprint estimate
(aqh_job_footprint), host only: the terms that grow with grids and tiles."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_footprint import _footprint, _within_margin


def _scene(ngrids, w, h, opaque=True):
    rng = np.random.default_rng(3)
    fr = S.Frame(width=w, height=h, xsamples=2, ysamples=2)
    g = S.regular_grids(ngrids, w, h, rng, n=1)
    if not opaque:
        g = dataclasses.replace(g, flags=g.flags & ~np.int32(S.GRID_OPAQUE))
    return S.Scene(fr, g, S.make_samples(fr, rng, 8))


def _lists(ngrids, w, h):
    """Both orders of the grid lists: the batched form's 16 super-tiles per grid, or every
    super-tile (128 pixels) in the plain form, up to 2^21 entries."""
    x0, y0, sw, sh = _scene(1, w, h).frame.sample_region
    nst = -(-sw // 128) * -(-sh // 128)
    return 2 * 4 * max(16 * ngrids + 4096, min(ngrids * nst, 1 << 21))


@pytest.mark.parametrize("opaque", [True, False], ids=["opaque", "transparent"])
@pytest.mark.parametrize("w,h,a,b", [(320, 240, 100, 5000), (1920, 1080, 100, 5000), (1920, 1080, 1000, 40000)])
def test_grids_add_their_list_room(aqh_lib, w, h, a, b, opaque):
    lo, hi = _scene(a, w, h, opaque=opaque), _scene(b, w, h, opaque=opaque)
    n = b - a
    # four vertices with P, Ci and Oi; tables; rectangle and nearest depth; depth slack and irregular mask
    per_grid = 4 * (16 + 32) + (5 * 4 + 3 * 8) + (16 + 4) + (8 + 4 * 32)
    terms = n * per_grid + 4 * (hi.grids.times.size - lo.grids.times.size) + _lists(b, w, h) - _lists(a, w, h)
    assert _within_margin(_footprint(hi) - _footprint(lo), terms)


def test_tiles_add_their_redo_entries(aqh_lib):
    """16 more rows of a frame 1000 pixels wide: one more row of 16x16 tiles (63 of them)."""
    a, b = _scene(10, 1000, 302), _scene(10, 1000, 318)
    ha, hb = a.frame.sample_region[3], b.frame.sample_region[3]
    assert a.frame.sample_region[2] == 1002 and (ha, hb) == (304, 320)
    px, disp = 1002 * (hb - ha), 1000 * 16
    # per sample: store, debug arrays, window word; per pixel: pattern choices; per display pixel: channels, rgba
    terms = px * 4 * (32 + 12 + 4) + px * 4 * 5 + disp * 40 + 63 * 8 * 4
    assert _within_margin(_footprint(b) - _footprint(a), terms)
