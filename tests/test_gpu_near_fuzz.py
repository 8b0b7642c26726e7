"""Random frames (tests/scenes_small.fuzz) made opaque and filled up with grids
until they are sampled near to far, against the oracle: exact.  The odd grids --
depth ties, zero depths, collapsed vertices, huge and mirrored quads, motion --
lie before, among and after the filling."""
import dataclasses

import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests import scenes_small as SS
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _grids_of(g):
    """The grids of a stream one by one."""
    out = []
    for i in range(g.ngrids):
        nv, nk = int((g.cu[i] + 1) * (g.cv[i] + 1)), int(g.nkeys[i])
        pb, cb, tb = int(g.pbase[i]), int(g.cbase[i]), int(g.tbase[i])
        t = g.times[tb:tb + nk] if nk > 1 else np.zeros(1, np.float32)
        out.append(S._pack(g.cu[i:i + 1], g.cv[i:i + 1], g.nkeys[i:i + 1], g.flags[i:i + 1], g.P[pb:pb + nv * nk],
                           g.Ci[cb:cb + nv], g.Oi[cb:cb + nv], np.asarray(t, np.float32), np.zeros(1, np.int32)))
    return out


def _scene(seed):
    sc = SS.fuzz(7000 + seed)
    rng = np.random.default_rng(seed)
    fr = dataclasses.replace(sc.frame, display_z=0, xsamples=(1, 2, 3, 4, 5, 6)[seed % 6], ysamples=(1, 2, 2, 4, 3, 6)[seed % 6])
    g = sc.grids
    Oi = g.Oi.copy()
    Oi[:, :3] = 1.0
    parts = _grids_of(dataclasses.replace(g, Oi=Oi, flags=g.flags | np.int32(S.GRID_OPAQUE)))
    _, _, w, h = fr.sample_region
    want = max(1100, int(26 * w * h / fr.spp)) - sum(p.micropolygons for p in parts)
    have = 0
    while have < want:
        n = int(rng.integers(1, 15))
        p = S.regular_grids(1, fr.width, fr.height, rng, n=n, jitter=float(rng.choice([0.0, 0.3, 0.7])),
                            zrange=(0.5, 60.0), slope=float(rng.choice([0.0, 0.05, 2.0])), origin_margin=6.0)
        if rng.random() < 0.3:
            p.P[:, 2] = float(rng.choice([20.0, 7.5]))
        parts.append(p)
        have += n * n
    parts = [parts[i] for i in rng.permutation(len(parts))]
    return S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 40))


@pytest.mark.parametrize("seed", range(120))
def test_random_deep_frame_matches_oracle(aqh_lib, oracle, seed):
    sc = _scene(seed)
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(seed % 2 == 1)
        res = h.render_scene(sc)
    finally:
        h.close()
    compare(res, oracle.render(sc))
