"""Opaque static tiles about as many of whose pixels are undecided as the near to
far sampler hands on singly, against the oracle: exact.  Small patches lie in
the plane of a background, so most of their pixels are found undecided only
when the tile's samples are resolved, after the tile was counted as decided."""
import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _grid(rng, n, x, y, z, spacing=1.0):
    g = S.regular_grids(1, 64, 64, rng, n=n, jitter=0.3, zrange=(1.0, 2.0), slope=0.0)
    g.P[:, :2] = np.array([x, y], np.float32) + spacing * (g.P[:, :2] - g.P[0, :2])
    g.P[:, 2] = z
    return g


def _scene(seed, xs, tiles=8):
    """A plane of 16x16 background grids with one patch of up to 4x4 pixels in each, in
    an order that puts patches before, among and after the background."""
    rng = np.random.default_rng(seed)
    w = 16 * tiles
    fr = S.Frame(width=w, height=w, xsamples=xs, ysamples=xs, q_dither=0.0)
    z = np.float32(rng.uniform(3.0, 50.0))
    parts = []
    for ty in range(-1, tiles + 1):
        for tx in range(-1, tiles + 1):
            parts.append(_grid(rng, 16, 16.0 * tx, 16.0 * ty, z))
            n = int(rng.integers(1, 5))
            at = rng.uniform(2.0, 13.0 - n, 2)
            parts.append(_grid(rng, n, 16.0 * tx + at[0], 16.0 * ty + at[1], z, rng.uniform(0.6, 0.9)))
    parts = [parts[i] for i in rng.permutation(len(parts))]
    return S.Scene(fr, S.concat_grids(parts), S.make_samples(fr, rng, 40))


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("seed,xs", [(0, 5), (1, 4), (2, 4), (3, 4), (4, 8)])
def test_tiles_at_the_limit_match_oracle(aqh_lib, oracle, seed, xs, batched):
    sc = _scene(seed, xs)
    ref = oracle.render(sc)
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        for _ in range(3):
            compare(h.render_scene(sc), ref, exact_pixels=True)
    finally:
        h.close()
