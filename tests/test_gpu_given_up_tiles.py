"""Opaque static frames of many tiles, most of which the near to far sampler
gives up, against the oracle: exact.  Once enough tiles were given up the rest
goes to the ordered kernel untried; tiles that would have been decided lie
before, between and after those that are not."""
import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _scene(seed, flat, w=640, h=420, xs=2, layers=4.0):
    """`flat`: which grids lie in one plane, by the position of their first vertex."""
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=w, height=h, xsamples=xs, ysamples=xs, q_dither=0.0)
    n = 12
    g = S.regular_grids(int(layers * w * h / (n * n)), w, h, rng, n=n, jitter=0.3, zrange=(1.0, 40.0), slope=0.02,
                        origin_margin=8.0)
    P = g.P.reshape(g.ngrids, (n + 1) ** 2, 4)
    plane = flat(P[:, 0, 0] / w, P[:, 0, 1] / h)
    P[plane, :, 2] = np.float32(7.3)
    g.P = P.reshape(-1, 4)
    return S.Scene(fr, g, S.make_samples(fr, rng, 50))


CASES = {
    "all": (lambda x, y: x < 9.0, 2), "top": (lambda x, y: y < 0.7, 2), "bottom": (lambda x, y: y > 0.4, 2),
    "stripes": (lambda x, y: (x * 5.0) % 1.0 < 0.8, 2), "none": (lambda x, y: x > 9.0, 2), "all_3x3": (lambda x, y: x < 9.0, 3),
}


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_frame_matches_oracle(aqh_lib, oracle, name, batched):
    flat, xs = CASES[name]
    sc = _scene(sorted(CASES).index(name), flat, xs=xs)
    ref = oracle.render(sc)
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(batched)
        for _ in range(2):
            compare(h.render_scene(sc), ref, exact_pixels=True)
    finally:
        h.close()
