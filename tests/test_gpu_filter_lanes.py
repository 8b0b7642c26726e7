"""Rolling windows tested at sample positions, half of each group of four samples
in each of a column's two lanes, and the sizes on either side of the choice of
kernel: against the oracle, exact.  Sample counts leave every remainder of four."""
import numpy as np
import pytest

from tests.test_gpu_filter_windows import _scene
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outside", [False, True], ids=["inside", "outside"])
@pytest.mark.parametrize("xs,ys", [(17, 1), (9, 2), (19, 1), (5, 5), (7, 3), (10, 10)])
@pytest.mark.parametrize("filt,fw", [("gaussian", 2.0), ("catmull-rom", 3.0), ("triangle", 4.0)])
def test_position_tests_match_oracle(hider, oracle, filt, fw, xs, ys, outside):
    sc = _scene(131, 23, xs, ys, filt, fw, 0, seed=xs + ys)
    if outside:   # some samples of a pixel lie beyond its edges, some on them
        rng = np.random.default_rng(xs)
        p = sc.samples.pos
        at = rng.random(p.shape) < 0.2
        p[at] = rng.choice(np.array([-0.6, 0.0, 0.5, 1.0, 1.4], np.float32), int(at.sum()))
    compare(hider.render_scene(sc), oracle.render(sc), exact_pixels=True)


@pytest.mark.parametrize("w,h,xs,ys,fw", [(300, 411, 2, 2, 4.0), (300, 411, 2, 2, 5.0), (520, 480, 2, 2, 4.0),
                                          (640, 480, 4, 4, 4.0), (640, 472, 4, 4, 5.0), (640, 500, 1, 1, 4.0)])
def test_kernel_choice_matches_oracle(hider, oracle, w, h, xs, ys, fw):
    sc = _scene(w, h, xs, ys, "mitchell", fw, 0, seed=w + h)
    compare(hider.render_scene(sc), oracle.render(sc), exact_pixels=True)


@pytest.mark.parametrize("xs,ys,fw", [(4, 4, 2.0), (4, 4, 3.0), (5, 3, 4.0), (6, 6, 5.0), (6, 6, 2.0)])
def test_asking_for_tiles_changes_no_pixel(aqh_lib, oracle, xs, ys, fw):
    """filter_ctas_per_sm makes windows that would roll go by tiles."""
    sc = _scene(300, 411, xs, ys, "catmull-rom", fw, 0, seed=xs)
    ref = oracle.render(sc)
    h = aqh_lib.Hider(0)
    try:
        for ctas in (0, 1, 8):
            h.set_tuning(filter_ctas_per_sm=ctas)
            compare(h.render_scene(sc), ref, exact_pixels=True)
    finally:
        h.close()
