"""Moving frames whose sample offsets leave the pixel, or whose lens samples
leave the lens, against the oracle, sample by sample: exact.  A sample is tested
wherever its pixel is, so a micropolygon's path does not say which tiles and
time slices can hit it."""
import numpy as np
import pytest

from tests.test_gpu_motion_paths import _scene
from tests.test_gpu_parity import close_or_same

pytestmark = pytest.mark.gpu

CASES = {
    "offsets_1x1": dict(pos=9.0, xs=1, ys=1), "lens": dict(lens=4.0, dof=True),
    "lens_1x1": dict(lens=4.0, dof=True, xs=1, ys=1), "offsets_and_lens": dict(pos=9.0, lens=4.0, dof=True),
}


@pytest.mark.parametrize("seed", range(5))
@pytest.mark.parametrize("name", sorted(CASES))
def test_offsets_outside_match_oracle(hider, oracle, name, seed):
    opts = dict(CASES[name])
    pos, lens = opts.pop("pos", 0.0), opts.pop("lens", 0.0)
    sc = _scene(seed=10 * seed + 1, move=(24.0, 24.0), static=0.1, **opts)
    rng = np.random.default_rng(seed)
    s = sc.samples
    if pos:
        s.pos = rng.uniform(-pos, 1.0 + pos, s.pos.shape).astype(np.float32)
    if lens:
        s.dof = rng.uniform(-lens, 1.0 + lens, s.dof.shape).astype(np.float32)
    ref = oracle.render(sc)
    assert (ref["winner"] >= 0).mean() > 0.01
    res = hider.render_scene(sc)
    for k in ("winner", "nfrag", "valid"):
        assert np.array_equal(res[k], ref[k]), "%s differs at %d samples" % (k, int((res[k] != ref[k]).sum()))
    assert np.array_equal(res["occlz"].view(np.uint32), ref["occlz"].view(np.uint32))
    assert close_or_same(res["sdata"], ref["sdata"]).all()
