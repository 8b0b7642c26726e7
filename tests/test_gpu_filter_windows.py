"""The rolling filters of 3x3 and 5x5 windows, colour and output variables,
against the oracle: exact, since every sum keeps the reference's order.  Image
sizes around the runs of rows and columns a thread block owns, with and
without window masks (16 samples or fewer have them), windows that hold every
sample of the neighbourhood and windows that do not."""
import numpy as np
import pytest

from aqsis_gb300 import scene as S
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def _scene(w, h, xs, ys, filt, fw, naov, seed, crop=None):
    rng = np.random.default_rng(seed)
    fr = S.Frame(width=w, height=h, xsamples=xs, ysamples=ys, filter=filt, xfilter=fw, yfilter=fw, q_dither=0.0,
                 crop=crop)
    g = S.regular_grids(max(1, w * h // 60), w, h, rng, n=7, origin_margin=5.0)
    sc = S.Scene(fr, g, S.make_samples(fr, rng, 40))
    return S.with_aov(sc, naov, seed=seed) if naov else sc


@pytest.mark.parametrize("filt,fw", [("catmull-rom", 3.0), ("gaussian", 2.0), ("mitchell", 4.0), ("sinc", 5.0)])
@pytest.mark.parametrize("xs,ys", [(1, 1), (5, 3), (4, 4), (6, 5), (8, 8)])
@pytest.mark.parametrize("w,h", [(1, 1), (127, 7), (130, 17), (300, 411)])
def test_rolling_windows_match_oracle(hider, oracle, filt, fw, xs, ys, w, h):
    sc = _scene(w, h, xs, ys, filt, fw, 0, seed=w + 10 * xs)
    compare(hider.render_scene(sc), oracle.render(sc), exact_pixels=True)


@pytest.mark.parametrize("naov", [1, 2, 3, 4, 5, 11])
@pytest.mark.parametrize("fw,xs,ys", [(3.0, 4, 4), (4.0, 5, 3), (5.0, 6, 6), (1.0, 4, 4), (6.0, 2, 2)])
def test_output_variables_match_oracle(hider, oracle, naov, fw, xs, ys):
    sc = _scene(37, 19, xs, ys, "catmull-rom", fw, naov, seed=naov, crop=(2, 33, 1, 18))
    a, b = hider.render_scene(sc), oracle.render(sc)
    compare(a, b, exact_pixels=True)
    assert np.array_equal(a["aov"].view(np.uint32), np.asarray(b["aov"], np.float32).reshape(a["aov"].shape).view(np.uint32))


def test_output_variables_of_device_grids(aqh_lib, oracle):
    import torch
    sc = _scene(50, 30, 4, 4, "mitchell", 4.0, 3, seed=9)
    g = sc.grids
    d = {k: torch.from_numpy(np.ascontiguousarray(getattr(g, k))).cuda() for k in (
        "cu", "cv", "nkeys", "flags", "pbase", "cbase", "tbase", "times", "P", "Ci", "Oi", "aov")}
    torch.cuda.synchronize()
    h = aqh_lib.Hider(0)
    try:
        h.set_mode(True)
        h.frame_begin(sc.frame)
        h.set_samples(sc.samples)
        h.set_aov_count(3)
        h.submit_grids_device(g.ngrids, *[d[k].data_ptr() for k in (
            "cu", "cv", "nkeys", "flags", "pbase", "cbase", "tbase", "times", "P", "Ci", "Oi")], g.micropolygons)
        assert h.L.aqh_submit_aov_device(h.ctx, d["aov"].data_ptr()) == 0
        for _ in range(2):   # the second frame replays the first one's graph
            h.render()
            a = h.read_aov()
            b = oracle.render(sc)["aov"]
            assert np.array_equal(a.view(np.uint32), np.asarray(b, np.float32).reshape(a.shape).view(np.uint32))
        assert h.stats()["graphs_built"] == 1
    finally:
        h.close()


@pytest.mark.parametrize("fw", [1.0, 2.0, 4.0])
@pytest.mark.parametrize("gain,gamma", [(1.0, 2.2), (1.3, 1.8), (0.7, 0.45), (2.0, 20.0), (1.0, 0.1), (-1.0, 2.2),
                                        (1e-12, 2.0), (1e6, 2.4)])
def test_exposure_and_display(hider, fw, gain, gamma):
    """Exposure is the double power of the float channel rounded to float, the
    display the double rounding of the exposed channel plus dither: both from
    the same frame without exposure.  Gains and gammas inside and outside the
    range the float form of the power covers."""
    sc = _scene(61, 33, 3, 3, "gaussian", fw, 0, seed=7)
    rng = np.random.default_rng(1)
    sc.frame.q_dither = 0.5
    dither = sc.samples.dither = rng.random(61 * 33, dtype=np.float32)
    c = hider.render_scene(sc, samples=False)["channels"]
    sc.frame.gain, sc.frame.gamma = gain, gamma
    res = hider.render_scene(sc, samples=False)
    f32, f64 = np.float32, np.float64
    want = c.copy()
    with np.errstate(invalid="ignore", over="ignore"):
        lit = c[..., :3] if gain == 1.0 else c[..., :3] * f32(gain)
        want[..., :3] = np.power(lit.astype(f64), f64(f32(1.0) / f32(gamma))).astype(f32)
        assert np.array_equal(res["channels"].view(np.uint32)[~np.isnan(want)], want.view(np.uint32)[~np.isnan(want)])
        assert np.array_equal(np.isnan(res["channels"]), np.isnan(want))
        q = want[..., [0, 1, 2, 6]].astype(f64) * 255.0 + 0.5 * dither.reshape(33, 61, 1).astype(f64)
        q = np.where(np.isnan(q), 0.0, np.clip(np.floor(q - 0.5) + 1, 0, 255)).astype(np.uint8)
    assert np.array_equal(res["quantized"], q)
