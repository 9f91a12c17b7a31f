"""The weighted median where planes are not finite at the pixel (a plane fitted
to three points on a line is): +infinity, -infinity, NaN, the largest float and
one that overflows inside the image, as few or most of the samples, against
the oracle's sorts bit for bit. The CPU variant orders a NaN as +infinity (the
reference's std::sort has no order for it), so its oracle gets a plane at
+infinity in the NaN's place. Requires a GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ODD = {"inf": (0, 0, np.inf), "-inf": (0, 0, -np.inf), "nan": (0, 0, np.nan), "max": (0, 0, np.finfo(np.float32).max),
       "over": (0, 3e38, 3e38)}


@pytest.mark.parametrize("W,H", [(16, 16), (41, 41), (97, 43)])
@pytest.mark.parametrize("share", [0.01, 0.3, 0.8, 1.0])
@pytest.mark.parametrize("odd", ["inf", "-inf", "nan", "nan,-inf,max,over"])
def test_planes_that_are_not_finite(W, H, share, odd):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    import pyoracle as O

    rng = np.random.default_rng([W, H, int(100 * share), len(odd)])
    bgr = np.clip(rng.normal(128, 12, (H, W, 3)), 0, 255).astype(np.uint8)
    plane = np.stack([rng.uniform(-0.05, 0.05, (H, W)), rng.uniform(-0.05, 0.05, (H, W)), rng.uniform(0, 60, (H, W))],
                     -1).astype(np.float32)
    palette = np.array([ODD[k] for k in odd.split(",")], np.float32)
    hit = rng.random((H, W)) < share
    plane[hit] = palette[rng.integers(0, len(palette), int(hit.sum()))]
    fail = np.where(rng.random((H, W)) < 0.4, 255, 0).astype(np.uint8)

    nan = np.isnan(plane[..., 2])
    as_inf = plane.copy()
    as_inf[nan] = (0, 0, np.inf)
    want = O.weighted_median(bgr, fail, as_inf)
    if nan.any():  # no plane of its own is (0, 0, +infinity) then
        assert "inf" not in odd.split(",")
        want[np.isposinf(want[..., 2])] = ODD["nan"]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ctx = E.Context(0)
    try:
        wt = torch.zeros(766, device="cuda")
        ctx.patch_weights_d(wt)
        with np.errstate(invalid="ignore"):
            want_gpu = O.weighted_median_gpu(bgr, fail, plane, wt.cpu().numpy())
        for median, ref in ((ctx.weighted_median_d, want), (ctx.weighted_median_gpu_d, want_gpu)):
            pl, out = dev(plane), torch.zeros((H, W), device="cuda")
            median(dev(bgr), dev(fail), pl, out, W, H)
            torch.cuda.synchronize()
            got = pl.cpu().numpy()
            assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), int((got.view(np.uint32) != ref.view(np.uint32)).any(-1).sum())
    finally:
        ctx.close()
