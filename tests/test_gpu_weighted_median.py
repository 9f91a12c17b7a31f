"""The weighted median's select path (both variants) against the oracle's sorts,
bit for bit, where it can go wrong: windows clipped on every side, all samples
on one plane, few planes (many ties at one z), different planes that meet at
one z, a flat image (running weights exactly at the half), weights of very
different size, planes with one z of either sign of zero. Requires a GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _planes(kind, W, H, rng):
    pl = np.zeros((H, W, 3), np.float32)
    if kind == "one":
        pl[:] = (0.02, -0.03, 7.5)
    elif kind == "few":
        pal = np.stack([rng.uniform(-0.05, 0.05, 5), rng.uniform(-0.05, 0.05, 5), rng.uniform(4, 40, 5)], -1)
        pl[:] = pal[rng.integers(0, 5, (-(-H // 6), -(-W // 6)))].repeat(6, 0)[:H].repeat(6, 1)[:, :W]
    elif kind == "meet":  # different planes, whole z values that many share
        pl[..., 0] = rng.integers(-1, 2, (H, W))
        pl[..., 1] = rng.integers(-1, 2, (H, W))
        pl[..., 2] = rng.integers(0, 3, (H, W))
    elif kind == "zero":
        pl[..., 2] = np.where(rng.random((H, W)) < 0.5, np.float32(-0.0), np.float32(0.0))
    else:
        pl[..., 0], pl[..., 1] = rng.uniform(-0.05, 0.05, (H, W)), rng.uniform(-0.05, 0.05, (H, W))
        pl[..., 2] = rng.uniform(0, 60, (H, W))
    return pl


@pytest.mark.parametrize("W,H", [(16, 16), (41, 41), (97, 43), (30, 64)])
@pytest.mark.parametrize("kind", ["one", "few", "meet", "zero", "random"])
@pytest.mark.parametrize("image", ["flat", "noise", "steps"])
def test_weighted_median_both_variants(W, H, kind, image):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    import pyoracle as O

    rng = np.random.default_rng([W, H, len(kind), len(image)])
    bgr = np.full((H, W, 3), 90, np.uint8)
    if image == "noise":
        bgr = np.clip(rng.normal(128, 12, (H, W, 3)), 0, 255).astype(np.uint8)
    elif image == "steps":
        bgr[:, : W // 2] = 250
        bgr[: H // 3] = (0, 128, 255)
    plane = _planes(kind, W, H, rng)
    fail = np.where(rng.random((H, W)) < 0.4, 255, 0).astype(np.uint8)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ctx = E.Context(0)
    try:
        wt = torch.zeros(766, device="cuda")
        ctx.patch_weights_d(wt)
        for median, want in ((ctx.weighted_median_d, O.weighted_median(bgr, fail, plane)),
                             (ctx.weighted_median_gpu_d, O.weighted_median_gpu(bgr, fail, plane, wt.cpu().numpy()))):
            pl, out = dev(plane), torch.zeros((H, W), device="cuda")
            median(dev(bgr), dev(fail), pl, out, W, H)
            torch.cuda.synchronize()
            got = pl.cpu().numpy()
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), int((got != want).any(-1).sum())
    finally:
        ctx.close()
