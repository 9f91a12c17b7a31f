"""CRTrees and the segmentation pyramid where their kernels change form: the
one-block and the grid version of CRTrees (10000 nodes), the one-block, the
few-tiles and the general radix sort (8192 and 131072 items), the one-tile scan
(2048). Labels and every ISP array equal the oracle's. Requires a GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    ctx = E.Context(0)
    yield E, ctx, torch
    ctx.close()


@pytest.mark.parametrize("N", [1, 2, 33, 1023, 1025, 9999, 10000, 10001, 30000])
@pytest.mark.parametrize("kind", ["near", "any", "star"])
def test_crtrees_sizes(eng, N, kind):
    import pyoracle as O
    E, ctx, torch = eng
    rng = np.random.default_rng([N, len(kind)])
    i = np.arange(N)
    if kind == "near":
        nn = np.clip(i + rng.integers(-3, 4, N), 0, N - 1)
    elif kind == "any":
        nn = rng.integers(0, N, N)
    else:
        nn = rng.integers(0, max(1, N // 50), N)
    nn = np.where(nn == i, (i + 1) % N, nn).astype(np.int32)  # a node's successor is another node
    want, n = O.crtrees(nn)
    out = torch.zeros(N, dtype=torch.int32, device="cuda")
    got = ctx.crtrees_d(torch.from_numpy(nn).cuda(), N, out)
    assert got == n and np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("W,H", [(17, 16), (32, 64), (91, 90), (64, 128), (127, 65), (256, 129), (180, 183)])
def test_pyramid_sizes(eng, W, H):
    import pyoracle as O
    E, ctx, torch = eng
    rng = np.random.default_rng([W, H])
    img = np.clip(rng.normal(120, 25, (H, W, 3)), 0, 255).astype(np.uint8)
    img[: H // 2, W // 3:] //= 2
    ctx.segment_d(torch.from_numpy(img).cuda(), W, H)
    g, o = ctx.pyramid(), O.segment(O.lab(img))
    assert np.array_equal(g["level_sizes"], o["level_sizes"])
    for k in ("clus", "bd", "bdl"):
        assert np.array_equal(g[k], o[k]), k
    assert np.array_equal(g["mean"].view(np.uint32), np.asarray(o["mean"], np.float32).reshape(-1).view(np.uint32))
