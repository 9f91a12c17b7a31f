"""The Census volumes and WTA of both views at the edges of the Hamming kernel's
geometry (four pixels and four disparities a lane, strips of 64 columns, tiles
of 8 x 4), with volumes at every byte alignment, against the oracle bit for
bit. Requires a GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D", [(16, 16, 2), (17, 18, 3), (65, 16, 5), (64, 17, 63), (127, 21, 64), (200, 16, 130),
                                   (1100, 16, 1024)])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_census_volumes(W, H, D, shift):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    import pyoracle as O

    rng = np.random.default_rng([W, H, D])
    # few colours: equal costs, so that the first of them has to win
    L, R = (rng.integers(0, 4, (H, W, 3)).astype(np.uint8) * 60 for _ in range(2))
    left = O.cost_stage(L, R, D)
    want = [(left["vol"], left["wta"]), O.cost_to_right(left["vol"], W, H, D)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    n = E.volume_bytes(W, H, D)
    bufs = [torch.full((n + 8,), 77, dtype=torch.uint8, device="cuda") for _ in range(2)]
    vols = [b[shift:shift + n] for b in bufs]
    wta = [torch.zeros((H, W), device="cuda") for _ in range(2)]
    cen = [torch.zeros((H, W), dtype=torch.int32, device="cuda") for _ in range(2)]
    ctx = E.Context(0)
    try:
        ctx.cost_census_d(dev(L), dev(R), W, H, D, *cen, vols[0], wta[0], vols[1], wta[1])
        torch.cuda.synchronize()
        for k in range(2):
            vol, win = want[k]
            assert np.array_equal(E.volume_to_dhw(vols[k].cpu().numpy(), W, H, D).reshape(D, H, W), vol.reshape(D, H, W))
            assert (bufs[k][:shift] == 77).all() and (bufs[k][shift + n:] == 77).all()
            assert np.array_equal(wta[k].cpu().numpy(), win.reshape(H, W))
    finally:
        ctx.close()
