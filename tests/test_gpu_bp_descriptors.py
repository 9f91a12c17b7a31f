"""More views on one BP stream than a launch descriptor holds (16): every phase
of a tick then takes two launches, with the data cost and the edge messages in
one launch (few windows) and in two (more than 6000). Every pair's result is
the one it has alone, bit for bit. Requires a GPU."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,W,H,post,fp16", [(17, 97, 43, 1, 0), (16, 64, 48, 2, 1), (18, 333, 271, 0, 1)])
def test_two_descriptors(n, W, H, post, fp16):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    from scenes import make_scene

    D = 24
    views = n * (2 if post == 2 else 1)
    assert 16 < views <= 32 and (views * -(-W * H // 256) > 6000) == (W > 300)
    scenes = [make_scene(W, H, D, 600 + i) for i in range(n)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dL, dR = [dev(s.left) for s in scenes], [dev(s.right) for s in scenes]
    out = [torch.zeros((H, W), dtype=torch.float32, device="cuda") for _ in scenes]
    arr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
    ctx = E.Context(0)
    try:
        prm = E.default_params(post=post, msg_fp16=fp16)
        single = [ctx.run_pair(s.left, s.right, D, prm) for s in scenes]
        E._check(E.lib().hbp_set_bp_streams(ctx.h, 1))
        E._check(E.lib().hbp_run_batch_d(ctx.h, n, arr(dL), arr(dR), W, H, D, C.byref(prm), arr(out), None))
        torch.cuda.synchronize()
        for a, b in zip(single, out):
            assert np.array_equal(a.view(np.uint32), b.cpu().numpy().view(np.uint32))
    finally:
        ctx.close()
