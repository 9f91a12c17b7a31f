"""The BP streams that a batch takes by itself (the autotuner off): one below
1700 data-cost windows of 256 pixels in flight, two below 8000, three above,
however many views they belong to. Every stream launches its own views' steps,
so a batch's launches tell its streams. Requires a GPU."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,W,H,streams", [(3, 96, 64, 1), (4, 450, 375, 2), (4, 800, 655, 3)])
def test_streams_follow_the_windows(n, W, H, streams):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    from scenes import make_scene

    windows = n * -(-W * H // 256)
    assert streams == (1 if windows < 1700 else 2 if windows < 8000 else 3)
    D = 32
    scenes = [make_scene(W, H, D, 400 + i) for i in range(n)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dL, dR = [dev(s.left) for s in scenes], [dev(s.right) for s in scenes]
    out = [torch.zeros((H, W), dtype=torch.float32, device="cuda") for _ in scenes]
    arr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
    ctx = E.Context(0)
    try:
        prm = E.default_params(post=0)
        E._check(E.lib().hbp_set_autotune(ctx.h, 0))

        def launches(fixed):
            E._check(E.lib().hbp_set_bp_streams(ctx.h, fixed))
            before = E.lib().hbp_launch_count()
            E._check(E.lib().hbp_run_batch_d(ctx.h, n, arr(dL), arr(dR), W, H, D, C.byref(prm), arr(out), None))
            return E.lib().hbp_launch_count() - before

        by_count = {s: launches(s) for s in (1, 2, 3)}
        assert by_count[1] < by_count[2] < by_count[3]
        assert launches(0) == by_count[streams]
    finally:
        ctx.close()
