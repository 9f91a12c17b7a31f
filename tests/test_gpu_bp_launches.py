"""The BP step as one launch and as two: a pair alone runs its data cost and
edge messages in one launch (eight lanes per edge at coarse levels, four below),
a batch of more than 6000 windows of 256 pixels in separate ones (a thread or
four lanes per edge). Neither changes a bit of any pair's result. Requires a
GPU."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, D, NP = 451, 373, 48, 10  # 658 windows a view, the last one partial


@pytest.mark.parametrize("streams,fp16", [(0, 0), (1, 1)])
def test_batch_of_many_windows_equals_single_pairs(streams, fp16):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    from scenes import make_scene

    assert NP * -(-W * H // 256) > 6000
    scenes = [make_scene(W, H, D, 300 + i) for i in range(NP)]
    ctx = E.Context(0)
    try:
        prm = E.default_params(post=0, msg_fp16=fp16)
        single = [ctx.run_pair(s.left, s.right, D, prm) for s in scenes]
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        dL = [dev(s.left) for s in scenes]
        dR = [dev(s.right) for s in scenes]
        out = [torch.zeros((H, W), dtype=torch.float32, device="cuda") for _ in scenes]
        arr = lambda ts: (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])
        E._check(E.lib().hbp_set_autotune(ctx.h, 0))
        E._check(E.lib().hbp_set_bp_streams(ctx.h, streams))
        E._check(E.lib().hbp_run_batch_d(ctx.h, NP, arr(dL), arr(dR), W, H, D, C.byref(prm), arr(out), None))
        torch.cuda.synchronize()
        for a, b in zip(single, out):
            assert np.array_equal(a.view(np.uint32), b.cpu().numpy().view(np.uint32))
    finally:
        ctx.close()
