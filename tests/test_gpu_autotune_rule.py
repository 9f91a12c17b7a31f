"""The stream counts that the autotuner tries on a default context: a class with
one count to try takes the fixed rule's (the two views of a small pair run on
one stream), larger classes try the rule's count too, and none tries more than
four. Requires a GPU."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,W,H,post,tried", [
    (1, 96, 64, 2, [1]),      # two views, 48 windows
    (1, 720, 496, 2, [2]),    # two views, 2790
    (3, 96, 64, 1, [1]),      # 72
    (3, 960, 724, 0, [2, 3]),   # 8145
    (4, 800, 655, 0, [2, 3, 4]),  # 8188
    (6, 96, 64, 1, [2, 4])])
def test_counts_tried(n, W, H, post, tried):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    from scenes import make_scene

    D = 32
    scenes = [make_scene(W, H, D, 500 + i) for i in range(n)]
    ctx = E.Context(0)
    try:
        prm = E.default_params(post=post)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        dL, dR = [dev(s.left) for s in scenes], [dev(s.right) for s in scenes]
        out = [torch.zeros((H, W), dtype=torch.float32, device="cuda") for _ in scenes]
        arr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
        for _ in range(len(tried)):
            E._check(E.lib().hbp_run_batch_d(ctx.h, n, arr(dL), arr(dR), W, H, D, C.byref(prm), arr(out), None))
        rows = (C.c_double * 90)()
        k = E.lib().hbp_autotune_table(ctx.h, rows, 10)
        table = np.array(rows[:9 * k]).reshape(k, 9)
        assert np.all(table[:, 5] == n * (2 if post == 2 else 1))
        assert table[:, 6].astype(int).tolist() == tried
    finally:
        ctx.close()
