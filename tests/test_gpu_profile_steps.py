"""The breakdown (profile mode 3) of a single pair shows the launches that its
steps run: data cost and edge messages together (kind 9), apart only on every
16th BP tick, and the pair's result is the unprofiled one. Requires a GPU."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, D = 160, 120, 48


def test_breakdown_of_a_single_pair():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hbp_b200 as E
    from scenes import make_scene

    s = make_scene(W, H, D, 91)
    ctx = E.Context(0)
    try:
        prm = E.default_params(post=1)
        plain = ctx.run_pair(s.left, s.right, D, prm)
        E._check(E.lib().hbp_profile_enable(ctx.h, 3))
        profiled = ctx.run_pair(s.left, s.right, D, prm)
        cells = 10 * 32
        ms, timed, every = (C.c_double * cells)(), (C.c_long * cells)(), (C.c_long * cells)()
        E._check(E.lib().hbp_profile_breakdown(ctx.h, ms, timed, every))
        E._check(E.lib().hbp_profile_enable(ctx.h, 0))
        ms, timed, every = (np.array(v[:]).reshape(10, 32).sum(1) for v in (ms, timed, every))
        assert np.array_equal(plain.view(np.uint32), profiled.view(np.uint32))
        assert np.all(every[1:3] == 0)
        assert timed[9] > 0 and ms[9] > 0
        steps, levels = every[4] + every[9], every[6]
        assert every[0] == steps + levels  # a node phase per step, and a level's last select
        assert every[4] == every[5] and 0 < every[4] <= (steps + 2 * levels + 1) // 16 + 1
    finally:
        ctx.close()
