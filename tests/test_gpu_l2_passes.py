"""Passes over inner elements under an explicit L2 budget: the A-scans of a pass
fit in it (down to one pass's least width, 8 inner elements), and the image is
that of one pass up to the FP32 rounding of the passes' order. Whole-number
A-scans whose sums stay below 2^24 make it exact."""
import ctypes

import numpy as np
import pytest

from dream_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_in,cols,passes", [(100, 63, 2), (100, 50, 3), (100, 48, 3), (100, 99, 2), (100, 100, 1),
                                              (40, 16, 3), (40, 23, 3), (40, 8, 5), (40, 3, 5), (17, 16, 2), (7, 3, 1)])
def test_pass_widths(n_in, cols, passes):
    """cols: A-scan columns of the inner loop that the budget holds, per outer element."""
    from dream_b200 import _lib
    L = _lib.load()
    n_out, K = 5, 700
    rng = np.random.default_rng(n_in + cols)
    Gt, Gr = synth.linear_array(n_out, 0.5), synth.linear_array(n_in, 0.2)
    Ro = synth.grid_xz(7, 30, (-5.0, 5.0), (1.0, 14.0))
    f = lambda a, t: torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).to("cuda", t)
    Y = f(rng.integers(-20, 21, size=(K, n_out * n_in)), torch.float32)
    geo = [f(a, torch.float64) for a in (Ro, Gt, Gr, np.array([[0.1]]))]
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def image(budget):
        plan = _lib.plan_create(_lib.TFM, K, len(Ro), n_out, n_in, _lib.PREC_F32_STORE, 0)
        _lib.check(L.dream_das_set_grid_hint(plan.handle, 30))
        _lib.check(L.dream_das_set_l2_block(plan.handle, budget))
        Im = torch.empty(len(Ro), device="cuda")
        oob = torch.zeros(1, dtype=torch.int64, device="cuda")
        _lib.check(L.dream_das_run_device_async(plan.handle, p(Y), p(geo[0]), p(geo[1]), p(geo[2]), 0.04,
                                                _lib.DELAY_SINGLE, p(geo[3]), 1500.0, p(Im), p(oob), None))
        torch.cuda.synchronize()
        return Im, int(oob.item()), L.dream_das_plan_launch_count(plan.handle)

    one, oob1, n1 = image(-1)
    blk, oob, n = image(cols * n_out * K * 4)
    assert torch.equal(one, blk) and oob == oob1
    assert n == passes * n1
