"""Batches of different shared-memory needs alive at the same time: a batch of
small frames made after one of large frames, and an allocation-free call between
them, must leave the older batch able to run. Whole-number A-scans whose sums
stay below 2^24: every image is exact."""
import ctypes

import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _frame(n, storage):
    from dream_b200.batch import make_frame
    rng = np.random.default_rng(n)
    G = synth.linear_array(n, 0.4)
    Ro = synth.grid_xz(9, 41, (-6.0, 6.0), (1.0, 18.0))
    Y = np.asfortranarray(rng.integers(-20, 21, size=(900, n * n)).astype(np.float64))
    f = make_frame(Y, G, G, Ro, 0.04, np.array([[0.1]]), 1500.0, "tfm", storage=storage)
    ref = oracle.das(Y, G, G, Ro, 0.04, np.array([[0.1]]), 1500.0, "tfm", "ignore", np.float64)[0]
    return f, ref


def _holds(f, ref):
    torch.cuda.synchronize()
    return np.array_equal(f.Im.cpu().numpy().astype(np.float64).ravel(), ref.ravel())


@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_small_batch_after_large(storage):
    from dream_b200 import _lib
    from dream_b200.batch import DASBatch
    large, ref_l = _frame(104, storage)  # legs of 52 outer elements at a time: more than 48 KB
    small, ref_s = _frame(8, storage)
    a = DASBatch([large], storage=storage, autotune=False)
    a.run()
    assert _holds(large, ref_l)
    b = DASBatch([small], storage=storage, autotune=False)
    for f in (large, small):
        f.Im.zero_()
    a.run()
    b.run()
    assert _holds(large, ref_l) and _holds(small, ref_s)
    small.Im.zero_()
    large.Im.zero_()
    _lib.check(_lib.load().dream_das_batch_run_noalloc(
        ctypes.cast(b._arr, ctypes.c_void_p), 1, _lib.PREC_BF16_STORE if storage == "bf16" else _lib.PREC_F32_STORE,
        torch.cuda.current_device(), None, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    a.run()
    assert _holds(large, ref_l) and _holds(small, ref_s)
