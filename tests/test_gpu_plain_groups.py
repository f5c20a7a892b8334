"""The plain TFM / RCA kernels where terms are tested one by one: inner elements too
many for the leg table, around the groups of eight; outer elements all of whose
terms lie past the A-scan's end or before its start beside others that straddle
them. Images equal the oracle's bit for bit, out-of-bounds counts are the oracle's,
and so is the index table."""
import ctypes

import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run(method, n_out, n_in, K, delay, dtype, seed):
    from dream_b200 import _lib
    from dream_b200.beamformer import parse_method
    rng = np.random.default_rng(seed)
    nt, nr = (n_in, n_out) if method == "rca_rowtx" else (n_out, n_in)
    if method == "tfm":
        Gt, Gr = synth.linear_array(nt, 0.5), synth.linear_array(nr, 0.1)
        Ro = synth.grid_xz(11, 37, (-9.0, 7.0), (1.0, 21.0))
    else:
        Gt, Gr = synth.rca_arrays(nt, nr, 0.2)
        Ro = synth.grid_xyz(5, 3, 37, (-5.0, 6.0), (-4.0, 4.0), (1.0, 16.0))
    f = lambda a: np.asfortranarray(a, dtype=dtype)
    args = (f(rng.normal(size=(K, nt * nr))), f(Gt), f(Gr), f(Ro), dtype(0.04), f([[delay]]), dtype(1500.0), method)
    ref, _, oob_ref, idx = oracle.das(*args, "ignore", dtype, return_idx=True)
    L = _lib.load()
    plan = _lib.plan_create(parse_method(method), K, len(Ro), nt, nr,
                            _lib.PREC_F64 if dtype == np.float64 else _lib.PREC_F32, 0)
    t = [torch.from_numpy(np.ascontiguousarray(a.T)).cuda() for a in (args[0], args[3], args[1], args[2], args[5])]
    p = [ctypes.c_void_p(x.data_ptr()) for x in t]
    Im = torch.empty(len(Ro), dtype=t[0].dtype, device="cuda")
    oob = ctypes.c_int64(0)
    for hint in (0, 37):
        _lib.check(L.dream_das_set_grid_hint(plan.handle, hint))
        _lib.check(L.dream_das_run_device(plan.handle, *p[:4], 0.04, _lib.DELAY_SINGLE, p[4], 1500.0,
                                          ctypes.c_void_p(Im.data_ptr()), 1, ctypes.byref(oob), None))
        assert np.array_equal(Im.cpu().numpy(), ref.reshape(-1)), f"hint {hint}"
        assert oob.value == oob_ref
    table = torch.empty((nt * nr, len(Ro)), dtype=torch.int64, device="cuda")
    _lib.check(L.dream_das_indices_device(plan.handle, p[1], p[2], p[3], 0.04, _lib.DELAY_SINGLE, p[4], 1500.0,
                                          ctypes.c_void_p(table.data_ptr()), ctypes.byref(oob), None))
    assert np.array_equal(table.cpu().numpy(), np.where((idx >= 0) & (idx < K), idx, -1)) and oob.value == oob_ref
    return oob_ref, len(Ro) * nt * nr


@pytest.mark.parametrize("dtype,n_in", [(np.float64, 801), (np.float64, 807), (np.float64, 808), (np.float32, 1601),
                                        (np.float32, 1607)])
@pytest.mark.parametrize("K,delay", [(200, 0.1), (400, -3.0)])
def test_without_a_leg_table(n_in, dtype, K, delay):
    _run("tfm", 2, n_in, K, delay, dtype, n_in)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("method", ["tfm", "rca_coltx", "rca_rowtx"])
@pytest.mark.parametrize("K,delay", [(90, 0.0), (250, 0.0), (300, -12.0), (300, -40.0), (300, 1000.0)])
def test_elements_out_of_bounds(method, K, delay, dtype):
    out, all_terms = _run(method, 9, 19 if method == "tfm" else 13, K, delay, dtype, K)  # RCAs: edges inside Gr
    assert 0 < out < all_terms or abs(delay) >= 40.0
