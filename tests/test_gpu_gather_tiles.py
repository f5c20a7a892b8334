"""Edges of the FP32/BF16-storage gather: outer counts around its groups of 4
and 8 and its blocks of legs, inner counts around its chunks of 8, A-scans that
end (or start, with negative delays) inside the image, grids that tiles do not
divide, weights, inner shards and non-finite legs.

A sample index that is off by one changes the image by a white-noise sample, so
the tolerance is that of the sums alone: a term passes at most 9 FP32 roundings
(product, 5 tree or chain additions, two partial sums, the compensated sum's
result), so |error| <= 9 * 2^-24 * sum |w y| < 6e-7 * sum |w y|."""
import ctypes

import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _frame(method, n_out, n_in, grid, K, seed, delay=0.1):
    rng = np.random.default_rng(seed)
    nt, nr = (n_in, n_out) if method == "rca_rowtx" else (n_out, n_in)
    if method == "tfm":
        Gt, Gr = synth.linear_array(nt, 0.5), synth.linear_array(nr, 0.4)
        Ro = synth.grid_xz(grid[0], grid[1], (-9.0, 7.0), (1.0, 21.0))
    else:
        Gt, Gr = synth.rca_arrays(nt, nr, 0.3)
        Ro = synth.grid_xyz(grid[0], 3, grid[1], (-5.0, 6.0), (-4.0, 4.0), (1.0, 16.0))
    Y = np.asfortranarray(rng.normal(size=(K, nt * nr)).astype(np.float32).astype(np.float64))
    return Y, Gt, Gr, Ro, 0.04, np.array([[delay]]), 1500.0


def _check(args, method, storage="f32", weights=None):
    from dream_b200 import beamformer
    Y = args[0]
    if storage == "bf16":
        Y = torch.from_numpy(Y).to(torch.bfloat16).double().numpy()
    Yw = np.asfortranarray(Y if weights is None else Y * weights)
    ref, _, oob = oracle.das(Yw, *args[1:], method, "ignore", np.float64)[:3]
    tol = 6e-7 * oracle.das(np.abs(Yw), *args[1:], method, "ignore", np.float64)[0]
    seen = []
    report, beamformer._report = beamformer._report, lambda st, name="DAS": seen.append(st)
    try:
        Im = beamformer.das_mixed(torch.from_numpy(args[0].astype(np.float32)).cuda(), *args[1:], method, "ignore",
                                  "cuda", storage, weights=None if weights is None else weights.astype(np.float32))
    finally:
        beamformer._report = report
    Im = Im.cpu().numpy().astype(np.float64)
    bad = np.abs(Im - ref) > tol + 1e-30
    assert not bad.any(), f"{bad.sum()} of {bad.size} points, worst {np.abs(Im - ref).max()}"
    assert (seen[0] != 0) == (oob > 0)


@pytest.mark.parametrize("n_out", [1, 3, 4, 5, 8, 11, 12, 52, 53, 63, 64, 65, 105])
@pytest.mark.parametrize("weighted", [False, True])
def test_outer_counts(n_out, weighted):
    w = np.random.default_rng(n_out).uniform(0.5, 1.5, n_out * 9).astype(np.float32).astype(np.float64) if weighted else None
    _check(_frame("tfm", n_out, 9, (7, 41), 900, n_out), "tfm", weights=w)


@pytest.mark.parametrize("n_in", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_inner_counts(n_in, storage):
    _check(_frame("tfm", 13, n_in, (9, 33), 900, n_in), "tfm", storage)


@pytest.mark.parametrize("method", ["tfm", "rca_coltx", "rca_rowtx"])
@pytest.mark.parametrize("grid", [(1, 37), (3, 5), (9, 17), (33, 40)])
@pytest.mark.parametrize("K,delay", [(150, 0.1), (400, -2.0), (900, 0.3)])
def test_ragged_grids_and_short_ascans(grid, method, K, delay):
    _check(_frame(method, 19, 21, grid, K, 5 + K, delay), method)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_legs(bad):
    args = _frame("tfm", 9, 20, (9, 33), 900, 3)
    args[2][7, 0] = bad
    _check(args, "tfm")
    args = _frame("tfm", 9, 20, (9, 33), 900, 4)
    args[1][2, 1] = bad
    _check(args, "tfm")


def test_inner_shard_and_out_of_bounds_count():
    """A shard's partial image and its out-of-bounds count, both sides of an A-scan's end."""
    from dream_b200 import _lib
    args = _frame("rca_coltx", 10, 21, (9, 17), 200, 8)
    Y, Gt, Gr, Ro, dt, dl, cp = args
    lo, hi = 5, 18
    cols = (np.arange(10)[:, None] * 21 + np.arange(lo, hi)).reshape(-1)
    mask = np.zeros(210)
    mask[cols] = 1.0
    ref = oracle.das(np.asfortranarray(Y * mask), *args[1:], "rca_coltx", "ignore", np.float64)[0]
    idx = oracle.das(Y, *args[1:], "rca_coltx", "ignore", np.float64, return_idx=True)[3]
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).to("cuda", d)
    Yd, f64 = t(Y[:, cols], torch.float32), [t(a, torch.float64) for a in (Ro, Gt, Gr, dl)]
    Im = torch.empty(Ro.shape[0], device="cuda")
    oob = torch.zeros(1, dtype=torch.int64, device="cuda")
    p = lambda x: ctypes.c_void_p(x.data_ptr())
    plan = _lib.plan_create(_lib.RCA_COLTX, 200, Ro.shape[0], 10, 21, _lib.PREC_F32_STORE, 0)
    L = _lib.load()
    _lib.check(L.dream_das_set_inner_shard(plan.handle, lo, hi))
    _lib.check(L.dream_das_run_device_async(plan.handle, p(Yd), p(f64[0]), p(f64[1]), p(f64[2]), dt, 0, p(f64[3]), cp,
                                            p(Im), p(oob), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    tol = 6e-7 * oracle.das(np.asfortranarray(np.abs(Y) * mask), *args[1:], "rca_coltx", "ignore", np.float64)[0]
    assert np.all(np.abs(Im.cpu().numpy() - ref) <= tol + 1e-30)
    assert int(oob.item()) == int((idx[cols] == oracle.OOB_MISS).sum()) > 0
