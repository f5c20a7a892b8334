"""Edges of the plain TFM / RCA tile kernel: inner counts around the gather
groups (16 and pairs of them) and the leg-table limits, grids that tiles do not
divide, A-scans that end inside the image, and non-finite legs. Images must
equal the oracle's bit for bit and the out-of-bounds status must match."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _frame(method, n_out, n_in, grid, K, dtype, seed, multi):
    rng = np.random.default_rng(seed)
    nt, nr = (n_in, n_out) if method == "rca_rowtx" else (n_out, n_in)
    if method == "tfm":
        Gt, Gr = synth.linear_array(nt, 0.5), synth.linear_array(nr, 0.4)
        Ro = synth.grid_xz(grid[0], grid[1], (-9.0, 7.0), (1.0, 21.0))
    else:
        Gt, Gr = synth.rca_arrays(nt, nr, 0.3)
        Ro = synth.grid_xyz(grid[0], 3, grid[1], (-5.0, 6.0), (-4.0, 4.0), (1.0, 16.0))
    f = lambda a: np.asfortranarray(a, dtype=dtype)
    delay = rng.uniform(-0.1, 0.5, (Ro.shape[0] if multi else 1, 1))
    return f(rng.normal(size=(K, nt * nr))), f(Gt), f(Gr), f(Ro), dtype(0.04), f(delay), dtype(1500.0)


def _compare(args, method, dtype, via):
    from dream_b200 import das, das_f
    mod = das if dtype == np.float64 else das_f
    t = (lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda() if isinstance(a, np.ndarray) else a) \
        if via == "device" else (lambda a: a)
    Im = mod.das(*(t(a) for a in args), method, "ignore", "cuda")
    Im = Im.cpu().numpy() if via == "device" else Im
    ref = oracle.das(*args, method, "ignore", dtype)[0]
    assert np.array_equal(Im, ref), f"{np.sum(Im != ref)} of {Im.size} pixels differ"


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n_in", [1, 15, 16, 17, 31, 32, 33, 48, 53, 64, 65, 97, 129, 300, 801])
def test_inner_counts(n_in, dtype):
    """One past each group and table limit; 801 FP64 legs exceed the table of one warp."""
    _compare(_frame("tfm", 3, n_in, (7, 41), 700, dtype, n_in, False), "tfm", dtype, "host")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("method", ["tfm", "rca_coltx", "rca_rowtx"])
@pytest.mark.parametrize("grid", [(1, 37), (3, 5), (9, 17), (33, 64), (40, 7)])
@pytest.mark.parametrize("K", [150, 900])
def test_ragged_grids_and_short_ascans(grid, method, K, dtype):
    _compare(_frame(method, 19, 21, grid, K, dtype, 5 + K, K == 150), method, dtype, "device")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_legs(bad, dtype):
    """A NaN or infinite element coordinate puts its terms, and only those, out of bounds."""
    args = _frame("tfm", 5, 20, (9, 33), 900, dtype, 3, False)
    args[2][7, 0] = bad
    _compare(args, "tfm", dtype, "host")
    args = _frame("tfm", 5, 20, (9, 33), 900, dtype, 4, False)
    args[1][2, 1] = bad
    _compare(args, "tfm", dtype, "host")
