"""Tiles of neighbouring lines of an RCA volume: rows of lines around the bands
of four, a last band that is partly filled, rows that share x or y, more lines
than the search looks at, points that end inside a row, planes. Whole-number
A-scans and images whose sums stay below 2^24: every result is exact, so a point
taken twice or never, or at another's place, shows."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

GRIDS = [(4, 4, 9), (2, 4, 33), (3, 3, 8), (5, 2, 17), (1, 9, 12), (9, 1, 12), (7, 13, 20), (8, 16, 32), (13, 6, 31),
         (2, 1100, 3), (3, 1024, 2), (4, 67, 5)]  # lines along x and along y, points per line


def _frame(method, grid, form, dtype=np.float64):
    n = 33  # 1089 terms per point: the search starts at 1024
    rng = np.random.default_rng(grid[0] * 1000 + grid[1])
    Gt, Gr = synth.rca_arrays(n, n, 0.3)
    Ro = synth.grid_xyz(*grid, (-4.0, 4.5), (-3.5, 4.0), (1.0, 14.0))
    if form == "swapped":  # rows share y
        Ro = Ro[:, [1, 0, 2]]
    elif form == "cut":  # the last row is not whole
        Ro = Ro[:-grid[2]]
    f = lambda a: np.asfortranarray(a, dtype=dtype)
    return f(rng.integers(-20, 21, size=(700, n * n))), f(Gt), f(Gr), f(Ro), dtype(0.04), f([[0.1]]), dtype(1500.0), method


@pytest.mark.parametrize("form", ["grid", "swapped", "cut"])
@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("method", ["rca_coltx", "rca_rowtx"])
def test_images_and_adjoint(method, grid, form):
    from dream_b200 import das, das_f
    from dream_b200.autograd import DASOperator
    from dream_b200.beamformer import das_mixed
    for dtype, mod in ((np.float64, das), (np.float32, das_f)):
        args = _frame(method, grid, form, dtype)
        assert np.array_equal(mod.das(*args, "ignore", "cuda"), oracle.das(*args, "ignore", dtype)[0])
    args = _frame(method, grid, form)
    ref = oracle.das(*args, "ignore", np.float64)[0]
    Y = torch.from_numpy(args[0].astype(np.float32)).cuda()
    for storage in ("f32", "bf16"):
        Im = das_mixed(Y, *args[1:], "ignore", "cuda", storage)
        assert np.array_equal(Im.cpu().numpy().astype(np.float64), ref)
    op = DASOperator(*args[1:4], float(args[4]), args[5], float(args[6]), method, 700)
    x = torch.from_numpy(np.random.default_rng(3).integers(-5, 6, size=op.No).astype(np.float32)).cuda()
    lhs = float(torch.from_numpy(ref.reshape(-1)).cuda() @ x.double())
    assert lhs == float((Y.double() * op.adjoint(x).double()).sum())
