"""Tiles of the operator's adjoint: square or long by the grid's spacing, on frames
whose last tiles are partly filled in either direction; points without lines (none
found, or one point per line), on frames below and above a tile per SM; few outer
elements. Whole-number images make the adjoint exact: a point taken twice, never or
at another's place shows. The automatic tile has to keep up with a caller's: within
one and a half times the better of two fixed tiles, and points in rows along x
within five times the same points in lines (one point per line would fill a
sixteenth of a tile's lanes)."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DT, CP, K = 0.04, 1500.0, 1300


def _points(lines, depth, form):
    x_half, z_hi = {"fine_depth": (15.0, 8.0), "coarse_depth": (4.0, 24.0)}.get(form, (9.0, 16.0))
    Ro = synth.grid_xz(lines, depth, (-x_half, x_half), (2.0, z_hi))
    if form == "rows":
        Ro = Ro.reshape(lines, depth, 3).transpose(1, 0, 2).reshape(-1, 3)
    if form == "cloud":
        Ro = Ro[np.random.default_rng(0).permutation(len(Ro))]
    return np.asfortranarray(Ro)


@pytest.mark.parametrize("form", ["fine_depth", "coarse_depth", "rows", "cloud"])
@pytest.mark.parametrize("lines,depth", [(1187, 33), (1200, 40), (201, 197), (224, 176), (1300, 31), (19000, 2), (37, 41),
                                         (32, 64)])
@pytest.mark.parametrize("n_out,n_in", [(3, 5), (1, 17)])
def test_every_point_once(n_out, n_in, lines, depth, form):
    from dream_b200.autograd import DASOperator
    Gt, Gr, Ro = synth.linear_array(n_out, 0.5), synth.linear_array(n_in, 0.4), _points(lines, depth, form)
    No, ncol = len(Ro), n_out * n_in
    dl = np.array([[0.1]])
    idx = oracle.das(np.zeros((K, ncol), order="F"), Gt, Gr, Ro, DT, dl, CP, "tfm", "ignore", np.float64,
                     return_idx=True)[3]
    rng = np.random.default_rng(No)
    x = rng.integers(-5, 6, No).astype(np.float32)
    w = rng.integers(1, 4, ncol).astype(np.float32)
    op = DASOperator(Gt, Gr, Ro, DT, dl, CP, "tfm", K)
    for weights in (None, w):
        Ya = op.adjoint(torch.from_numpy(x), None if weights is None else torch.from_numpy(w)).t().cpu().numpy()
        for c in range(ncol):
            ok = (idx[c] >= 0) & (idx[c] < K)
            ref = np.bincount(idx[c][ok], weights=x[ok].astype(np.float64), minlength=K)
            assert np.array_equal(Ya[c], ref * (1.0 if weights is None else w[c])), f"A-scan {c}"


def _ms(op, x):
    op.adjoint(x)
    best = np.inf
    for _ in range(7):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(200000)  # the launches are queued before the first one starts
        e0.record()
        op.adjoint(x)
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


@pytest.mark.parametrize("n_out,n_in,lines,depth,half,z_hi", [(64, 64, 1024, 40, 15.0, 27.0), (37, 53, 301, 203, 20.0, 37.0),
                                                              (2, 801, 48, 64, 15.0, 27.0), (8, 300, 48, 64, 15.0, 27.0)])
def test_automatic_tile_keeps_up(n_out, n_in, lines, depth, half, z_hi):
    from dream_b200 import _lib
    from dream_b200.autograd import DASOperator
    Gt, Gr = synth.linear_array(n_out, 0.5), synth.linear_array(n_in, 0.5)
    op = DASOperator(Gt, Gr, synth.grid_xz(lines, depth, (-half, half), (2.0, z_hi)), DT, np.zeros((1, 1)), CP, "tfm", 1777)
    x = torch.randn(op.No, device="cuda")
    auto = _ms(op, x)
    fixed = []
    for tile in ((8, 32), (16, 16)):
        _lib.check(_lib.load().dream_das_set_tile(op.plan.handle, *tile))
        fixed.append(_ms(op, x))
    assert auto <= 1.5 * min(fixed), (auto, fixed)


def test_rows_along_x():
    from dream_b200.autograd import DASOperator
    G = synth.linear_array(24, 0.5)
    t = {}
    for form in ("lines", "rows"):
        op = DASOperator(G, G, _points(256, 256, form), DT, np.zeros((1, 1)), CP, "tfm", K)
        t[form] = _ms(op, torch.randn(op.No, device="cuda"))
    assert t["rows"] <= 5.0 * t["lines"], t
