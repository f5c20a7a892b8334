"""Image points and per-point delays that are not numbers, or infinite, in the
operator's adjoint: they have no sample in any A-scan (the gather counts their
terms as out of bounds), so the adjoint must leave them out and keep every other
point of their tile. Point sets with and without a grid hint, grids fine enough
for shared-memory windows and too coarse for them, whole chunks of eight inner
elements and partial ones.

Tolerance per sample against the FP64 adjoint at the oracle's indices: a tile of
windows rounds |x| to 2^-22 of the largest |x|, direct terms round once, and at
most m partial sums are added in FP32: m * (w max|x| 2^-21.5 + 2^-24 sum |w x|)."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DT, CP, K = 0.04, 1500.0, 1600
FORMS = ["fine_grid", "coarse_grid", "shuffled", "shuffled_rca"]


def _scene(form, n_in):
    if form == "shuffled_rca":
        Gt, Gr = synth.rca_arrays(7, n_in, 0.3) if n_in >= 7 else synth.rca_arrays(n_in, 7, 0.3)
        Ro, method = synth.grid_xyz(8, 6, 23, (-4.0, 4.0), (-4.0, 4.0), (3.0, 18.0)), "rca_coltx"
    else:
        Gt, Gr, method = synth.linear_array(7, 0.5), synth.linear_array(n_in, 0.4), "tfm"
        Ro = synth.grid_xz(30, 37, (-4.0, 4.0), (3.0, 9.0)) if form == "fine_grid" else \
            synth.grid_xz(24, 46, (-14.0, 14.0), (3.0, 24.0))
    if form.startswith("shuffled"):
        Ro = np.asfortranarray(Ro[np.random.default_rng(1).permutation(len(Ro))])
    return Gt, Gr, Ro, method


@pytest.mark.parametrize("n_in", [8, 17])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("what,bad", [("x", np.nan), ("z", np.nan), ("delay", np.nan), ("z", np.inf), ("delay", -np.inf)])
def test_points_without_a_sample(what, bad, form, n_in):
    from dream_b200.autograd import DASOperator
    Gt, Gr, Ro, method = _scene(form, n_in)
    No, ncol = len(Ro), len(Gt) * len(Gr)
    rng = np.random.default_rng(No + n_in)
    dl = rng.uniform(0.0, 0.4, (No, 1)) if what == "delay" else np.array([[0.1]])
    sick = np.array([0, 5, 300, 301, No - 1])
    if what == "delay":
        dl[sick] = bad
    else:
        Ro[sick, {"x": 0, "z": 2}[what]] = bad
    idx = oracle.das(np.zeros((K, ncol), order="F"), Gt, Gr, Ro, DT, dl, CP, method, "ignore", np.float64,
                     return_idx=True)[3]
    idx = np.where((idx >= 0) & (idx < K), idx, -1)
    assert (idx[:, sick] < 0).all() and (np.delete(idx, sick, 1) >= 0).all()
    x = rng.normal(size=No).astype(np.float32)
    w = rng.uniform(0.5, 1.5, ncol).astype(np.float32)
    op = DASOperator(Gt, Gr, Ro, DT, dl, CP, method, K)
    for weights in (None, w):
        wc = np.ones(ncol) if weights is None else w.astype(np.float64)
        ref, size, terms = (np.zeros((ncol, K)) for _ in range(3))
        for c in range(ncol):
            ok = idx[c] >= 0
            np.add.at(ref[c], idx[c][ok], wc[c] * x[ok].astype(np.float64))
            np.add.at(size[c], idx[c][ok], wc[c] * np.abs(x[ok]).astype(np.float64))
            np.add.at(terms[c], idx[c][ok], 1.0)
        Ya = op.adjoint(torch.from_numpy(x), None if weights is None else torch.from_numpy(w))
        Ya = Ya.t().cpu().numpy().astype(np.float64)
        tol = terms * (wc[:, None] * np.abs(x).max() * 2.0 ** -21.5 + size * 2.0 ** -24)
        wrong = ~(np.abs(Ya - ref) <= tol)
        assert not wrong.any(), f"{wrong.sum()} samples, worst {np.nanmax(np.abs(Ya - ref))}"
