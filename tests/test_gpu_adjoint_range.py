"""Images with NaN, infinite or extreme values in the operator's adjoint. A NaN
or infinite value reaches the samples of its own terms and no others; images of
any magnitude keep the accuracy of images around one.

Tolerance per sample against the FP64 adjoint at the oracle's indices: a tile of
windows rounds |x| to 2^-22 of the largest finite |x|, direct terms round once,
at most m partial sums are added in FP32, and an atomic FP32 addition in global
memory takes subnormal operands and results as zero (2^-126 each):
m * (w max|x| 2^-21.5 + 2^-23 sum |w x| + 2^-125)."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

K, DT, CP = 900, 0.04, 1500.0


def _check(form, x_of, weighted):
    from dream_b200.autograd import DASOperator
    if form == "rca":
        Gt, Gr = synth.rca_arrays(9, 6, 0.3)
        Ro, method = synth.grid_xyz(9, 7, 40, (-3.0, 3.0), (-3.0, 3.0), (2.0, 12.0)), "rca_rowtx"
    else:
        Gt, Gr, method = synth.linear_array(6, 0.5), synth.linear_array(9, 0.4), "tfm"
        Ro = synth.grid_xz(33, 40, (-5.0, 5.0), (2.0, 12.0))
        if form == "shuffled":
            Ro = np.asfortranarray(Ro[np.random.default_rng(1).permutation(len(Ro))])
    ncol, No = len(Gt) * len(Gr), len(Ro)
    dl = np.array([[0.1]])
    idx = oracle.das(np.zeros((K, ncol), order="F"), Gt, Gr, Ro, DT, dl, CP, method, "ignore", np.float64,
                     return_idx=True)[3]
    idx = np.where((idx >= 0) & (idx < K), idx, -1)
    rng = np.random.default_rng(No)
    x = x_of(rng, No).astype(np.float32)
    w = rng.uniform(0.5, 1.5, ncol).astype(np.float32) if weighted else np.ones(ncol, np.float32)
    top = np.abs(x[np.isfinite(x)]).max(initial=0.0).astype(np.float64)
    ref, size, terms = (np.zeros((ncol, K)) for _ in range(3))
    for c in range(ncol):
        ok = idx[c] >= 0
        v = float(w[c]) * x[ok].astype(np.float64)
        np.add.at(ref[c], idx[c][ok], v)
        np.add.at(size[c], idx[c][ok], np.abs(v))
        np.add.at(terms[c], idx[c][ok], 1.0)
    op = DASOperator(Gt, Gr, Ro, DT, dl, CP, method, K)
    Ya = op.adjoint(torch.from_numpy(x), torch.from_numpy(w) if weighted else None).t().cpu().numpy().astype(np.float64)
    fin = np.isfinite(ref)
    assert np.array_equal(Ya[~fin], ref[~fin], equal_nan=True)
    tol = terms * (w[:, None] * top * 2.0 ** -21.5 + size * 2.0 ** -23 + 2.0 ** -125)
    wrong = ~(np.abs(Ya[fin] - ref[fin]) <= tol[fin])
    assert not wrong.any(), f"{wrong.sum()} of {fin.sum()} samples"


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("form", ["tfm", "rca", "shuffled"])
@pytest.mark.parametrize("scale", [1e36, 1e30, 1e-10, 1e-30, 2.0 ** -103, 2.0 ** -105, 2.0 ** -107, 1e-33, 1e-36, 1e-38])
def test_magnitudes(scale, form, weighted):
    _check(form, lambda rng, n: scale * rng.normal(size=n), weighted)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("form", ["tfm", "rca", "shuffled"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["one", "tile", "all"])
def test_non_finite_values(where, bad, form, weighted):
    def x_of(rng, n):
        x = rng.normal(size=n)
        x[{"one": slice(137, 138), "tile": slice(0, 400), "all": slice(None)}[where]] = bad
        return x
    _check(form, x_of, weighted)
