"""Weights that are not finite, or overflow with the image's values, in the
operator's adjoint: only the samples that a term falls on may become non-finite,
whatever the A-scan length's alignment, and no other A-scan changes."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("K", [900, 901])
@pytest.mark.parametrize("weight,scale", [(np.inf, 1.0), (-np.inf, 1.0), (np.nan, 1.0), (3e38, 1e30)])
@pytest.mark.parametrize("method", ["tfm", "rca_rowtx"])
def test_only_samples_with_terms(method, weight, scale, K):
    from dream_b200.autograd import DASOperator
    if method == "tfm":
        Gt, Gr = synth.linear_array(6, 0.5), synth.linear_array(9, 0.4)
        Ro = synth.grid_xz(33, 40, (-5.0, 5.0), (2.0, 12.0))
    else:
        Gt, Gr = synth.rca_arrays(9, 6, 0.3)
        Ro = synth.grid_xyz(9, 7, 40, (-3.0, 3.0), (-3.0, 3.0), (2.0, 12.0))
    ncol = len(Gt) * len(Gr)
    dl = np.array([[0.1]])
    idx = oracle.das(np.zeros((K, ncol), order="F"), Gt, Gr, Ro, 0.04, dl, 1500.0, method, "ignore", np.float64,
                     return_idx=True)[3]
    idx = np.where((idx >= 0) & (idx < K), idx, -1)
    rng = np.random.default_rng(3)
    x = (scale * rng.uniform(0.5, 1.0, len(Ro))).astype(np.float32)  # positive: no sum cancels
    w = rng.uniform(0.5, 1.5, ncol).astype(np.float32)
    op = DASOperator(Gt, Gr, Ro, 0.04, dl, 1500.0, method, K)
    plain = op.adjoint(torch.from_numpy(x), torch.from_numpy(w)).t().cpu().numpy()
    sick = [1, 20, ncol - 1]
    w[sick] = weight
    Ya = op.adjoint(torch.from_numpy(x), torch.from_numpy(w)).t().cpu().numpy()
    for c in range(ncol):
        touched = np.zeros(K, bool)
        touched[idx[c][idx[c] >= 0]] = True
        if c in sick:
            assert not np.isfinite(Ya[c][touched]).any()
        else:  # the order of the additions may differ between the two calls
            assert np.abs(Ya[c] - plain[c]).max() <= 1e-5 * np.abs(plain[c]).max()
        assert not Ya[c][~touched].any(), f"A-scan {c}: {np.count_nonzero(Ya[c][~touched])} samples without a term"
