"""Edges of the adjoint's window scatter: outer and inner counts around its
batches of 2 x 8 and blocks of 40, A-scans that end or start inside the image,
lengths that leave rows unaligned, grids coarse enough for windows wider than
shared memory holds, narrow grids and weights.

Tolerance, per sample, against the FP64 adjoint at the oracle's indices: every
batch rounds |x| once to 2^-22 of the image's largest |x| (plus one FP32 rounding
of the sum), so with m terms on a sample |error| <= m * w * max|x| * 2^-21.5 + the
FP32 accumulation of at most m partial sums, m * 2^-24 * sum |w x|."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(method, n_out, n_in, grid, K, seed, x_rng=(-9.0, 7.0), z_rng=(1.0, 21.0), delay=0.1, weighted=False):
    from dream_b200.autograd import DASOperator
    rng = np.random.default_rng(seed)
    nt, nr = (n_in, n_out) if method == "rca_rowtx" else (n_out, n_in)
    if method == "tfm":
        Gt, Gr = synth.linear_array(nt, 0.5), synth.linear_array(nr, 0.4)
        Ro = synth.grid_xz(grid[0], grid[1], x_rng, z_rng)
    else:
        Gt, Gr = synth.rca_arrays(nt, nr, 0.3)
        Ro = synth.grid_xyz(grid[0], 3, grid[1], (-5.0, 6.0), (-4.0, 4.0), z_rng)
    dl = np.array([[delay]])
    idx = oracle.das(np.zeros((K, nt * nr), order="F"), Gt, Gr, Ro, 0.04, dl, 1500.0, method, "ignore", np.float64,
                     return_idx=True)[3]
    x = rng.normal(size=Ro.shape[0]).astype(np.float32)
    w = rng.uniform(0.5, 1.5, nt * nr).astype(np.float32) if weighted else np.ones(nt * nr, np.float32)
    idx = np.where((idx >= 0) & (idx < K), idx, -1)
    ref = np.zeros((nt * nr, K))
    terms = np.zeros((nt * nr, K))
    size = np.zeros((nt * nr, K))
    for c in range(nt * nr):
        ok = idx[c] >= 0
        np.add.at(ref[c], idx[c][ok], float(w[c]) * x[ok].astype(np.float64))
        np.add.at(size[c], idx[c][ok], float(w[c]) * np.abs(x[ok]).astype(np.float64))
        np.add.at(terms[c], idx[c][ok], 1.0)
    op = DASOperator(Gt, Gr, Ro, 0.04, dl, 1500.0, method, K)
    Ya = op.adjoint(torch.from_numpy(x), torch.from_numpy(w) if weighted else None).t().cpu().numpy().astype(np.float64)
    tol = terms * (w[:, None] * np.abs(x).max() * 2.0 ** -21.5 + size * 2.0 ** -24)
    bad = np.abs(Ya - ref) > tol
    assert not bad.any(), f"{bad.sum()} samples, worst {np.abs(Ya - ref).max()}"


@pytest.mark.parametrize("n_out", [1, 2, 3, 39, 40, 41, 81])
@pytest.mark.parametrize("weighted", [False, True])
def test_outer_counts(n_out, weighted):
    _check("tfm", n_out, 8, (20, 33), 900, n_out, weighted=weighted)


@pytest.mark.parametrize("n_in", [1, 7, 8, 9, 17])
def test_inner_counts(n_in):
    _check("tfm", 5, n_in, (20, 33), 900, n_in, weighted=True)


@pytest.mark.parametrize("method", ["tfm", "rca_coltx", "rca_rowtx"])
@pytest.mark.parametrize("K,delay", [(150, 0.1), (400, -2.0), (901, 0.3), (640, -1.36)])
def test_cut_and_unaligned_ascans(method, K, delay):
    _check(method, 7, 9, (17, 40), K, K, delay=delay, weighted=K == 901)


@pytest.mark.parametrize("grid,x_rng,z_rng", [((1, 50), (0.0, 0.0), (1.0, 21.0)), ((9, 40), (-60.0, 60.0), (1.0, 160.0)),
                                              ((40, 9), (-1.0, 1.0), (2.0, 3.0)), ((260, 170), (-9.0, 7.0), (1.0, 21.0))])
def test_grids(grid, x_rng, z_rng):
    """A line, a grid of windows wider than 192 samples, a fine grid, and one of 16 x 16-point tiles."""
    _check("tfm", 6, 9, grid, 1200, grid[0], x_rng, z_rng, weighted=True)
