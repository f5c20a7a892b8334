"""NaN and infinities in either operand of conv_p, in all three modes: an output
meets only the products of samples inside both columns, as in the reference's
loops, so non-finite values reach their own outputs and no others. Bit for bit
against the oracle, NaN positions included."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mode", ["=", "+=", "-="])
@pytest.mark.parametrize("M,L,N", [(1, 1, 3), (5, 8, 2), (640, 2, 2), (200, 700, 2), (700, 700, 2), (1400, 33, 2),
                                   (30, 4097, 2), (897, 10, 4096)])
@pytest.mark.parametrize("where", ["B first", "B last", "B middle", "A ends", "both"])
def test_non_finite_operands(where, M, L, N, mode):
    from dream_b200.conv import conv_p
    rng = np.random.default_rng(M * 7 + L)
    A, B = np.asfortranarray(rng.normal(size=(M, N))), rng.normal(size=L)
    if where == "B first":
        B[0] = np.inf
    elif where == "B last":
        B[-1] = np.nan
    elif where in ("B middle", "both"):
        B[L // 2] = -np.inf
    if where in ("A ends", "both"):
        A[0, 0] = np.nan
        A[-1, -1] = np.inf
    Y = np.asfortranarray(rng.normal(size=(M + L - 1, N)))
    Y[::5] = -0.0
    ref = oracle.conv_p(A, B, None if mode == "=" else Y.copy(order="F"), mode)
    d = lambda a: torch.empty(a.shape[::-1], dtype=torch.float64, device="cuda").copy_(torch.from_numpy(a.T.copy())).t()
    out = conv_p(d(A), torch.from_numpy(B).cuda(), d(Y), mode).cpu().numpy()
    assert np.array_equal(out, ref, equal_nan=True)
    num = ~np.isnan(ref)
    assert np.array_equal(np.signbit(out[num]), np.signbit(ref[num]))
