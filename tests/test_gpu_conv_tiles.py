"""Edges of the convolution kernel's tiles (640 or 896 outputs), trips (8 or 10
steps) and triangle ends, in all three modes. Bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mode", ["=", "+=", "-="])
@pytest.mark.parametrize("M,L,N", [(1, 1, 3), (5, 8, 2), (639, 1, 2), (640, 2, 2), (641, 9, 3), (633, 8, 2),
                                   (200, 700, 2), (700, 700, 2), (1400, 33, 2), (30, 4097, 2), (2000, 4100, 1),
                                   (4, 3, 4200), (897, 10, 4096)])
def test_tile_edges(M, L, N, mode):
    from dream_b200.conv import conv_p
    rng = np.random.default_rng(M * 7 + L)
    A, B = np.asfortranarray(rng.normal(size=(M, N))), rng.normal(size=L)
    Y = np.asfortranarray(rng.normal(size=(M + L - 1, N)))
    Y[::5] = -0.0
    ref = oracle.conv_p(A, B, None if mode == "=" else Y.copy(order="F"), mode)
    d = lambda a: torch.empty(a.shape[::-1], dtype=torch.float64, device="cuda").copy_(torch.from_numpy(a.T.copy())).t()
    out = conv_p(d(A), torch.from_numpy(B).cuda(), d(Y), mode).cpu().numpy()
    assert np.array_equal(out, ref) and np.array_equal(np.signbit(out), np.signbit(ref))
