"""The branch-free root and quotients of the SIR kernels against IEEE ones, one
surface element per point: the SIR then holds the single amplitude
w / (2 pi r) / dt * 1000. Squared distances next to the middle of two
neighbouring roots (the hard cases of a square root's rounding), next to squares
of representable numbers, and random ones over many binades; sampling periods
whose quotients round either way. Bit for bit, in both SIR kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NO = 200000
TWO_PI = 2.0 * 3.14159265358979323846264338328  # the product that the reference forms


def _points(kind, rng):
    """Points on x = 0 and on z > 0 whose squared distance x*x + 0 + z*z, as the kernels round it, is the wanted one
    or a neighbour of it."""
    r = np.exp(rng.uniform(np.log(0.05), np.log(60.0), NO))
    if kind == "random":
        return np.stack([r * rng.uniform(-1, 1, NO), r * rng.uniform(-1, 1, NO), r], 1)
    ld = np.longdouble
    mid = ld(r) + ld(np.spacing(r)) / 2 if kind == "middle" else ld(r)
    s = (mid * mid).astype(np.float64)  # the double nearest to it: within half a unit of the boundary
    s = s + rng.integers(-1, 2, NO) * np.spacing(s)
    z = np.sqrt(s) * (1.0 - 2.0 ** -12)  # x*x makes up the rest
    x = np.sqrt(np.maximum((ld(s) - ld(z * z)), 0)).astype(np.float64)
    return np.stack([x, np.zeros(NO), z], 1)


@pytest.mark.parametrize("count", [NO, 3000])  # one point per lane, one warp per point
@pytest.mark.parametrize("kind", ["random", "middle", "square"])
@pytest.mark.parametrize("dt,v", [(0.1, 1.0), (0.037, -2.5), (1.0 / 3.0, 1e-7), (0.25, 3.1e9)])
def test_amplitudes(dt, v, kind, count):
    from dream_b200.dreamrect import dreamrect
    rng = np.random.default_rng(int(1e3 * dt))
    Ro = np.asfortranarray(_points(kind, rng)[:count])
    d, cp = 0.2, 1500.0  # one surface element: centre at -0.1 + 0.1 = 0
    x, y, z = Ro.T
    r = np.sqrt((x * x + y * y) + z * z)
    nt = 16
    delay = (r * 1000.0 / cp) - 8.0 * dt  # every point lands near sample 8
    H = dreamrect(torch.from_numpy(np.ascontiguousarray(Ro.T)).cuda().t(), [d, d], [d, d, dt, nt], delay, [v, cp, 0.0],
                  "ignore").cpu().numpy()
    want = (v * (d * d)) / (TWO_PI * r) / dt * 1000.0
    assert (np.count_nonzero(H, axis=0) == 1).all()
    got = H.sum(0)  # one term and zeros: exact
    bad = got != want
    assert not bad.any(), f"{bad.sum()} of {count} amplitudes differ"
