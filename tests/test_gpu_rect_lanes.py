"""dreamrect with one point per lane (large fields): rows around the groups of
8 terms, a last warp that is partly filled, per-point delays, windows cut by
both ends of the SIR, fields that miss it, points on the aperture itself, and
values outside the branch-free operations' range. SIRs and out-of-bounds
statuses must equal the oracle's bit for bit; and arrays whose rows end the
steps of 32 terms."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NO = 31 * 997  # more points than one round of lanes: the lane kernel's range


def _points(seed, z_lo=0.5):
    rng = np.random.default_rng(seed)
    return np.asfortranarray(np.stack([rng.uniform(-6, 6, NO), rng.uniform(-6, 6, NO), rng.uniform(z_lo, 25, NO)], 1))


def _compare(Ro, a, b, dx, dy, dt, nt, delay, v=1.0, cp=1500.0):
    from dream_b200.dreamrect import dreamrect
    d = torch.from_numpy(np.ascontiguousarray(Ro.T)).cuda().t()
    H = dreamrect(d, [a, b], [dx, dy, dt, nt], delay, [v, cp, 0.0], "ignore").cpu().numpy()
    ref, st, oob = oracle.rect(Ro, a, b, dx, dy, dt, nt, delay, v, cp)
    assert np.array_equal(H, ref), f"{np.sum(H != ref)} of {H.size} samples differ"


@pytest.mark.parametrize("nx", [1, 7, 8, 9, 16, 23])
def test_row_lengths(nx):
    _compare(_points(nx), 0.1 * nx, 0.5, 0.1, 0.1, 0.1, 190, 0.0)


@pytest.mark.parametrize("nt,delay", [(40, 0.0), (60, 9.0), (30, 40.0), (200, -3.0)])
def test_cut_windows(nt, delay):
    _compare(_points(nt), 2.0, 1.0, 0.1, 0.1, 0.1, nt, delay)


def test_per_point_delays():
    _compare(_points(3), 1.1, 0.7, 0.1, 0.1, 0.1, 150, np.random.default_rng(4).uniform(-2.0, 6.0, NO))


def test_points_on_the_aperture():
    Ro = _points(5)
    Ro[::64, 2] = 0.0
    Ro[::64, :2] *= 0.1
    _compare(Ro, 1.3, 0.9, 0.1, 0.1, 0.05, 400, 0.0)


@pytest.mark.parametrize("v,dt,nt", [(1e-305, 0.1, 100), (0.0, 0.1, 100), (1.0, 2e-5, 300), (-2.5, 0.37, 64)])
def test_value_ranges(v, dt, nt):
    """A velocity beyond the quotients' range, sample numbers beyond the packed format's, an odd sampling period."""
    _compare(_points(6), 0.9, 0.4, 0.1, 0.1, dt, nt, 0.0 if dt > 1e-3 else 5.0, v=v)


@pytest.mark.parametrize("size,d", [(0.9, 0.03), (1.0, 0.1), (2.2, 0.05), (0.7, 0.11)])
def test_array_rows(size, d):
    from dream_b200.dreamrect import dream_arr_rect
    rng = np.random.default_rng(int(100 * size))
    Ro = np.asfortranarray(np.stack([rng.uniform(-8, 8, 300), rng.uniform(-4, 4, 300), rng.uniform(0.0, 30, 300)], 1))
    gx, gy = np.meshgrid(np.arange(-3.0, 4.0), np.arange(-2.0, 3.0))
    G = np.asfortranarray(np.stack([gx.ravel(), gy.ravel(), np.zeros(gx.size)], 1))
    ref, st, oob = oracle.arr_rect(Ro, size, size, G, d, d, 0.05, 120, 8.0, 1.0, 1500.0, "xy", 15.0, "x", 10.0, 0.0)
    out = dream_arr_rect(Ro, [size, size], G, [d, d, 0.05, 120], 8.0, [1.0, 1500.0, 0.0], "xy", 15.0, "x", [10.0, 0.0],
                         "off", np.ones(len(G)), 1.0, "ignore")
    assert np.array_equal(out, ref)
