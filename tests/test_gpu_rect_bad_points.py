"""Large dreamrect fields with points that no window holds: NaN and infinite
coordinates, and points so far away that sample estimates are not trusted. They
have no sample in the SIR; every other point's SIR equals the oracle's bit for
bit, and the field takes at most twice the time of one without them (a bad point
costs a warp about 60000 / 32 steps, a fraction of the field's time; a repeat of
the whole field costs three times it). Per-point delays of
many thousand samples, which one point per lane computes with the IEEE root and
quotients."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NO = 31 * 997  # more points than one round of lanes: the lane kernel's range


def _points(seed):
    rng = np.random.default_rng(seed)
    return np.asfortranarray(np.stack([rng.uniform(-6, 6, NO), rng.uniform(-6, 6, NO), rng.uniform(0.5, 25, NO)], 1))


def _run(Ro, a, b, d, dt, nt, delay, cp=1500.0):
    from dream_b200.dreamrect import dreamrect
    t = torch.from_numpy(np.ascontiguousarray(Ro.T)).cuda().t()
    return lambda: dreamrect(t, [a, b], [d, d, dt, nt], delay, [1.0, cp, 0.0], "ignore")


def _ms(fn):
    best = np.inf
    for _ in range(5):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        fn()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


@pytest.mark.parametrize("bad", [(np.nan, 0.0, 5.0), (0.0, 0.0, np.inf), (0.0, 0.0, 1e12), (3e11, np.nan, 1.0)])
@pytest.mark.parametrize("many", [False, True])
def test_points_without_a_window(bad, many):
    Ro = _points(1)
    good = _run(Ro, 10.0, 15.0, 0.05, 0.1, 190, 0.0)
    good()
    t_good = _ms(good)
    sick = np.arange(NO)[::1999] if many else np.array([12345])
    Ro[sick] = bad
    fn = _run(Ro, 10.0, 15.0, 0.05, 0.1, 190, 0.0)
    H = fn().cpu().numpy()
    some = np.setdiff1d(np.concatenate([np.arange(0, NO, 61), np.arange(12320, 12370)]), sick)
    ref = oracle.rect(np.asfortranarray(Ro[some]), 10.0, 15.0, 0.05, 0.05, 0.1, 190, 0.0, 1.0, 1500.0)[0]
    assert np.array_equal(H[:, some], ref)
    assert not H[:, sick].any()
    assert _ms(fn) <= 2.0 * t_good


@pytest.mark.parametrize("nt", [60, 100])
def test_long_delays_by_lane(nt):
    """20 ps samples: numbers beyond the packed format's 65536, yet every SIR starts inside its window."""
    Ro = _points(2)
    dt = 2e-5
    ex, ey = np.maximum(np.abs(Ro[:, 0]) - 0.1, 0.0), np.maximum(np.abs(Ro[:, 1]) - 0.1, 0.0)
    delay = np.sqrt(ex ** 2 + ey ** 2 + Ro[:, 2] ** 2) * 1e3 / 1500.0 - 3 * dt
    H = _run(Ro, 0.2, 0.2, 0.05, dt, nt, delay)().cpu().numpy()
    ref, _, oob = oracle.rect(Ro, 0.2, 0.2, 0.05, 0.05, dt, nt, delay, 1.0, 1500.0)
    assert np.array_equal(H, ref)
    assert np.count_nonzero(ref) > 0 and oob > 0
