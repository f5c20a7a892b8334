"""Arrays whose elements have few surface elements: 32 consecutive terms per step,
whatever element they belong to. Steps that hold many elements, one and parts of
two, chunks of 32 elements with dead ones among them, a last element that is in or
out of bounds, points without trusted sample estimates, fields below and above a
wave of blocks. SIRs, statuses and out-of-bounds counts equal the oracle's. Cutting
the same aperture into more elements of fewer surface elements must not cost more
than its share: the same terms in 441 elements of 1 within three times their time in
49 elements of 9 (one step per element would take nine times it)."""
import ctypes

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _grid(nx, ny, pitch):
    gx, gy = np.meshgrid((np.arange(nx) - nx / 2) * pitch, (np.arange(ny) - ny / 2) * pitch)
    return np.asfortranarray(np.stack([gx.ravel(), gy.ravel(), np.zeros(gx.size)], 1))


def _counts(Ro, a, b, G, dx, dy, dt, nt, delay, level):
    """(SIRs, status, out-of-bounds terms) through the C entry, focused and steered."""
    from dream_b200 import _lib
    L = _lib.load()
    No = len(Ro)
    H = np.zeros((nt, No), order="F")
    d, f = np.array([delay]), np.array([15.0])
    oob = ctypes.c_int64(0)
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    st = L.dream_arr_rect_run(p(Ro), No, a, b, dx, dy, dt, nt, 0, p(d), 1.0, 1500.0, len(G), p(G), 3, p(f), 1, 20.0, 0.0,
                              0, None, 0.0, p(H), level, ctypes.byref(oob), 0)
    return H, st, oob.value


@pytest.mark.parametrize("No", [61, 4900])
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (1, 5), (3, 3), (5, 6), (31, 1), (1, 33), (6, 6), (7, 7), (10, 10), (3, 60)])
@pytest.mark.parametrize("elements", [(5, 1), (8, 4), (11, 9)])
def test_terms_across_elements(elements, nx, ny, No):
    rng = np.random.default_rng(No + nx * 100 + ny)
    if No > 1000 and nx * ny * elements[0] * elements[1] > 3600:
        No = 700
    Ro = np.asfortranarray(np.stack([rng.uniform(-9, 9, No), rng.uniform(-5, 5, No), rng.uniform(0.0, 25, No)], 1))
    Ro[::97, 2] = 0.0
    Ro[1::97] = (np.nan, 0.0, 5.0)
    Ro[2::97, 2] = 1e13
    G = _grid(*elements, 0.8)
    d = 0.06
    a, b = nx * d, ny * d
    for nt, delay in ((25, 7.0), (300, 0.0)):
        for level, name in ((1, "ignore"), (2, "warn")):
            H, st, oob = _counts(Ro, a, b, G, d, d, 0.1, nt, delay, level)
            ref, st_ref, oob_ref = oracle.arr_rect(Ro, a, b, G, d, d, 0.1, nt, delay, 1.0, 1500.0, "xy", 15.0, "x", 20.0,
                                                   0.0, err_level=name)
            assert np.array_equal(H, ref), f"{np.sum(H != ref)} samples differ"
            assert (st, oob) == (st_ref, oob_ref)


def test_more_smaller_elements():
    from dream_b200.dreamrect import dream_arr_rect
    rng = np.random.default_rng(1)
    No = 60000
    Ro = torch.from_numpy(np.stack([rng.uniform(-10, 10, No), rng.uniform(-10, 10, No), rng.uniform(1, 40, No)])).cuda().t()

    def ms(side, nx):
        G, d = _grid(side, side, 21 / side), 0.3
        fn = lambda: dream_arr_rect(Ro, [nx * d, nx * d], G, [d, d, 0.1, 400], 0.0, [1.0, 1500.0, 0.0], "off", 0.0, "off",
                                    [0.0, 0.0], "off", np.ones(len(G)), 1.0, "ignore")
        fn()
        best = np.inf
        for _ in range(5):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best
    assert ms(21, 1) <= 3.0 * ms(7, 3)
