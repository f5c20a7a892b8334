"""The device's grid hint equals grid_hint() on the host: changes at, before
and after block and grid boundaries, none at all, NaN coordinates, both
geometry precisions."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("No,n", [(1, 1), (2, 1), (2, 2), (60, 7), (60, 12), (256 * 300, 256), (256 * 300, 300 * 128),
                                  (200000, 100000), (200000, 199999), (200000, 200000), (512 * 512, 512)])
def test_device_hint_matches_host(No, n, dtype):
    from dream_b200 import _lib
    from dream_b200.beamformer import _device_grid_hint, grid_hint
    Ro = np.zeros((No, 3), dtype=dtype, order="F")
    Ro[:, 2] = np.arange(No)
    Ro[n:, (No + n) % 2] = 1.5
    prec = _lib.PREC_F64 if dtype == np.float64 else _lib.PREC_F32
    for bad in (False, True):
        if bad:
            Ro[No // 2, 0] = np.nan
        plan = _lib.plan_create(_lib.TFM, 10, No, 2, 2, prec, 0)
        t = torch.from_numpy(np.ascontiguousarray(Ro.T)).cuda().t()
        assert _device_grid_hint(plan, t, torch.cuda.current_stream().cuda_stream) == grid_hint(Ro)
