"""Leg tables of exactly 48 KB, the dynamic shared memory that a launch may ask
for without raising the kernel's limit when the kernel has no static arrays:
48 outer elements of the storage gathers (48 x 128 threads x 8 bytes), 65 - 96
inner elements of the plain FP32 kernel. The A-scans are whole numbers and the
FP32 image of the gather is a sum of fewer than 2^24 of them: exact."""
import numpy as np
import pytest

from dream_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _frame(method, nt, nr, dtype):
    rng = np.random.default_rng(nt)
    if method == "tfm":
        Gt, Gr = synth.linear_array(nt, 0.5), synth.linear_array(nr, 0.4)
        Ro = synth.grid_xz(9, 41, (-9.0, 7.0), (1.0, 21.0))
    else:
        Gt, Gr = synth.rca_arrays(nt, nr, 0.3)
        Ro = synth.grid_xyz(5, 3, 33, (-5.0, 6.0), (-4.0, 4.0), (1.0, 16.0))
    f = lambda a: np.asfortranarray(a, dtype=dtype)
    Y = rng.integers(-50, 51, size=(900, nt * nr))
    return f(Y), f(Gt), f(Gr), f(Ro), dtype(0.04), f([[0.1]]), dtype(1500.0)


@pytest.mark.parametrize("n", [47, 48, 49, 96])
@pytest.mark.parametrize("method", ["tfm", "rca_coltx"])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_storage_gather(n, method, storage):
    from dream_b200.beamformer import das_mixed
    args = _frame(method, n, 12 if method == "tfm" else n, np.float64)
    ref = oracle.das(*args, method, "ignore", np.float64)[0]
    Im = das_mixed(torch.from_numpy(args[0].astype(np.float32)).cuda(), *args[1:], method, "ignore", "cuda", storage)
    assert np.array_equal(Im.cpu().numpy().astype(np.float64), ref)


@pytest.mark.parametrize("n", [64, 65, 96, 97])
def test_plain_f32(n):
    from dream_b200 import das_f
    args = _frame("tfm", 5, n, np.float32)
    assert np.array_equal(das_f.das(*args, "tfm", "ignore", "cuda"), oracle.das(*args, "tfm", "ignore", np.float32)[0])
