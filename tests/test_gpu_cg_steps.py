"""Conjugate-gradient vector updates (csrc/cg.cu) against the same step in
torch: vector lengths around warps, blocks and the largest grid, and whole
solves on both paths."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ULP = 2.0 ** -23


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 65536, 256 * 1024, 256 * 1024 + 1, 3 * 256 * 1024 + 77])
def test_step_matches_torch(n):
    """Two steps in a row. Element-wise results round as torch's do; the dot
    products have positive terms, so their FP64 sums are within n 2^-53 and the
    FP32 scalars within 1 ulp (one rounding that may fall the other way), alpha
    and beta within 3."""
    from dream_b200 import _lib
    L = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda: torch.rand(n, device="cuda", generator=g) + 0.5
    x, r, p = rnd(), rnd(), rnd()
    rs = torch.empty(2, device="cuda")
    scratch = torch.empty(_lib.CG_SCRATCH_BYTES, dtype=torch.uint8, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t, i=0: ctypes.c_void_p(t.data_ptr() + 4 * i)
    _lib.check(L.dream_das_cg_start(ptr(r), n, ptr(scratch), 0, st))
    lam = 0.37
    for i in range(2):
        Ap = rnd()
        x0, r0, p0, rs0 = x.clone(), r.clone(), p.clone(), (r.double() @ r.double()).float()
        A1 = Ap + lam * p0
        _lib.check(L.dream_das_cg_step(ptr(x), ptr(r), ptr(p), ptr(Ap), n, lam, ptr(rs, i), ptr(scratch), 0, st))
        torch.cuda.synchronize()
        assert torch.equal(Ap, A1)
        alpha = (rs0 / (p0.double() @ A1.double()).float()).double()
        for got, base, step in ((x, x0, alpha * p0.double()), (r, r0, -alpha * A1.double())):
            bound = 5 * ULP * step.abs() + ULP * (base.double() + step).abs()
            assert bool(((got.double() - (base.double() + step)).abs() <= bound).all())
        rs1 = (r.double() @ r.double()).float()
        assert abs(float(rs[i]) - float(rs1)) <= ULP * float(rs1)
        beta = (rs1 / rs0).double()
        bound = 6 * ULP * beta * p0.double().abs() + ULP * (r.double() + beta * p0.double()).abs()
        assert bool(((p.double() - (r.double() + beta * p0.double())).abs() <= bound).all())


@pytest.mark.parametrize("start", [False, True])
def test_solve_matches_torch_path(start):
    """A tensor lam takes the torch updates. The paths differ by the rounding of
    FP32 dot products and the order of the adjoint's sums (1e-6), which three
    iterations may amplify: 1e-3 of the largest value."""
    from dream_b200 import synth
    from dream_b200.autograd import DASOperator, cg_reconstruct
    s = synth.cg_scene(seed=5, n_el=16, K=1024, nx=31, nz=57, x_rng=(-4.0, 4.0), z_rng=(5.0, 20.0))
    op = DASOperator(s.Gt, s.Gr, s.Ro, s.dt, s.delay, s.cp, "tfm", 1024)
    xt = torch.from_numpy(s.extra["reflectivity"]).float().cuda()
    w = torch.rand(op.ncol, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) + 0.5
    Y = op.adjoint(xt, w)
    x0 = 0.3 * xt if start else None
    x0_before = x0.clone() if start else None
    x, res = cg_reconstruct(op, Y, w, 1e-3, 3, x0=x0)
    xr, resr = cg_reconstruct(op, Y, w, torch.tensor(1e-3, device="cuda"), 3, x0=x0)
    assert res.shape == resr.shape == (3,) and x.shape == xr.shape
    assert float((x - xr).abs().max()) <= 1e-3 * float(xr.abs().max())
    assert float((res - resr).abs().max()) <= 1e-3 * float(resr.max())
    assert x0 is None or torch.equal(x0, x0_before)
