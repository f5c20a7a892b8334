"""Timed workloads of the beamformer, its operators and the A-scan models.

Every case is one call (or one short sequence of calls) that a program using
this package makes: plain and mixed-precision delay-and-sum of SAFT, TFM and
row-column frames, the differentiable operator, a model-based reconstruction,
a batch of uneven frames, full-matrix-capture synthesis and the spatial impulse
responses of a rectangular element and of an array. Sizes are those of the
package's scenes (dream_b200.synth), tests and benchmark, and ragged ones
between them. ``draw`` spreads each kind over its range.

Lengths are in mm, times in us, speeds in m/s.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dream_b200 import das as das64
from dream_b200 import das_f as das32
from dream_b200 import synth
from dream_b200.autograd import DASOperator, cg_reconstruct, das_gather
from dream_b200.batch import DASBatch, make_frame
from dream_b200.beamformer import das_mixed
from dream_b200.conv import fmc_synthesis
from dream_b200.dreamrect import dream_arr_rect, dreamrect

DEV = "cuda"


def listed():
    return [
        # a SAFT test image from NumPy arrays: the smallest call of a script that switches from DREAM's own module
        dict(name="saft_f64_host", kind="das", precision="f64", method="saft", host=True, multi_delay=False, nt=64,
             nr=0, K=2048, nx=64, ny=1, nz=64),
        # the reference call in its own precision on the benchmark's full-matrix-capture frame
        dict(name="tfm_f64", kind="das", precision="f64", method="tfm", host=False, multi_delay=False, nt=64, nr=64,
             K=3000, nx=512, ny=1, nz=512),
        # the reference's single-precision module, unequal arrays, odd sizes and one delay per point
        dict(name="tfm_f32_ragged", kind="das", precision="f32", method="tfm", host=False, multi_delay=True, nt=37,
             nr=53, K=1777, nx=301, ny=1, nz=203),
        # the headline frame: FP32-stored A-scans resident on the device
        dict(name="tfm_mixed_f32", kind="mixed", storage="f32", method="tfm", multi_delay=False, nt=64, nr=64, K=3000,
             nx=512, ny=1, nz=512),
        # BF16-stored A-scans on a ragged frame, as an acquisition with dead channels gives it
        dict(name="tfm_mixed_bf16_ragged", kind="mixed", storage="bf16", method="tfm", multi_delay=False, nt=61, nr=47,
             K=2501, nx=387, ny=1, nz=271),
        # a row-column volume: the largest beamforming call, its A-scans larger than the L2 cache
        dict(name="rca_mixed_f32", kind="mixed", storage="f32", method="rca_rowtx", multi_delay=False, nt=128, nr=128,
             K=4096, nx=128, ny=128, nz=256),
        # one training step on the frame: image, and the gradients of the A-scans and of the apodisation weights
        dict(name="tfm_gradients", kind="grad", method="tfm", nt=64, nr=64, K=3000, nx=512, nz=512),
        # model-based reconstruction, conjugate gradients on the normal equations
        dict(name="cg_32x32", kind="cg", nt=32, nr=32, K=2048, nx=256, nz=256, iters=10),
        # uneven frames of several probes in one launch
        dict(name="batch_12_uneven", kind="batch", n_frames=12, frames_seed=7, max_side=512),
        # A-scans of a whole full-matrix capture from 101 element responses
        dict(name="fmc_101", kind="fmc", M=2000, lt=101, pulse=150),
        # field of a 10 x 15 mm element, 60000 surface elements per point
        dict(name="sir_rect_field", kind="rect", a=10.0, b=15.0, d=0.05, dt=0.25, nt=300, nx=61, ny=61, nz=24),
        # a focused and steered 21 x 21 array seen from a 101 x 80 mm plane through a short window
        dict(name="sir_array_plane", kind="arr", side=21, size=0.9, d=0.03, dt=0.1, nt=13, nx=201, nz=161),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["das", "das", "mixed", "mixed", "mixed", "grad", "cg", "batch", "fmc", "rect", "arr"])
    if kind in ("das", "mixed"):
        method = rng.choice(["saft", "tfm", "tfm", "tfm", "rca_coltx", "rca_rowtx"])
        c = dict(kind=kind, method=method, multi_delay=rng.random() < 0.3, nt=rng.randint(8, 128),
                 nr=0 if method == "saft" else rng.randint(8, 128), K=rng.randint(512, 4096))
        if method.startswith("rca"):
            top = (96, 200) if kind == "mixed" else (40, 100)
            c["nr"] = c["nt"]
            c.update(nx=rng.randint(16, top[0]), ny=rng.randint(16, top[0]), nz=rng.randint(32, top[1]))
        else:
            c.update(nx=_log_int(rng, 32, 512), ny=1, nz=_log_int(rng, 32, 512))
        if kind == "mixed":
            c["storage"] = rng.choice(["f32", "bf16"])
        else:
            # whole frames come from the host where they are small
            c.update(precision=rng.choice(["f64", "f32"]), host=c["nt"] * max(c["nr"], 1) <= 1024 and rng.random() < 0.5)
        return c
    if kind == "grad":
        return dict(kind=kind, method="tfm", nt=rng.randint(8, 64), nr=rng.randint(8, 64), K=rng.randint(1024, 3000),
                    nx=_log_int(rng, 64, 512), nz=_log_int(rng, 64, 512))
    if kind == "cg":
        return dict(kind=kind, nt=rng.randint(12, 40), nr=rng.randint(12, 40), K=rng.randint(1024, 2048),
                    nx=rng.randint(100, 256), nz=rng.randint(100, 256), iters=rng.randint(4, 10))
    if kind == "batch":
        return dict(kind=kind, n_frames=rng.randint(2, 12), frames_seed=rng.randint(1, 10 ** 6),
                    max_side=rng.randint(64, 512))
    if kind == "fmc":
        return dict(kind=kind, M=_log_int(rng, 200, 2000), lt=_log_int(rng, 8, 101), pulse=rng.randint(20, 150))
    if kind == "rect":
        return dict(kind=kind, a=round(rng.uniform(0.4, 10.0), 3), b=round(rng.uniform(1.0, 15.0), 3),
                    d=rng.choice([0.05, 0.1]), dt=rng.choice([0.02, 0.1, 0.25]), nt=rng.randint(200, 2000),
                    nx=rng.randint(8, 61), ny=rng.randint(1, 61), nz=rng.randint(1, 24))
    return dict(kind="arr", side=rng.randint(3, 21), size=0.9, d=0.03, dt=0.1, nt=rng.randint(13, 200),
                nx=rng.randint(21, 101), nz=rng.randint(21, 81))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _generator(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed + 1) + salt)


def _stripe_offset(c, edges):
    """The reference's clamp of a coordinate against the stripe edges (lo, hi)."""
    lo, hi = edges
    return torch.where((c >= lo) & (c <= hi), torch.zeros_like(c), torch.where(c < lo, lo - c, hi - c))


def _leg_parts(Gt, Gr, P, method):
    """Coordinate differences of the transmit (column) and receive (row) legs: two functions of the element number
    that give (dx, dy, dz) in the dtype of the inputs."""
    x, y, z = P[:, 0], P[:, 1], P[:, 2]
    if method.startswith("rca"):
        nt, nr = Gt.shape[0], Gr.shape[0]
        gr, gt = Gr.t().reshape(-1), Gt.t().reshape(-1)
        gy = _stripe_offset(y, (gr[nt], gr[2 * nt - 1]))
        gx = _stripe_offset(x, (gt[0], gt[nr - 1]))
        return (lambda e: (Gt[e, 0] - x, gy, Gt[e, 2] - z)), (lambda e: (gx, Gr[e, 1] - y, Gr[e, 2] - z))
    return (lambda e: tuple(Gt[e, k] - P[:, k] for k in range(3))), (lambda e: tuple(Gr[e, k] - P[:, k] for k in range(3)))


def _leg(parts, ocp):
    dx, dy, dz = parts
    return torch.sqrt(dx * dx + dy * dy + dz * dz) * ocp


def _ascans(Gt, Gr, dt, cp, method, K, z_max, x_half, seed):
    """A-scans of ten point scatterers (5 MHz Gaussian-windowed sine) in noise, (K, columns) column-major FP32."""
    gen = _generator(seed, 1)
    r = np.random.default_rng(seed)
    S = np.stack([r.uniform(-0.6 * x_half, 0.6 * x_half, 10), np.zeros(10), r.uniform(0.25 * z_max, 0.9 * z_max, 10)], 1)
    if method.startswith("rca"):
        S[:, 1] = r.uniform(-0.6 * x_half, 0.6 * x_half, 10)
    amp = r.uniform(0.5, 1.0, 10)
    Gt, Gr, S = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in (Gt, Gr, S))
    tx, rx = _leg_parts(Gt, Gr, S, method)
    a = torch.stack([_leg(tx(e), 1000.0 / cp) for e in range(Gt.shape[0])])  # (nt, 10), us
    if method == "saft":
        t = 2.0 * a
    else:
        b = torch.stack([_leg(rx(e), 1000.0 / cp) for e in range(Gr.shape[0])])
        o, i = (b, a) if method == "rca_rowtx" else (a, b)
        t = (o[:, None, :] + i[None, :, :]).reshape(-1, 10)
    C = t.shape[0]
    Y = torch.randn((C, K), generator=gen, device=DEV, dtype=torch.float32) * 0.01
    half = int(math.ceil(0.5 / dt)) + 1
    offs = torch.arange(-half, half + 1, device=DEV)
    cols = torch.arange(C, device=DEV)[:, None]
    for s in range(10):  # one scatterer at a time: every sample is touched once, so the sum has one order
        k = torch.floor(t[:, s] / dt).long()[:, None] + offs
        tau = k * dt - t[:, s][:, None]
        val = amp[s] * torch.exp(-tau * tau / 0.02) * torch.sin(2.0 * math.pi * 5.0 * tau)
        ok = (k >= 0) & (k < K)
        Y.view(-1)[(cols * K + k)[ok]] += val[ok].float()
    return Y.t()


def _frame(c, seed):
    """Geometry, delay and A-scans of one das call."""
    method, rca = c["method"], c["method"].startswith("rca")
    r = np.random.default_rng(7919 * (seed + 1))
    cp = float(r.uniform(1450.0, 1550.0))
    dt = 0.025 if rca else 0.04
    # imaged depth after the A-scan length, so that most paths fit in it
    z_max = min(35.0 if rca else 50.0, 0.35 * c["K"] * dt * cp / 1000.0)
    x_half = min(19.0 if rca else 20.0, 0.5 * z_max)
    if rca:
        Gt, Gr = synth.rca_arrays(c["nt"], c["nr"], 0.3)
        Ro = synth.grid_xyz(c["nx"], c["ny"], c["nz"], (-x_half, x_half), (-x_half, x_half),
                            (5.0 if z_max > 10 else 1.0, z_max))
    else:
        Gt = synth.linear_array(c["nt"], 0.5)
        Gr = synth.linear_array(c["nr"], 0.5) if c["nr"] else np.zeros((0, 3), order="F")
        Ro = synth.grid_xz(c["nx"], c["nz"], (-x_half, x_half), (2.0, z_max))
    delay = r.uniform(0.0, 0.4, Ro.shape[0] if c.get("multi_delay") else 1)
    Y = _ascans(Gt, Gr, dt, cp, method, c["K"], z_max, x_half, seed)
    return dict(Y=Y, Gt=Gt, Gr=Gr, Ro=Ro, dt=dt, delay=delay.reshape(-1, 1), cp=cp)


def _fortran(a, dtype):
    """Column-major device tensor of a NumPy array, as device-resident programs keep it."""
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).to(device=DEV, dtype=dtype).t()


def _batch_specs(c):
    specs = synth.batch_specs(c["frames_seed"], c["n_frames"])
    for sp in specs:
        sp["side"] = min(sp["side"], c["max_side"])
    return specs


def _batch_frames(c, seed):
    out = []
    for i, sp in enumerate(_batch_specs(c)):
        K, cp, dt = sp["K"], sp["cp"], sp["dt"]
        z_max = min(50.0, 0.35 * K * dt * cp / 1000.0)
        x_half = min(20.0, 0.5 * z_max)
        G = synth.linear_array(sp["n_el"], 0.5)
        Ro = synth.grid_xz(sp["side"], sp["side"], (-x_half, x_half), (2.0, z_max))
        out.append(dict(Y=_ascans(G, G, dt, cp, "tfm", K, z_max, x_half, 101 * seed + i), Gt=G, Gr=G, Ro=Ro, dt=dt,
                        delay=np.zeros((1, 1)), cp=cp))
    return out


def _weights(n, seed):
    return torch.rand(n, generator=_generator(seed, 2), device=DEV) + 0.5


def _synthesis_inputs(c, seed):
    """Element responses (a plateau with decaying edges, as a small element's are) and a Gaussian-windowed sine."""
    r = np.random.default_rng(seed)
    k = np.arange(c["M"])[:, None]
    start = r.uniform(0.1, 0.5, c["lt"]) * c["M"]
    width = r.uniform(0.02, 0.3, c["lt"]) * c["M"]
    x = (k - start) / width
    H = np.where((x >= 0) & (x <= 1), 1.0 / (1.0 + 3.0 * np.clip(x, 0.0, 1.0)), 0.0)
    H += 1e-3 * r.normal(size=H.shape) * (x >= 0)
    tau = (np.arange(c["pulse"]) - c["pulse"] / 2) * 0.02
    return H, np.exp(-tau * tau / (2.0 * 0.2 ** 2)) * np.sin(2.0 * np.pi * 4.0 * tau)


def _rect_inputs(c, seed):
    r = np.random.default_rng(seed)
    if c["kind"] == "rect":
        half = 1.5 * max(c["a"], 1.0)
        ax = [np.linspace(-half, half, c["nx"]), np.linspace(-half, half, c["ny"]) if c["ny"] > 1 else np.zeros(1),
              np.linspace(2.0, 65.0, c["nz"]) if c["nz"] > 1 else np.full(1, 10.0)]
        shift, cp = r.uniform(0.0, 0.2, 3), 1000.0 if c["dt"] > 0.2 else 1500.0
    else:
        ax = [np.linspace(-50.0, 50.0, c["nx"]), np.zeros(1), np.linspace(1.0, 80.0, c["nz"])]
        shift, cp = r.uniform(0.0, 0.4, 3), 1500.0
    Ro = np.stack([g.reshape(-1) for g in np.meshgrid(*ax, indexing="ij")], 1) + shift
    delay = 0.0 if c["kind"] == "rect" else (50.0 - 0.075 * c["nt"]) * 1e3 / cp
    return Ro, delay, cp


def _array_grid(c):
    p = np.arange(c["side"]) - (c["side"] - 1) / 2.0
    gx, gy = np.meshgrid(p, p)
    return np.stack([gx.ravel(order="F"), gy.ravel(order="F"), np.zeros(gx.size)], 1)


def _centres(size, d):
    """Surface-element centres by repeated addition, as the reference's loops step them."""
    out, v = [], -size / 2.0 + d / 2.0
    while v <= size / 2.0:
        out.append(v)
        v += d
    return out


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    if kind == "das":
        f = _frame(c, seed)
        ndt, tdt = (np.float64, torch.float64) if c["precision"] == "f64" else (np.float32, torch.float32)
        if c["host"]:
            f["Y"] = np.asfortranarray(f["Y"].cpu().numpy().astype(ndt))
            for k in ("Gt", "Gr", "Ro", "delay"):
                f[k] = np.asfortranarray(f[k].astype(ndt))
        else:
            f["Y"] = f["Y"].to(tdt)
            for k in ("Gt", "Gr", "Ro", "delay"):
                f[k] = _fortran(f[k], tdt)
        return dict(c, f=f)
    if kind == "mixed":
        f = _frame(c, seed)
        for k in ("Gt", "Gr", "Ro", "delay"):
            f[k] = _fortran(f[k], torch.float64)
        return dict(c, f=f)
    if kind in ("grad", "cg"):
        f = _frame(dict(c, method="tfm"), seed)
        op = DASOperator(f["Gt"], f["Gr"], f["Ro"], f["dt"], f["delay"], f["cp"], "tfm", c["K"])
        w = _weights(op.ncol, seed)
        g = torch.randn(op.No, generator=_generator(seed, 3), device=DEV)
        if kind == "grad":
            return dict(c, op=op, Y=f["Y"].requires_grad_(), w=w.requires_grad_(), g=g)
        return dict(c, op=op, Y=f["Y"], w=w)
    if kind == "batch":
        frames = [make_frame(f["Y"], f["Gt"], f["Gr"], f["Ro"], f["dt"], f["delay"], f["cp"], "tfm", DEV)
                  for f in _batch_frames(c, seed)]
        # the library's own tiles: tuned ones would differ from one timing run to the next
        return dict(c, batch=DASBatch(frames, autotune=False), images=[f.Im for f in frames])
    if kind == "fmc":
        H, p = _synthesis_inputs(c, seed)
        return dict(c, H=_fortran(H, torch.float64), p=torch.from_numpy(p).to(DEV))
    Ro, delay, cp = _rect_inputs(c, seed)
    return dict(c, Ro=_fortran(Ro, torch.float64), delay=delay, cp=cp, G=_array_grid(c) if kind == "arr" else None)


def run(state):
    s, kind = state, state["kind"]
    if kind == "das":
        f = s["f"]
        fn = das64.das if s["precision"] == "f64" else das32.das
        return fn(f["Y"], f["Gt"], f["Gr"], f["Ro"], f["dt"], f["delay"], f["cp"], s["method"], "ignore", "cuda")
    if kind == "mixed":
        f = s["f"]
        return das_mixed(f["Y"], f["Gt"], f["Gr"], f["Ro"], f["dt"], f["delay"], f["cp"], s["method"], "ignore",
                         "cuda", storage=s["storage"])
    if kind == "grad":
        im = das_gather(s["Y"], s["w"], s["op"])
        gY, gw = torch.autograd.grad(im, (s["Y"], s["w"]), s["g"])
        return [im.detach(), gY, gw]
    if kind == "cg":
        return list(cg_reconstruct(s["op"], s["Y"], s["w"], lam=1e-3, iters=s["iters"]))
    if kind == "batch":
        s["batch"].run()
        return s["images"]
    if kind == "fmc":
        return fmc_synthesis(s["H"], s["p"])
    s_par, m_par = [s["d"], s["d"], s["dt"], s["nt"]], [1.0, s["cp"], 0.0]
    if kind == "rect":
        return dreamrect(s["Ro"], [s["a"], s["b"]], s_par, s["delay"], m_par, "ignore")
    return dream_arr_rect(s["Ro"], [s["size"], s["size"]], s["G"], s_par, s["delay"], m_par, "xy", 50.0, "x",
                          [-25.0, 0.0], "off", np.ones(len(s["G"])), 1.0, "ignore")


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        per = [work(dict(kind="mixed", storage="f32", method="tfm", nt=s["n_el"], nr=s["n_el"], K=s["K"], nx=s["side"],
                         ny=1, nz=s["side"])) for s in _batch_specs(c)]
        return {k: sum(p[k] for p in per) for k in ("bytes", "flops")}
    if kind == "fmc":
        n, m1, m2 = c["lt"] ** 2, 2 * c["M"] - 1, 2 * c["M"] + c["pulse"] - 2
        return {"bytes": 8 * (c["M"] * c["lt"] + c["pulse"] + n * m2),
                "flops": 2.0 * n * (c["M"] ** 2 + m1 * c["pulse"])}
    if kind in ("rect", "arr"):
        side_a, side_b = (c["a"], c["b"]) if kind == "rect" else (c["size"], c["size"])
        terms = len(_centres(side_a, c["d"])) * len(_centres(side_b, c["d"])) * (c["side"] ** 2 if kind == "arr" else 1)
        n = c["nx"] * c.get("ny", 1) * c["nz"]
        # an array's short window keeps few elements per point: its terms in the window are what cannot be left out
        share = 0.05 if kind == "arr" else 1.0
        return {"bytes": 8 * n * (3 + c["nt"]), "flops": 15.0 * n * terms * share}
    n = c["nx"] * c.get("ny", 1) * c["nz"]
    cols = c["nt"] if c.get("method") == "saft" else c["nt"] * c["nr"]
    size = 8 if c.get("precision") == "f64" else 4
    one = {"bytes": cols * c["K"] * size + 4 * n * size, "flops": 3.0 * n * cols}  # two legs, scale, accumulate
    if kind == "grad":
        return {"bytes": 2 * one["bytes"] + cols * c["K"] * 4, "flops": 2 * one["flops"]}
    if kind == "cg":
        return {k: (2 * c["iters"] + 1) * v for k, v in one.items()}
    return one


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _index_blocks(f, method, dtype, block=1 << 27):
    """Yields (points, first column, sample index (points, columns), in-bounds mask) of every term, the index
    computed in `dtype` with the operations of the beamformer, unfused. The columns follow the A-scans."""
    T = lambda a: torch.as_tensor(np.asarray(a), device=DEV).to(dtype)
    Gt, Gr, Ro, delay = (T(f[k]) for k in ("Gt", "Gr", "Ro", "delay"))
    num = lambda v: torch.tensor(v, dtype=dtype, device=DEV)
    rnd = (lambda v: float(np.float32(v))) if dtype == torch.float32 else float
    dt, cp, K = rnd(f["dt"]), rnd(f["cp"]), f["Y"].shape[0]
    Fs, ocp = num((1.0 / dt) * 1000.0), num(1.0 / cp)
    d_ms = (delay.double() / 1000.0).to(dtype).reshape(-1)
    No, nt, nr = Ro.shape[0], Gt.shape[0], Gr.shape[0]
    n_out, n_in = (1, nt) if method == "saft" else ((nr, nt) if method == "rca_rowtx" else (nt, nr))
    step = max(1, block // n_in)
    for n0 in range(0, No, step):
        sl = slice(n0, min(No, n0 + step))
        P, d = Ro[sl], (d_ms[sl] if d_ms.numel() > 1 else d_ms)
        tx, rx = _leg_parts(Gt, Gr, P, method)
        t_leg = torch.stack([_leg(tx(e), ocp) + d for e in range(nt)], 1)
        if method == "saft":
            legs = [None]
            inner = 2.0 * t_leg
        elif method == "rca_rowtx":
            legs, inner = [_leg(rx(e), ocp) for e in range(nr)], t_leg
        else:
            legs, inner = [t_leg[:, e] for e in range(nt)], torch.stack([_leg(rx(e), ocp) for e in range(nr)], 1)
        for o in range(n_out):
            p = (inner if legs[o] is None else legs[o][:, None] + inner) * Fs
            ok = (p > -1.0) & (p < K)
            k = torch.where(ok, p, torch.zeros_like(p)).long()
            yield sl, o * n_in, k, ok


def _image(f, method, dtype, samples, w=None):
    """sum over the terms of w * samples[k, column] in FP64."""
    Yc = samples.t().contiguous()  # (columns, K)
    K = Yc.shape[1]
    im = torch.zeros(np.asarray(f["Ro"]).shape[0], dtype=torch.float64, device=DEV)
    for sl, c0, k, ok in _index_blocks(f, method, dtype):
        n = k.shape[1]
        v = Yc.view(-1)[k + (torch.arange(n, device=DEV) + c0) * K].double()
        v = torch.where(ok, v, torch.zeros_like(v))
        im[sl] += (v @ w[c0:c0 + n] if w is not None else v.sum(1))
    return im


def _scatter(f, method, x):
    """DAS^T x, (columns, K) in FP64."""
    C, K = f["Y"].shape[1], f["Y"].shape[0]
    S = torch.zeros(C * K, dtype=torch.float64, device=DEV)
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    for sl, c0, k, ok in _index_blocks(f, method, torch.float64):
        n = k.shape[1]
        S.index_add_(0, (k + (torch.arange(n, device=DEV) + c0) * K).reshape(-1),
                     torch.where(ok, x[sl][:, None].expand(-1, n), zero).reshape(-1))
    return S.view(C, K)


def _sir(Ro, delay, cp, c, G, el_delay):
    """Spatial impulse responses (nt, points) in FP64, one array element and a block of points at a time."""
    num = lambda v: torch.tensor(v, dtype=torch.float64, device=DEV)
    a, b = (c["a"], c["b"]) if c["kind"] == "rect" else (c["size"], c["size"])
    xs, ys = num(_centres(a, c["d"])), num(_centres(b, c["d"]))
    nt, dt, P = c["nt"], c["dt"], num(Ro)
    H = torch.zeros((P.shape[0], nt), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 26) // (len(xs) * len(ys)))
    for n0 in range(0, P.shape[0], step):
        Hb, nb = H[n0:n0 + step], min(step, P.shape[0] - n0)
        row = (torch.arange(nb, device=DEV) * nt)[:, None, None]
        for m in range(len(G)):
            x, y, z = (P[n0:n0 + step, k] - float(G[m][k]) for k in range(3))
            rx, ry = x[:, None] - xs, y[:, None] - ys
            r = torch.sqrt((rx * rx)[:, None, :] + (ry * ry)[:, :, None] + (z * z)[:, None, None])
            it = torch.round((r * 1000.0 / cp - (delay - float(el_delay[m]))) / dt)
            ok = (it >= 0) & (it < nt)
            if c["kind"] == "arr":  # few terms fall in the window
                sel = ok.nonzero(as_tuple=True)
                r, it, ok = r[sel], it[sel], None
                at = sel[0] * nt + it.long()
            else:
                at = row + torch.where(ok, it, torch.zeros_like(it)).long()
            v = c["d"] * c["d"] / (2.0 * math.pi * r) / dt * 1000.0
            v = v if ok is None else torch.where(ok, v, torch.zeros_like(v))
            Hb.view(-1).index_add_(0, at.reshape(-1), v.reshape(-1))
    return H.t()


def _convolve(A, B, n):
    """Full convolution of the rows of A and B, n samples."""
    m = 1 << (n - 1).bit_length()
    return torch.fft.irfft(torch.fft.rfft(A, m) * torch.fft.rfft(B, m), m)[..., :n]


def exact(case, seed):
    c, kind = dict(case), case["kind"]
    if kind in ("das", "mixed"):
        f = _frame(c, seed)
        dtype = torch.float32 if c.get("precision") == "f32" else torch.float64
        im = _image(f, c["method"], dtype, f["Y"])
        return im.cpu().numpy() if c.get("host") else im
    if kind == "grad":
        f = _frame(c, seed)
        w = _weights(f["Y"].shape[1], seed).double()
        g = torch.randn(f["Ro"].shape[0], generator=_generator(seed, 3), device=DEV).double()
        S = _scatter(f, "tfm", g)
        return [_image(f, "tfm", torch.float64, f["Y"], w), (S * w[:, None]).t(), (S * f["Y"].t()).sum(1)]
    if kind == "cg":
        f = _frame(dict(c, method="tfm"), seed)
        w = _weights(f["Y"].shape[1], seed).double()
        fwd = lambda Y: _image(f, "tfm", torch.float64, Y, w)
        A = lambda p: fwd((_scatter(f, "tfm", p) * w[:, None]).t()) + 1e-3 * p
        b = fwd(f["Y"].double())
        x, r, p, hist = torch.zeros_like(b), b.clone(), b.clone(), []
        rs = r @ r
        for _ in range(c["iters"]):
            Ap = A(p)
            alpha = rs / (p @ Ap)
            x, r = x + alpha * p, r - alpha * Ap
            rs, old = r @ r, rs
            p = r + (rs / old) * p
            hist.append(rs.sqrt())
        return [x, torch.stack(hist)]
    if kind == "batch":
        return [_image(f, "tfm", torch.float64, f["Y"]) for f in _batch_frames(c, seed)]
    if kind == "fmc":
        H, p = _synthesis_inputs(c, seed)
        H, p = torch.from_numpy(H.T.copy()).to(DEV), torch.from_numpy(p).to(DEV)
        n1 = 2 * c["M"] - 1
        return torch.cat([_convolve(_convolve(H, H[t], n1), p, n1 + c["pulse"] - 1) for t in range(c["lt"])]).t()
    Ro, delay, cp = _rect_inputs(c, seed)
    if kind == "rect":
        return _sir(Ro, delay, cp, c, [(0.0, 0.0, 0.0)], [0.0])
    G = _array_grid(c)
    r_max = math.hypot(np.abs(G[:, 0]).max(), np.abs(G[:, 1]).max())
    foc = (math.sqrt(r_max ** 2 + 2500.0) - np.sqrt(G[:, 0] ** 2 + G[:, 1] ** 2 + 2500.0)) * 1e3 / cp
    steer = (np.abs(G[:, 0]).max() + G[:, 0]) * math.sin(-25.0 * math.pi / 180.0) * 1e3 / cp
    return _sir(Ro, delay, cp, c, G, foc + steer)
