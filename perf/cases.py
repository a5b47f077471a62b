"""The work this package is measured on: simulations, and simulations with gradients, through its public entry points.

Four calls are covered:

* ``simulate``: ``blochparty_b200.simulate`` from host tensors to host results, packing and copies included;
* ``gradient``: the same call with inputs that require grad, and the vector-Jacobian product of its outputs;
* ``resident``: a packed case held on the GPU (``engine.pack``, ``plan_windows``), one forward of it
  (``run_forward``, ``finish_signal``): a program that steps many times through one packed case;
* ``resident_gradient``: the same with ``adjoint.Checkpointed``, forward and backward, for the RF waveform's gradient
  (a flip-train optimisation).

Sequences: 2D and 3D spoiled Cartesian GRE with hard pulses and dummy scans, slab-selective 3D GRE (200-step sinc,
one or four echoes), and multi-slice TSE (300-step sincs). Phantoms are seeded maps of a few tissues with smooth
B0 and B1+ fields; positions and maps are float32 values held as float64, so that what a result is off by is the
engine's own error and not the rounding of its inputs.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import blochparty_b200 as bpb
from blochparty_b200 import _lib, adjoint, engine, sequences

F64, C128 = torch.float64, torch.complex128
FOV = 0.25
TWO_PI = 2.0 * math.pi
# (T1, T2, PD): fat, white matter, grey matter, CSF
TISSUES = ((0.3, 0.08, 0.9), (0.8, 0.07, 0.8), (1.3, 0.09, 0.7), (4.0, 2.0, 1.0))


def listed():
    return [
        # the smallest call: a sequence tried out on a coarse grid, where launches and host work count
        dict(name="gre2d_16", call="simulate", seq="gre2d", n=16, spv=1, coils=4, lines=16, dummies=5),
        # an ordinary 2D scan: 64 x 64, 8 coils, 200 dummy TRs to the steady state
        dict(name="gre2d_64", call="simulate", seq="gre2d", n=64, spv=1, coils=8, lines=64, dummies=200),
        # ragged sizes: 95 x 95 spins and samples, 13 coils, B0 and B1+ maps, a starting magnetization
        dict(name="gre2d_95_13coils", call="simulate", seq="gre2d", n=95, spv=1, coils=13, lines=95, dummies=20,
             m_init=True),
        # an ordinary 3D scan on an odd grid: 29,791 spins, 31 x 31 lines of 31 samples, 200 dummy TRs
        dict(name="gre3d_31", call="simulate", seq="gre3d", n=31, spv=1, coils=8, lines=961, dummies=200),
        # a multi-slice TSE: nearly all RF steps, 393,216 spins through the slices
        dict(name="tse_128", call="simulate", seq="tse", n=128, spv=8, coils=8, lines=8, dummies=0),
        # a slab-selective 3D GRE of 1,048,576 spins, its first 24 TRs, held on the GPU
        dict(name="gre3d_64_resident", call="resident", seq="slab", n=64, spv=4, coils=8, lines=24, dummies=0),
        # the largest: a 4-echo 3D GRE of 128^3 x 4 = 8,388,608 spins, its first 8 TRs, held on the GPU
        dict(name="head_128_resident", call="resident", seq="echoes", n=128, spv=4, coils=8, lines=8, dummies=0),
        # the same scan at 64^3 x 4 spins as one whole call from host tensors
        dict(name="head_64", call="simulate", seq="echoes", n=64, spv=4, coils=8, lines=8, dummies=0),
        # ... with its readouts through the nonuniform FFT, at 48^3 x 4 spins
        dict(name="head_48_nufft", call="simulate", seq="echoes", n=48, spv=4, coils=8, lines=16, dummies=0,
             readout="nufft"),
        # a flip-train fit of one whole call: 128 x 128, 8 coils, gradients of the RF waveform and the T1 map
        dict(name="gre2d_128_fit", call="gradient", seq="gre2d", n=128, spv=1, coils=8, lines=128, dummies=0,
             wrt="t1 rf"),
        # a map fit of one whole call: every tissue map, B1+ and the coils of a small 3D GRE
        dict(name="gre3d_24_maps", call="gradient", seq="gre3d", n=24, spv=1, coils=8, lines=64, dummies=40,
             wrt="pd t1 t2 db0 b1 coils"),
        # a flip-train optimisation held on the GPU: the 4-echo scan at 64^3 x 4 spins, its first 8 TRs
        dict(name="head_64_flips", call="resident_gradient", seq="echoes", n=64, spv=4, coils=8, lines=8, dummies=0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("gre2d", "gre2d", "gre3d", "tse", "slab", "echoes", "echoes", "fit", "maps", "flips", "nufft"))
    coils = rng.choice((1, 2, 4, 7, 8, 8, 8, 12, 13, 16))
    if kind == "gre2d":
        n = log_int(12, 160)
        return dict(call="simulate", seq="gre2d", n=n, spv=1, coils=coils, lines=rng.randint(max(1, n // 2), n),
                    dummies=rng.randint(0, 200), m_init=rng.random() < 0.3)
    if kind == "gre3d":
        n = rng.randint(10, 40)
        return dict(call="simulate", seq="gre3d", n=n, spv=1, coils=coils, lines=rng.randint(n, n * n),
                    dummies=rng.randint(0, 200))
    if kind == "tse":
        return dict(call="simulate", seq="tse", n=rng.choice((64, 80, 96, 128)), spv=rng.randint(1, 8), coils=coils,
                    lines=rng.randint(1, 4), dummies=0)
    if kind == "fit":
        n = log_int(24, 128)
        return dict(call="gradient", seq="gre2d", n=n, spv=1, coils=min(coils, 8), lines=rng.randint(n // 2, n),
                    dummies=0, wrt=rng.choice(("rf", "t1 rf", "t1 t2", "pd t1 t2 rf")))
    if kind == "maps":
        return dict(call="gradient", seq="gre3d", n=rng.randint(10, 28), spv=1, coils=min(coils, 8),
                    lines=rng.randint(10, 64), dummies=rng.randint(0, 60), wrt="pd t1 t2 db0 b1 coils")
    if kind == "nufft":
        return dict(call="simulate", seq="echoes", n=rng.choice((40, 48, 56, 64)), spv=4, coils=min(coils, 16),
                    lines=rng.randint(2, 16), dummies=0, readout="nufft")
    seq = "slab" if kind == "slab" else "echoes"
    call = rng.choice(("resident", "resident", "simulate")) if kind != "flips" else "resident_gradient"
    n = log_int(20, 100) if call == "resident" else log_int(20, 64)
    return dict(call=call, seq=seq, n=n, spv=rng.randint(1, 4), coils=coils if call != "resident_gradient" else 8,
                lines=rng.randint(2, 8), dummies=0)


# ---------------------------------------------------------------- inputs


def _shape(case):
    """(grid axes, dimensions of the grid) of the phantom."""
    return (2, case["n"]) if case["seq"] in ("gre2d", "tse") else (3, case["n"])


def _phantom(case, seed):
    """Positions (N, 3), PD, T1, T2, dB0, B1 on the GPU, float64 holding float32 values."""
    g = torch.Generator(device="cuda").manual_seed(1000 + seed)
    rnd = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=F64)
    dims, n = _shape(case)
    ax = (torch.arange(n, device="cuda", dtype=F64) - n // 2) * (FOV / n)
    vox = torch.stack(list(reversed(torch.meshgrid(*[ax] * dims, indexing="ij"))), -1).reshape(-1, dims)
    u = vox / (0.5 * FOV)
    label = torch.zeros(vox.shape[0], dtype=torch.long, device="cuda")  # 0: outside, PD 0
    for k, r in ((1, 0.9), (3, 0.8), (2, 0.62)):  # scalp, grey matter, white matter: nested
        label[((u / (r * (0.85 + 0.2 * rnd(dims)))) ** 2).sum(-1) <= 1.0] = k
    for k in (4, 4, 3, 2):  # ventricles, nuclei, lesions
        c, a = (rnd(dims) - 0.5) * 0.9, 0.08 + 0.25 * rnd(dims)
        label[(((u - c) / a) ** 2).sum(-1) <= 1.0] = k
    table = torch.tensor(((1.0, 0.1, 0.0),) + TISSUES, device="cuda", dtype=F64)
    table[1:] *= 0.9 + 0.2 * rnd(4, 3)
    db0, b1 = torch.zeros_like(vox[:, 0]), torch.ones_like(vox[:, 0])
    for field, amp in ((db0, 60.0), (b1, 0.07)):  # smooth: three low spatial frequencies
        for _ in range(3):
            field += amp * (2 * float(rnd(1)) - 1) * torch.cos(u @ (3.0 * (rnd(dims) - 0.5)) + 6.0 * float(rnd(1)))
    s = case["spv"]
    rep = lambda t: t.repeat_interleave(s, 0)
    pos = torch.zeros(vox.shape[0] * s, 3, device="cuda", dtype=F64)
    pos[:, :dims] = rep(vox)
    maps = [rep(table[label, 2]), rep(table[label, 0]), rep(table[label, 1]), rep(db0), rep(b1)]
    if case["seq"] == "tse":  # three 5 mm slices, the spins of a voxel spread through the thickness
        pos[:, 2] = (torch.arange(s, device="cuda", dtype=F64).add(0.5).div(s).sub(0.5) * 5e-3).repeat(vox.shape[0])
        pos = torch.cat([pos + torch.tensor((0.0, 0.0, z), device="cuda", dtype=F64) for z in (-5e-3, 0.0, 5e-3)])
        maps = [m.repeat(3) for m in maps]
    elif s > 1:
        pos += (rnd(pos.shape[0], 3) - 0.5) * (FOV / n)
    return [t.float().to(F64) for t in (pos, *maps)]


def _sequence(case, seed):
    r = np.random.RandomState(seed)
    n, lines, dummies = case["n"], case["lines"], case["dummies"]
    if case["seq"] == "tse":  # the slices' pulses differ from seed to seed in the flip angles
        return sequences.tse_2d(n, FOV, slices=(-5e-3, 0.0, 5e-3), slice_thickness=5e-3, etl=16, esp=12e-3, tr=3.0,
                                rf_duration=3e-3, rf_steps=300, n_shots=min(lines, max(1, n // 16)),
                                excite_flip_deg=float(r.uniform(85, 95)), refocus_flip_deg=float(r.uniform(150, 180)))
    flips = r.uniform(8.0, 22.0, size=dummies + lines)
    if case["seq"] in ("gre2d", "gre3d"):
        te = 20e-6 + 0.5e-3 + (n // 2 + 0.5) * 10e-6
        kw = dict(tr=te + n * 10e-6 + 3e-3, te=te, rf="hard", rf_duration=20e-6, rf_steps=1)
        shape = (lines, n) if case["seq"] == "gre2d" else (-(-lines // n), n, n)
    else:
        esp = (n + 132) * 10e-6
        te = 1e-3 + 1e-3 + (n // 2 + 0.5) * 10e-6
        echoes = 4 if case["seq"] == "echoes" else 1
        kw = dict(tr=te + echoes * esp + 5e-3, te=te, rf="sinc", rf_duration=2e-3, rf_steps=200, slab_thickness=0.2,
                  n_echoes=echoes, echo_spacing=esp)
        shape = (1, lines, n)
    keep = dummies + lines
    total = dummies + int(np.prod(shape[:-1]))
    seq = sequences.gre(shape, FOV, flip_deg=np.resize(flips, total), n_dummy=dummies, dwell=10e-6, **kw)
    if total > keep:  # a 3D scan stopped after `lines` lines: whole TRs
        rf = np.asarray(seq.is_rf)
        cut = int(np.flatnonzero(rf & ~np.concatenate([[False], rf[:-1]]))[keep])
        seq = bpb.Sequence(seq.dt[:cut], seq.rf[:cut], seq.grad[:cut], seq.adc_phase[:cut], seq.is_rf[:cut],
                           seq.adc[:cut], seq.spoil[:cut])
    return seq


def _inputs(case, seed):
    """(phantom maps on the GPU, coils, m_init, sequence)."""
    maps = _phantom(case, seed)
    pos = maps[0]
    theta = TWO_PI * torch.arange(case["coils"], device="cuda", dtype=F64) / case["coils"]  # on a circle around z
    dx, dy = pos[:, :1] - 0.18 * torch.cos(theta), pos[:, 1:2] - 0.18 * torch.sin(theta)
    coils = torch.polar(0.18 / torch.sqrt(dx * dx + dy * dy).clamp_min(9e-3), torch.atan2(dy, dx) - theta)
    coils = coils.to(torch.complex64).to(C128)
    m0 = None
    if case.get("m_init"):
        g = torch.Generator(device="cuda").manual_seed(2000 + seed)
        m0 = (0.3 * maps[1][:, None] * torch.randn(pos.shape[0], 3, generator=g, device="cuda", dtype=F64)).float().to(F64)
    return maps, coils, m0, _sequence(case, seed)


def _cotangents(case, n, n_adc, seed, like=torch.float32):
    """Seeded dL/dsignal (C, A) and dL/dm (N, 3), of a size that lets both matter."""
    g = torch.Generator(device="cuda").manual_seed(3000 + seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float32)
    return torch.complex(rnd(case["coils"], n_adc), rnd(case["coils"], n_adc)), math.sqrt(n_adc) * rnd(n, 3)


def prepare(case, seed):
    maps, coils, m0, seq = _inputs(case, seed)
    call = case["call"]
    if call in ("resident", "resident_gradient"):
        dev = torch.device("cuda", torch.cuda.current_device())
        pos, pd, t1, t2, db0, b1 = maps
        inp = bpb.api.Inputs(pos, pd, t1, t2, db0, b1, coils, seq.dt, seq.rf, seq.grad, seq.adc_phase, None,
                             list(seq.is_rf), list(seq.adc), list(seq.spoil), m0)
        pk = engine.pack(inp, dev)
        s = dict(case=case, pk=pk, state0=engine.initial_state(pd, m0, dev))
        s["state"] = torch.empty_like(s["state0"])
        if call == "resident":
            windows = engine.plan_windows(pk.flags, _lib.lib().bp_forward_samp_max(pk.n_coils))
            s.update(windows=torch.from_numpy(windows).to(dev), n_windows=windows.shape[0],
                     raw=torch.zeros(max(pk.n_adc, 1), 2 * pk.n_coils, dtype=F64, device=dev),
                     status=torch.zeros(1, dtype=torch.int32, device=dev))
        else:
            every, outer = adjoint.choose_checkpoints(len(seq), pk.n)
            s["run"] = adjoint.Checkpointed(pk, every, dev, outer, saved=True)
            s["h"] = torch.view_as_real(_cotangents(case, 1, pk.n_adc, seed)[0].T.contiguous()).reshape(pk.n_adc, -1)
            s["lam"] = torch.empty(3, pk.n, device=dev)
            s["w"] = (-TWO_PI * seq.dt).to(dev)[:, None]
        return s
    host = [t.cpu() for t in maps]
    s = dict(case=case, seq=seq, coils=coils.cpu(), m0=None if m0 is None else m0.cpu())
    s["ph"] = bpb.Phantom(host[0], *host[1:5], b1=host[5])
    if call == "gradient":
        n_adc = int(sum(seq.adc))
        g_sig, g_m = _cotangents(case, len(host[1]), n_adc, seed)
        s["cotangents"] = [g_sig.cpu(), g_m.cpu()]
    return s


def run(s):
    case = s["case"]
    call = case["call"]
    if call == "simulate":
        with torch.no_grad():
            r = bpb.simulate(s["ph"], s["seq"], s["coils"], m_init=s["m0"], readout=case.get("readout", "fp32"))
        return {"signal": r.signal, "m": r.m}
    if call == "gradient":
        ph, seq, coils = s["ph"], s["seq"], s["coils"]
        leaves = {}
        for k in case["wrt"].split():
            src = seq.rf if k == "rf" else coils if k == "coils" else getattr(ph, k)
            leaves[k] = src.detach().requires_grad_()
        lf = lambda k: leaves.get(k, getattr(ph, k))
        ph = bpb.Phantom(ph.pos, lf("pd"), lf("t1"), lf("t2"), lf("db0"), b1=lf("b1"))
        seq = bpb.Sequence(seq.dt, leaves.get("rf", seq.rf), seq.grad, seq.adc_phase, seq.is_rf, seq.adc, seq.spoil)
        r = bpb.simulate(ph, seq, leaves.get("coils", coils), m_init=s["m0"])
        grads = torch.autograd.grad([r.signal, r.m], list(leaves.values()), s["cotangents"])
        return {"signal": r.signal.detach(), "m": r.m.detach(), **{"d_" + k: g for k, g in zip(leaves, grads)}}
    pk = s["pk"]
    s["state"].copy_(s["state0"])
    if call == "resident":
        s["raw"].zero_()
        engine.run_forward(pk, s["state"], s["windows"], 0, s["n_windows"], s["raw"], s["status"])
        return {"signal": engine.finish_signal(pk, s["raw"]), "m": s["state"][0:3] + s["state"][3:6]}
    ck = s["run"]
    ck.forward(s["state"])
    sig = engine.finish_signal(pk, ck.raw)
    s["lam"].zero_()
    _, _, seg = ck.backward(s["h"], s["lam"], _lib.BP_SEG_WX | _lib.BP_SEG_WY | _lib.BP_SPIN_NO_OFFSETS
                            | _lib.BP_SPIN_NONE, False, True)
    return {"signal": sig, "m": s["state"][0:3] + s["state"][3:6], "d_rf": seg[:, 1:3] * s["w"], "d_m0": s["lam"]}


# ---------------------------------------------------------------- the work, and how close results have to be


def _counts(case):
    """(spins, segments, RF segments, samples, free segments that differ from the one before)."""
    n, seq = case["n"], case["seq"]
    spins = n ** _shape(case)[0] * case["spv"] * (3 if seq == "tse" else 1)
    trs = case["lines"] + case["dummies"]
    if seq == "tse":
        shots = 3 * min(case["lines"], max(1, n // 16))
        return spins, shots * (300 + 2 + 16 * (300 + 3 + n)), shots * 17 * 300, shots * 16 * n, shots * (2 + 16 * 4)
    if seq in ("gre2d", "gre3d"):
        return spins, trs * (n + 5), trs, case["lines"] * n, trs * 6
    e = 4 if seq == "echoes" else 1
    return spins, trs * (200 + 2 + e * (n + 2)), trs * 200, trs * e * n, trs * (3 + 4 * e)


def work(case):
    """Every input read once, every result written once. Flops of the forward: a rotation with its relaxation in
    every RF segment (61), a new precession and relaxation per distinct free segment (34), one complex step (8) and
    a complex product per coil (8) for every sample; readouts through the nonuniform FFT spread 27 weights per run
    instead. A reverse sweep: the states again, then 103 per RF segment, 9 per free one and 8 per sample and coil;
    with gradients of the maps 130, 30, and 16 with the coils'."""
    spins, segs, n_rf, n_adc, n_free = _counts(case)
    c = case["coils"]
    bytes_ = spins * (4 * 8 + 8 * c + 4 * 3) + segs * 44 + n_adc * c * 8
    per_spin = 61 * n_rf + 34 * n_free + n_adc * (8 + 8 * c)
    if case.get("readout") == "nufft":
        per_spin = 61 * n_rf + 34 * n_free + n_adc / case["n"] * (48 + 27 * (8 + 8 * c))
    if "gradient" in case["call"]:
        wrt = case.get("wrt", "rf").split()
        maps = any(k != "rf" for k in wrt)
        per_spin += (61 + (130 if maps else 103)) * n_rf + (30 if maps else 9) * (n_free + n_adc)
        per_spin += n_adc * c * (16 if "coils" in wrt else 8)
        bytes_ += n_adc * c * 8 + spins * 4 * 3 + spins * 4 * len([k for k in wrt if k not in ("rf", "coils")])
        bytes_ += (spins * c * 8 if "coils" in wrt else 0) + (segs * 8 if "rf" in wrt else 0)
    return {"bytes": float(bytes_), "flops": float(spins * per_spin)}


def tolerance(case):
    """About four times the distance from 64 bits: the state is float32 with compensation, and what remains are the
    float32 increments of the RF steps: 2e-6 over a few slab pulses, 9e-6 over a TSE's trains of 300-step pulses; in
    gradients the float32 states of the reverse sweep, 1.3e-4 in the RF waveform's."""
    if "gradient" in case["call"]:
        return {"rel": 5e-4}
    return {"rel": 4e-5} if case["seq"] == "tse" else {"rel": 1e-5}


# ---------------------------------------------------------------- the same in 64 bits


def _rf_step(m, s, sq, sp):
    """One RF segment (Strang): relax dt/2, rotate about -2 pi dt (b1 rf, offset), relax dt/2."""
    mx, my, mz = m
    dt, rfx, rfy, g = sq["dt"][s], sq["rfx"][s], sq["rfy"][s], sq["grad"][s]
    w = -TWO_PI * dt
    if sp["cache"].get("key") != (dt, g):  # what the steps of one pulse share
        sp["cache"] = dict(key=(dt, g), e=(torch.exp(-0.5 * dt * sp["r1"]), torch.exp(-0.5 * dt * sp["r2"])),
                           wz=w * (sp["pos"][0] * g[0] + sp["pos"][1] * g[1] + sp["pos"][2] * g[2] + sp["db0"]))
    e1, e2 = sp["cache"]["e"]
    wx, wy, wz = w * rfx * sp["b1"], w * rfy * sp["b1"], sp["cache"]["wz"]
    mx, my, mz = mx * e2, my * e2, sp["pd"] + (mz - sp["pd"]) * e1
    phi = torch.sqrt(wx * wx + wy * wy + wz * wz + 1e-30)
    c, s1, s2 = torch.cos(phi), torch.sin(phi) / phi, 2.0 * (torch.sin(0.5 * phi) / phi) ** 2
    k = s2 * (wx * mx + wy * my + wz * mz)
    nx = c * mx + s1 * (wy * mz - wz * my) + k * wx
    ny = c * my + s1 * (wz * mx - wx * mz) + k * wy
    nz = c * mz + s1 * (wx * my - wy * mx) + k * wz
    return nx * e2, ny * e2, sp["pd"] + (nz - sp["pd"]) * e1


def _sim64(sp, coils, sq, m, reuse):
    """(raw coil sums (C, A), m) of the sequence ``sq`` from ``m``; ``reuse``: recurring pulses composed once into
    their affine maps (the same arithmetic, for the long pulses of a TSE)."""
    is_rf, adc, spoil = sq["is_rf"], sq["adc"], sq["spoil"]
    S, s, cols, maps = len(is_rf), 0, [], {}
    zero = torch.zeros_like(sp["pd"])
    while s < S:
        if is_rf[s]:
            e = s + 1
            while e < S and is_rf[e] and not spoil[e - 1]:
                e += 1
            if reuse and e - s > 16:
                key = sq["bytes"](s, e)
                if key not in maps:
                    basis = [(zero, zero, zero)] + [tuple(zero + (i == j) for j in range(3)) for i in range(3)]
                    outs = []
                    for b in basis:
                        for q in range(s, e):
                            b = _rf_step(b, q, sq, sp)
                        outs.append(b)
                    maps[key] = outs
                o, *cl = maps[key]
                m = tuple(o[i] + sum((cl[j][i] - o[i]) * m[j] for j in range(3)) for i in range(3))
            else:
                for q in range(s, e):
                    m = _rf_step(m, q, sq, sp)
        else:
            e = s + 1
            while e < S and not is_rf[e] and not spoil[e - 1]:
                e += 1
            t = np.cumsum(sq["dt_np"][s:e])
            k = np.cumsum(sq["grad_np"][s:e] * sq["dt_np"][s:e, None], 0)
            tt, kk = torch.from_numpy(t).cuda(), torch.from_numpy(k).cuda()
            idx = np.flatnonzero(adc[s:e])
            z = torch.complex(m[0], m[1])
            if idx.size:
                ii = torch.from_numpy(idx).cuda()
                part, step = 0, max(1, (1 << 26) // idx.size)
                for a in range(0, z.shape[0], step):
                    sl = slice(a, a + step)
                    cyc = torch.stack([p[sl] for p in sp["pos"]], -1) @ kk[ii].T + sp["db0"][sl, None] * tt[ii]
                    w = torch.exp(torch.complex(-tt[ii] * sp["r2"][sl, None], -TWO_PI * (cyc - torch.round(cyc.detach()))))
                    part = part + (z[sl, None] * coils[sl]).T @ w
                cols.append(part)
            cyc = sp["pos"][0] * kk[-1, 0] + sp["pos"][1] * kk[-1, 1] + sp["pos"][2] * kk[-1, 2] + sp["db0"] * tt[-1]
            z = z * torch.exp(torch.complex(-tt[-1] * sp["r2"], -TWO_PI * (cyc - torch.round(cyc.detach()))))
            m = (z.real, z.imag, sp["pd"] + (m[2] - sp["pd"]) * torch.exp(-tt[-1] * sp["r1"]))
        if spoil[e - 1]:
            m = (zero, zero, m[2])
        s = e
    sig = torch.cat(cols, 1) if cols else torch.zeros(coils.shape[1], 0, dtype=C128, device="cuda")
    return sig, m


def exact(case, seed):
    spins, segs, n_rf, n_adc, _ = _counts(case)
    grad = "gradient" in case["call"]
    # gradients by autograd over blocks of spins (the loss is linear in the signal and in m, so they add up)
    block = spins if not grad else max(1, int(60e9 / (450.0 * n_rf + 150.0 * n_adc + 100.0 * segs)))
    if grad and -(-spins // block) * (n_rf + n_adc / 64) > 12000:
        return None
    maps, coils, m0, seq = _inputs(case, seed)
    wrt = case.get("wrt", "rf").split() if grad else []
    rf = seq.rf.cuda().requires_grad_("rf" in wrt)
    rf_rows = np.flatnonzero(np.asarray(seq.is_rf))
    psi = seq.adc_phase[torch.from_numpy(np.flatnonzero(np.asarray(seq.adc)))].cuda()
    turn = torch.exp(torch.complex(torch.zeros_like(psi), -psi))
    g_sig, g_m = _cotangents(case, spins, psi.shape[0], seed) if case["call"] == "gradient" else (None, None)
    h = _cotangents(case, 1, psi.shape[0], seed)[0].to(C128) if case["call"] == "resident_gradient" else None
    rec = np.concatenate([seq.dt.numpy()[:, None], seq.rf.numpy(), seq.grad.numpy()], 1)
    raw, ms, grads = 0, [], {k: [] for k in wrt + ["m0"]}
    for a in range(0, spins, block):
        got = rf[torch.from_numpy(rf_rows).cuda()]
        vx, vy = (got[:, i].unbind(0) if "rf" in wrt else got[:, i].tolist() for i in (0, 1))
        sq = dict(dt=seq.dt.tolist(), grad=[tuple(g) for g in seq.grad.tolist()], dt_np=seq.dt.numpy(),
                  grad_np=seq.grad.numpy(), is_rf=np.asarray(seq.is_rf), adc=np.asarray(seq.adc),
                  spoil=np.asarray(seq.spoil), rfx=dict(zip(rf_rows.tolist(), vx)),
                  rfy=dict(zip(rf_rows.tolist(), vy)), bytes=lambda i, j: rec[i:j].tobytes())
        sl = slice(a, a + block)
        part = dict(zip(("pos", "pd", "t1", "t2", "db0", "b1"), (t[sl] for t in maps)), coils=coils[sl])
        for k in wrt:
            if k != "rf":
                part[k] = part[k].detach().requires_grad_()
        sp = dict(pos=part["pos"].unbind(-1), pd=part["pd"], r1=1.0 / part["t1"], r2=1.0 / part["t2"],
                  db0=part["db0"], b1=part["b1"], cache={})
        z = torch.zeros_like(part["pd"])
        start = torch.stack([z, z, part["pd"]]) if m0 is None else m0[sl].T
        if h is not None:
            start = start.detach().requires_grad_()
        with torch.set_grad_enabled(grad):
            r, m = _sim64(sp, part["coils"], sq, start.unbind(0), reuse=not grad)
            m = torch.stack(m)
            sig = r * turn
        raw = raw + r.detach()
        ms.append(m.detach())
        if grad:
            leaves = {k: rf if k == "rf" else part[k] for k in wrt}
            outs, cots = ([sig, m.T], [g_sig.to(C128), g_m[sl].to(F64)]) if h is None else ([r], [h])
            if h is not None:
                leaves["m0"] = start
            for k, g in zip(leaves, torch.autograd.grad(outs, list(leaves.values()), cots)):
                grads[k].append(g)
        del sp, part, r, m, sig
    m, sig = torch.cat(ms, 1), raw * turn
    join = lambda k: sum(grads[k]) if k == "rf" else torch.cat(grads[k], 1 if k == "m0" else 0)
    if case["call"] == "resident":
        return {"signal": sig, "m": m}
    if case["call"] == "resident_gradient":
        return {"signal": sig, "m": m, "d_rf": join("rf"), "d_m0": join("m0")}
    return {"signal": sig, "m": m.T.contiguous(), **{"d_" + k: join(k) for k in wrt}}
