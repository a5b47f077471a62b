"""Sequences whose runs of samples are short (samples during RF, a gradient of its own for every sample, a few samples to a
set of factors): both forwards and both backwards that ``engine.short_runs`` chooses between, against the float64 oracle
(1e-5 relative L2 and 2e-4 of a gradient's largest value, the bars of the forward's and the gradients' other tests)."""

from dataclasses import replace

import numpy as np
import pytest
import torch

import blochparty_b200 as bpb
from blochparty_b200 import _lib, adjoint, engine, sequences
from oracle import bloch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _phantom(n, seed=0):
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=F64)
    f32 = lambda t: t.float().double()
    return bpb.Phantom(f32((rnd(n, 3) - 0.5) * 0.2), f32(0.5 + rnd(n)), f32(0.2 + rnd(n)), f32(0.03 + 0.1 * rnd(n)),
                       f32((rnd(n) - 0.5) * 200), f32(0.8 + 0.4 * rnd(n)))


def _sequence(length, trs=3, samples=40, on_rf=False, seed=1):
    """``length`` samples to a set of factors (0: samples on the RF segments), now and then one that spoils, or none."""
    r = np.random.RandomState(seed)
    b, grads = sequences.SequenceBuilder(), []
    for i in range(trs):
        b.rf_waveform((r.rand(20, 2) - 0.4) * 4000, 10e-6, grad=(300.0, 0.0, 1000.0))
        b.delay(0.2e-3, grad=(1000.0, 500.0, 0.0))
        if length == 0:
            b.rf_waveform((r.rand(samples, 2) - 0.4) * 3000, 10e-6, grad=(300.0, 0.0, 1000.0))
            for j in range(1, samples + 1):
                b._adc[-j] = j % 11 != 5
            b._spoil[-3] = i == 1
        else:
            for k in range(0, samples, length):
                m = min(length, samples - k)
                b._append(np.full(m, 10e-6), (0.0, 0.0), tuple((r.rand(3) - 0.5) * 5000), 0.1 * k, False, True)
            b._adc[-7] = False
            b._spoil[-9] = i == 1
        b.delay(1e-3, grad=(r.rand(3) - 0.5) * 8000)
        b.spoil()
    return b.build()


def _coils(n, c, seed=2):
    g = torch.Generator().manual_seed(seed)
    rnd = lambda: torch.rand(n, c, generator=g, dtype=F64).float().double() - 0.5
    return torch.complex(rnd(), rnd())


@pytest.mark.parametrize("n,coils", [(1, 1), (33, 9), (130, 17), (1000, 32), (24001, 8), (38001, 3)])
@pytest.mark.parametrize("length", [0, 1, 2, 3, 5])
def test_both_forwards(n, coils, length):
    ph, seq, c = _phantom(n), _sequence(length), _coils(n, coils)
    sig, m = bloch.simulate(bloch.case_from(ph, seq, c))
    dev = torch.device("cuda", 0)
    inp = bpb.api.Inputs(ph.pos, ph.pd, ph.t1, ph.t2, ph.db0, ph.b1, c, seq.dt, seq.rf, seq.grad, seq.adc_phase, None,
                         list(seq.is_rf), list(seq.adc), list(seq.spoil), None)
    pk = engine.pack(inp, dev)
    win = engine.plan_windows(pk.flags, _lib.lib().bp_forward_samp_max(coils))
    wdev, W = torch.from_numpy(win).to(dev), win.shape[0]
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    rel = lambda a, b: float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))
    for windowed in (False, True):
        for cuts in ([], [1, W // 2]):
            state = engine.initial_state(ph.pd, None, dev)
            raw = torch.zeros(pk.n_adc, 2 * coils, dtype=F64, device=dev)
            for a, b in zip([0, *cuts], [*cuts, W]):
                engine.run_forward(pk, state, wdev, a, b, raw, status, windowed=windowed)
            got = engine.finish_signal(pk, raw).cpu().to(sig.dtype)
            assert rel(got, sig) < 1e-5 and rel(engine.final_m(state).double(), m) < 1e-5, (windowed, cuts)
    _lib.check_status(status, "bp_forward")


def _loss(sig, m):
    w = torch.randn(sig.shape, generator=torch.Generator().manual_seed(5), dtype=F64)
    return (sig.real.double() * w).sum() + 0.5 * (sig.imag.double() * w.flip(1)).sum() + 3.0 * (m.double() ** 2).sum()


@pytest.mark.parametrize("length,coils", [(0, 3), (1, 8), (2, 9), (3, 17), (3, 32)])
@pytest.mark.parametrize("names", [("rf",), ("t1", "t2", "coils"), ("pd", "db0", "rf")])
def test_both_backwards(length, coils, names, monkeypatch):
    """The rule forced either way, with intervals and without: each the same bits wherever the checkpoints lie."""
    n = 41
    ph, seq, c = _phantom(n, 3), _sequence(length), _coils(n, coils)
    _, want = bloch.gradients(bloch.case_from(ph, seq, c), _loss, names)
    for windowed in (True, False):
        seen, init = [], adjoint.Checkpointed.__init__

        def spy(self, *a, **kw):
            init(self, *a, **kw)
            seen.append(self.windowed)

        with monkeypatch.context() as mp:
            mp.setattr(engine, "short_runs", lambda *a, **kw: windowed)
            mp.setattr(adjoint.Checkpointed, "__init__", spy)
            got = []
            for every in (32, 96, None):
                p = replace(ph, **{k: getattr(ph, k).clone().requires_grad_() for k in names if k not in ("rf", "coils")})
                s = replace(seq, rf=seq.rf.clone().requires_grad_("rf" in names))
                co = c.clone().requires_grad_("coils" in names)
                r = bpb.simulate(p, s, co, checkpoint_every=every)
                leaves = [s.rf if k == "rf" else co if k == "coils" else getattr(p, k) for k in names]
                got.append(torch.autograd.grad(_loss(r.signal, r.m), leaves))
        assert seen == [windowed] * 3
        for k, g, *others, w in zip(names, *got, [want[k] for k in names]):
            assert all(torch.equal(g, o) for o in others), (windowed, k)
            u, v = (torch.view_as_real(t) if t.is_complex() else t for t in (g, w))
            assert float((u - v).abs().max() / v.abs().max()) < 2e-4, (windowed, k)
