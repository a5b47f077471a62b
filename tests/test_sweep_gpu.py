"""The sweep over runs of like segments (``bp_cotangent``, ``bp_sweep``): gradients against the float64 oracle's
autograd, and against the segment-by-segment sweep (``bp_adjoint``) where the oracle would take long. The bar is the
gradient tests' 2e-4 of a gradient's largest value (float32 states in a reverse sweep; 1e-5 to 5e-5 here)."""

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


def _sequence(lengths, rf_steps=37, seed=1):
    """Pulses of one offset, readouts of the given lengths (a first half dwell, or none), a spoil on a sample, a
    readout that follows another at once, and samples that stop and go within one set of factors."""
    g = np.random.RandomState(seed)
    b = sequences.SequenceBuilder()
    for i, k in enumerate(lengths):
        b.rf_waveform((g.rand(rf_steps, 2) - 0.4) * 2500 * (10 if i % 2 else 1), 10e-6, grad=(300.0, 0.0, 1000.0))
        b.delay(0.3e-3, grad=(2000.0, float(g.rand() - 0.5) * 3000, 0.0))
        b.readout(k, 10e-6, grad=(-2500.0, 300.0, 400.0), phase=0.3 * i)
        if i % 3 == 0 and k > 4:
            b._adc[-4] = False  # a gap in the samples of one set of factors
        if i % 3 == 1:
            b._adc[-1] = True
            b.readout(3, 20e-6, grad=(100.0, 0.0, 0.0))
        if i % 3 == 2:
            b._spoil[-2] = True  # the last sample spoils
            b._append(np.full(5, 20e-6), (0.0, 0.0), (500.0, 0.0, 0.0), 0.1, False, True)  # samples from the first on
        b.delay(1e-3, grad=(g.rand(3) - 0.5) * 8000)
        b.spoil()
    return b.build()


def _coils(n, c, seed=2):
    g = torch.Generator().manual_seed(seed)
    rnd = lambda: torch.rand(n, c, generator=g, dtype=F64).float().double() - 0.5
    return torch.complex(rnd(), rnd())


def _gradients(ph, seq, coils, names, every=None):
    ph = replace(ph, **{k: getattr(ph, k).clone().requires_grad_() for k in names if k not in ("rf", "coils")})
    if "rf" in names:
        seq = replace(seq, rf=seq.rf.clone().requires_grad_())
    if "coils" in names:
        coils = coils.clone().requires_grad_()
    r = bpb.simulate(ph, seq, coils, checkpoint_every=every)
    leaves = [seq.rf if k == "rf" else coils if k == "coils" else getattr(ph, k) for k in names]
    return dict(zip(names, torch.autograd.grad(_loss(r.signal, r.m), leaves)))


def _loss(sig, m):
    g = torch.Generator().manual_seed(5)
    w = torch.randn(sig.shape, generator=g, dtype=F64) * (1.0 + 100.0 * (torch.arange(sig.shape[1]) % 17 == 3))
    return (sig.real.double() * w).sum() + 0.5 * (sig.imag.double() * w.flip(1)).sum() + 3.0 * (m.double() ** 2).sum()


def _spy(monkeypatch):
    seen = []
    sweeps = adjoint.Checkpointed.sweeps

    def spy(self, *a):
        seen.append(sweeps(self, *a))
        return seen[-1]

    monkeypatch.setattr(adjoint.Checkpointed, "sweeps", spy)
    return seen


def _close(a, b, names, bar=2e-4):
    for k in names:
        u, v = (torch.view_as_real(t) if t.is_complex() else t for t in (a[k], b[k]))
        err = float((u - v).abs().max() / v.abs().max())
        assert err < bar, (k, err)


@pytest.mark.parametrize("n,coils,lengths,names", [
    (33, 8, (8, 9, 33), ("pd", "t1", "t2", "db0", "b1", "coils", "pos")),
    (100, 1, (1, 2, 5, 31), ("t1", "rf")),
    (129, 9, (95, 64, 130), ("rf", "coils")),
    (61, 17, (40, 32, 16), ("pd", "t1", "t2", "db0", "b1", "rf")),
    (64, 8, (300, 20, 7), ("rf",)),
    (40, 3, (260, 12, 45), ("t2", "db0", "coils")),
])
def test_against_the_oracle(n, coils, lengths, names, monkeypatch):
    seen = _spy(monkeypatch)
    ph, seq, c = _phantom(n), _sequence(lengths), _coils(n, coils)
    got = _gradients(ph, seq, c, names, every=64)
    assert seen and all(seen)
    again = _gradients(ph, seq, c, names, every=32 * 100)
    kept = _gradients(ph, seq, c, names)  # every state from the forward, no replay
    for k in names:  # the same bits wherever the checkpoints lie
        assert torch.equal(got[k], again[k]) and torch.equal(got[k], kept[k]), k
    _, want = bloch.gradients(bloch.case_from(ph, seq, c), _loss, names)
    _close(got, want, names)


@pytest.mark.parametrize("n", [37888, 37889, 40001])
@pytest.mark.parametrize("names", [("rf",), ("t1", "t2", "db0", "coils"), ("pd", "b1", "rf")])
def test_against_the_segment_sweep(n, names, monkeypatch):
    """Both spin layouts of the kernels, at and past the line between them."""
    ph, seq, c = _phantom(n, 3), _sequence((17, 64), rf_steps=70), _coils(n, 8)
    with monkeypatch.context() as m:
        seen = _spy(m)
        got = _gradients(ph, seq, c, names)
        assert seen and all(seen)
    with monkeypatch.context() as m:
        m.setattr(adjoint, "rf_relaxation_invertible", lambda pk: False)  # (bp_adjoint with a replay)
        seen = _spy(m)
        want = _gradients(ph, seq, c, names)
        assert seen and not any(seen)
    _close(got, want, names)


@pytest.mark.parametrize("t2", [10e-6, 20e-6, 50e-6, 100e-6, 150e-6, 200e-6, 1e-3])
@pytest.mark.parametrize("names", [("rf",), ("t2", "db0", "b1"), ("t1", "rf")])
@pytest.mark.parametrize("every", [None, 64])
def test_short_t2(t2, names, every):
    """Relaxation as fast as the pulses: integrating a state backward over a duration t multiplies its rounding errors
    by exp(t / T2), so past t / T2 = 2 the states come forward from saved ones."""
    n = 37
    g = torch.Generator().manual_seed(7)
    ph = _phantom(n, 4)
    ph = replace(ph, t2=(t2 * (0.9 + 0.2 * torch.rand(n, generator=g, dtype=F64))).float().double())
    b = sequences.SequenceBuilder()
    r = np.random.RandomState(3)
    for i in range(2):
        b.rf_waveform((r.rand(200, 2) - 0.3) * 4000, 10e-6, grad=(300.0, 0.0, 1000.0))
        b.readout(20, min(10e-6, 0.2 * t2), grad=(-2500.0, 300.0, 400.0), phase=0.3 * i)
        b.delay(0.2e-3, grad=(2000.0, 0.0, 0.0))
    seq, c = b.build(), _coils(n, 4)
    got = _gradients(ph, seq, c, names, every=every)
    _, want = bloch.gradients(bloch.case_from(ph, seq, c), _loss, names)
    _close(got, want, names)


@pytest.mark.parametrize("names", [("t1", "t2", "coils"), ("pos", "rf"), ("rf",)])
def test_long_intervals(names, monkeypatch):
    """An interval of more segments than one sweep takes, and one with more runs of samples than the sums' workspace
    holds: swept in pieces, the same bits as with short intervals and with every state kept."""
    n = 50
    ph, seq, c = _phantom(n, 6), _sequence((95, 64, 130, 33) * 5, rf_steps=20), _coils(n, 9)
    assert len(seq) > 2048 + 64
    seen = _spy(monkeypatch)
    want = _gradients(ph, seq, c, names, every=64)
    for every, room in ((3200, None), (3200, 3), (320, 1), (None, None), (None, 2)):
        with monkeypatch.context() as m:
            if room:
                m.setattr(engine, "Z_BYTES", 8 * n * room)
            got = _gradients(ph, seq, c, names, every=every)
        for k in names:
            assert torch.equal(got[k], want[k]), (every, room, k)
    assert seen and all(seen)
    _, exact = bloch.gradients(bloch.case_from(ph, seq, c), _loss, names)
    _close(want, exact, names)


def test_weights_far_apart():
    """A loss that weighs early samples 10^9 above late ones, and one coil 10^9 below another: the late pulses' RF
    gradient, which only late samples reach, and the faint coil's keep their precision."""
    n = 45
    ph, c = _phantom(n, 10), _coils(n, 3)
    b = sequences.SequenceBuilder()
    for i in range(3):
        b.rf_waveform((np.random.RandomState(i).rand(40, 2) - 0.4) * 2500, 10e-6, grad=(300.0, 0.0, 1000.0))
        b.readout(50, 10e-6, grad=(-2500.0, 300.0, 400.0)).delay(1e-3, grad=(3e3, 1e3, 0.0)).spoil()
    seq = b.build()
    weight = torch.tensor([1e9, 1.0, 1e-3], dtype=F64).repeat_interleave(50)[None, :] * torch.tensor(
        [[1.0], [1e-9], [1.0]], dtype=F64)

    def loss(sig, m):
        w = weight * torch.randn(sig.shape, generator=torch.Generator().manual_seed(5), dtype=F64)
        return (sig.real.double() * w).sum() + 0.5 * (sig.imag.double() * w).sum()

    rf, co = seq.rf.clone().requires_grad_(), c.clone().requires_grad_()
    r = bpb.simulate(ph, replace(seq, rf=rf), co, checkpoint_every=64)
    g_rf, g_c = torch.autograd.grad(loss(r.signal, r.m), (rf, co))
    _, want = bloch.gradients(bloch.case_from(ph, seq, c), loss, ("rf", "coils"))
    starts = np.flatnonzero(np.diff(np.asarray(seq.is_rf).astype(int), prepend=0) == 1)
    for s in starts:
        _close({"rf": g_rf[s:s + 40]}, {"rf": want["rf"][s:s + 40]}, ("rf",))
    for i in range(3):
        _close({"c": g_c[:, i]}, {"c": want["coils"][:, i]}, ("c",))


def test_runs_of_any_length(monkeypatch):
    """Runs longer than the forward's longest, the samples' numbers in hundreds: their part of the maps' gradients."""
    ph, c, names = _phantom(40, 11), _coils(40, 4), ("t2", "db0", "coils")
    b = sequences.SequenceBuilder()
    for i in range(2):
        b.rf(20e-6, flip_deg=30.0).readout(900, 5e-6, grad=(-900.0, 300.0, 400.0)).delay(1e-3)
    seq = b.build()
    run = adjoint.engine.sample_runs
    assert run(np.full(900, 8 | 2, dtype=np.int32))[0][:, 2].max() <= engine.RUN_MAX
    monkeypatch.setattr(engine, "RUN_MAX", 1 << 20)
    got = _gradients(ph, seq, c, names, every=3200)
    _, want = bloch.gradients(bloch.case_from(ph, seq, c), _loss, names)
    _close(got, want, names)


def test_many_graphs_alive():
    """Every window's states are kept while more than half of the device is free, else the checkpoints' replay: the same
    gradients, bit for bit."""
    n, names = 60, ("t1", "coils")
    ph, seq, c = _phantom(n, 12), _sequence((40, 17)), _coils(n, 2)
    kept, init = [], adjoint.Checkpointed.__init__

    def spy(self, *a, **kw):
        init(self, *a, **kw)
        kept.append(self.kept is not None)

    out = []
    with pytest.MonkeyPatch.context() as m:
        m.setattr(adjoint.Checkpointed, "__init__", spy)
        for share in (0.9, 0.4):
            m.setattr(torch.cuda, "mem_get_info", lambda *a: (int(share * (180 << 30)), 180 << 30))
            m.setattr(torch.cuda, "memory_reserved", lambda *a: 0)
            m.setattr(torch.cuda, "memory_allocated", lambda *a: 0)
            out.append(_gradients(ph, seq, c, names))
    assert kept == [True, False]
    assert all(torch.equal(out[0][k], out[1][k]) for k in names)


@pytest.mark.parametrize("states", [8, 10, 1000])
@pytest.mark.parametrize("ends_with_rf", [False, True])
def test_backward_twice_from_saved_states(states, ends_with_rf):
    """The RF waveform's gradient from one forward, backward twice (a graph kept for a second gradient): the same bits
    with the saved states in blocks, whose last one the first backward has written over, as with all of them kept."""
    n = 70
    ph, seq, c = _phantom(n, 13), _sequence((40, 17, 64, 9) * 3), _coils(n, 3)
    if ends_with_rf:
        cut = int(np.flatnonzero(np.asarray(seq.is_rf))[-1]) + 1
        seq = bpb.Sequence(seq.dt[:cut], seq.rf[:cut], seq.grad[:cut], seq.adc_phase[:cut], seq.is_rf[:cut], seq.adc[:cut],
                           seq.spoil[:cut])
    dev = torch.device("cuda", 0)
    inp = bpb.api.Inputs(ph.pos, ph.pd, ph.t1, ph.t2, ph.db0, ph.b1, c, seq.dt, seq.rf, seq.grad, seq.adc_phase, None,
                         list(seq.is_rf), list(seq.adc), list(seq.spoil), None)
    pk = engine.pack(inp, dev)
    g = torch.Generator().manual_seed(1)
    h, lam0 = torch.randn(pk.n_adc, 6, generator=g).to(dev), torch.randn(3, n, generator=g).to(dev)
    mask = _lib.BP_SEG_WX | _lib.BP_SEG_WY | _lib.BP_SPIN_NO_OFFSETS | _lib.BP_SPIN_NONE
    out = []
    for budget in (24 * n * states, 1 << 40):
        run = adjoint.Checkpointed(pk, 64, dev, saved=True, budget_bytes=budget)
        assert run.saved is not None and run.saved.final == ends_with_rf
        assert len(run.blocks()) > 1 or budget >= 24 * n * 1000
        run.forward(engine.initial_state(ph.pd, None, dev))
        for _ in range(2):
            lam = lam0.clone()
            seg = run.backward(h, lam, mask, False, True)[2]
            out.append((seg.clone(), lam))
        run.check()
    for seg, lam in out[1:]:
        assert torch.equal(seg, out[0][0]) and torch.equal(lam, out[0][1])
