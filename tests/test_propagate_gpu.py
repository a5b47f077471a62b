"""The forward in its two kernels (``bp_propagate``, ``bp_readout``) where it can go wrong: tile and fragment edges,
runs of samples of every length, chunk and window edges, saved states, against the float64 oracle. The bound is the
plain float32 bar of the forward's other tests (1e-5 relative L2; a signal's error is a few 1e-7 here)."""

import numpy as np
import pytest
import torch

import blochparty_b200 as bpb
from blochparty_b200 import _lib, engine, sequences
from blochparty_b200.api import Inputs
from oracle import bloch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _phantom(n, seed=0):
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=F64)
    f32 = lambda t: t.float().double()
    return bpb.Phantom(f32((rnd(n, 3) - 0.5) * 0.2), f32(0.5 + rnd(n)), f32(0.2 + rnd(n)), f32(0.02 + 0.1 * rnd(n)),
                       f32((rnd(n) - 0.5) * 200), f32(0.8 + 0.4 * rnd(n)))


def _sequence(lengths, seed=1, rf_adc=True):
    """Pulses (small and large steps) and readouts of the given lengths, a sample after an RF segment, a spoil on a
    sample, and a second readout that follows the first one at once with other factors."""
    g = np.random.RandomState(seed)
    b = sequences.SequenceBuilder()
    for i, k in enumerate(lengths):
        b.rf_waveform((g.rand(37, 2) - 0.5) * 2500, 10e-6, grad=(g.rand(3) - 0.5) * 2000)
        b.rf(60e-6, amplitude=9000.0, phase=1.1 * i, n_steps=2)
        if rf_adc and i % 2:
            b._adc[-1] = True
        b.delay(0.3e-3, grad=(2000.0, float(g.rand() - 0.5) * 3000, 0.0))
        b.readout(k, 10e-6, grad=(-2500.0, 300.0, 400.0), phase=0.3 * i)
        if i % 3 == 1:
            b._adc[-1] = True  # the closing half dwell samples too: a run after a run
            b.readout(3, 20e-6, grad=(100.0, 0.0, 0.0))
        if i % 3 == 2:
            b._spoil[-2] = True  # the last sample spoils
        b.delay(1e-3, grad=(g.rand(3) - 0.5) * 20000)
        b.spoil()
    return b.build()


def _check(r, sig, m):
    l2 = lambda a, b: float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))
    assert l2(r.signal.to(sig.dtype), sig) < 1e-5 and l2(r.m.double(), m) < 1e-5, (l2(r.signal.to(sig.dtype), sig),
                                                                                  l2(r.m.double(), m))


@pytest.mark.parametrize("n,coils,lengths", [
    (1, 1, (1, 2, 5)), (31, 8, (8, 9, 16, 17)), (33, 9, (31, 32, 33)), (128, 16, (95, 130, 64)), (1500, 17, (40, 1, 300)),
    (37888, 3, (33, 7)), (37889, 8, (20, 65)), (38400 + 1, 24, (12, 33)),
])
def test_against_the_oracle(n, coils, lengths):
    """One and two spins per thread (37,888 spins is the last of one), ragged tiles and coil groups, run lengths at
    the edges of the 16- and 32-sample blocks and past the longest run."""
    ph, seq = _phantom(n), _sequence(lengths)
    g = torch.Generator().manual_seed(2)
    rnd = lambda: torch.rand(n, coils, generator=g, dtype=F64).float().double() - 0.5
    c = torch.complex(rnd(), rnd()) * 10.0 ** (torch.arange(coils) - coils // 2).clamp(-3, 3).double()
    m0 = (torch.rand(n, 3, generator=g, dtype=F64) - 0.3).float().double()
    sig, m = bloch.simulate(bloch.case_from(ph, seq, c, m0))
    r = bpb.simulate(ph, seq, c, m_init=m0)
    _check(r, sig, m)
    for i in range(coils):  # every coil by itself: their scales differ by 10^6
        err = float(torch.linalg.vector_norm(r.signal[i].to(sig.dtype) - sig[i]) / torch.linalg.vector_norm(sig[i]))
        assert err < 1e-5, (i, err)


@pytest.mark.parametrize("n,coils", [(256, 4), (4096, 8), (40000, 13)])
def test_signal_to_float32_rounding(n, coils):
    """One pulse and one readout, so that the state's own error is small: the coil sums are as good as float32 ones with
    rounded operations, without a bias (the bound: 2^-23, a rounding of each factor; sums with truncated operations are
    2e-7 off whatever the size)."""
    ph = _phantom(n, 8)
    b = sequences.SequenceBuilder().rf(20e-6, flip_deg=35.0).delay(0.3e-3, grad=(2000.0, 500.0, 0.0))
    seq = b.readout(95, 10e-6, grad=(-2500.0, 300.0, 400.0)).build()
    c = bpb.birdcage_sensitivities(ph.pos, coils).to(torch.complex64).to(torch.complex128)
    sig, _ = bloch.simulate(bloch.case_from(ph, seq, c))
    r = bpb.simulate(ph, seq, c).signal.to(sig.dtype)
    err, bias = float((r - sig).norm() / sig.norm()), complex(((r - sig) * sig.conj()).sum()) / float(sig.norm()) ** 2
    assert err < 2.0 ** -23 and abs(bias) < 2.0 ** -24, (err, bias)


def test_coils_of_far_apart_sensitivities():
    """A coil 10^10 below the others of its group keeps its precision (the plain float32 bar, as above: random
    sensitivities cancel, so that a signal is a small part of the sum of its terms' sizes)."""
    n = 700
    ph, seq, g = _phantom(n, 9), _sequence((33, 64), 9, rf_adc=False), torch.Generator().manual_seed(3)
    rnd = lambda: torch.rand(n, 9, generator=g, dtype=F64).float().double() - 0.5
    scale = torch.tensor([1.0, 1e-10, 1e3, 1e-7, 1.0, 1e7, 1e-12, 1.0, 1e-5], dtype=F64)
    c = (torch.complex(rnd(), rnd()) * scale).to(torch.complex64).to(torch.complex128)
    sig, _ = bloch.simulate(bloch.case_from(ph, seq, c))
    r = bpb.simulate(ph, seq, c).signal.to(sig.dtype)
    for i in range(9):
        err = float((r[i] - sig[i]).norm() / sig[i].norm())
        assert err < 1e-5, (i, err)


def _packed(ph, seq, coils):
    dev = torch.device("cuda", 0)
    inp = Inputs(ph.pos, ph.pd, ph.t1, ph.t2, ph.db0, ph.b1, coils, seq.dt, seq.rf, seq.grad, seq.adc_phase, None,
                 list(seq.is_rf), list(seq.adc), list(seq.spoil), None)
    pk = engine.pack(inp, dev)
    win = engine.plan_windows(pk.flags, _lib.lib().bp_forward_samp_max(pk.n_coils))
    return pk, win, torch.from_numpy(win).to(dev), engine.initial_state(ph.pd, None, dev)


@pytest.mark.parametrize("n", [200, 38000])
@pytest.mark.parametrize("room", [None, 2])
def test_divided_forward(n, room, monkeypatch):
    """The forward divided at any window: the windows' samples alone (a run cut by the division is formed in two
    parts, each from its own first sample: to rounding), or whole runs where they start (the same sums and states, bit
    for bit); with a workspace for a few runs only; and the states saved by slot are the ones a division passes on."""
    ph, seq = _phantom(n, 3), _sequence((95, 64, 33, 200, 31), 4)
    coils = bpb.birdcage_sensitivities(ph.pos, 8)
    pk, win, wdev, state0 = _packed(ph, seq, coils)
    W = win.shape[0]
    if room:
        monkeypatch.setattr(engine, "Z_BYTES", 8 * n * room)
    status = torch.zeros(1, dtype=torch.int32, device=pk.device)

    def run(cuts, **kw):
        state = state0.clone()
        raw = torch.zeros(pk.n_adc, 16, dtype=F64, device=pk.device)
        states = []
        for a, b in zip([0, *cuts], [*cuts, W]):
            states.append(state.clone())
            engine.run_forward(pk, state, wdev, a, b, raw, status, **kw)
        return raw, state, states

    rel = lambda a, b: float((a - b).norm() / b.norm())
    raw, state, _ = run([])
    cuts = sorted({1, 3, 4, W // 2, W - 1})
    r2, s2, states = run(cuts)
    assert torch.equal(state, s2) and rel(r2, raw) < 1e-6
    r3, s3, _ = run(cuts, whole_runs=True)
    assert torch.equal(state, s3) and rel(r3, raw) < (1e-15 if room is None else 1e-6)
    slot = torch.full((W,), -1, dtype=torch.int32)
    for i, c in enumerate([0, *cuts]):
        slot[c] = i
    saved = torch.full((len(states), 6, n), -1.0, device=pk.device)
    engine.run_forward(pk, state0.clone(), wdev, 0, W, None, status, wstates=saved, wslot=slot.to(pk.device))
    torch.cuda.synchronize()
    for i, s in enumerate(states):
        assert torch.equal(saved[i], s), i
    _lib.check_status(status, "bp_propagate")


@pytest.mark.parametrize("n", [1000, 30000, 38000])
def test_states_saved_over_many_chunks(n):
    """A state saved at every window of a sequence of many chunks (one warp with helpers, one warp, four warps per
    CTA; no barrier between a chunk's steps in the last two), again and again: each the state a division passes on."""
    ph, seq = _phantom(n, 5), _sequence((64, 95) * 8, 6)
    pk, _, _, state0 = _packed(ph, seq, bpb.birdcage_sensitivities(ph.pos, 1))
    win = engine.plan_windows(pk.flags, 32, seg_max=32)
    wdev, W = torch.from_numpy(win).to(pk.device), win.shape[0]
    assert pk.flags.shape[0] > 6 * 256 and W > 60
    status = torch.zeros(1, dtype=torch.int32, device=pk.device)
    want, state = [], state0.clone()
    for w in range(W):
        want.append(state.clone())
        engine.run_forward(pk, state, wdev, w, w + 1, None, status)
    for _ in range(3):
        saved = torch.full((W, 6, n), -1.0, device=pk.device)
        engine.run_forward(pk, state0.clone(), wdev, 0, W, None, status, wstates=saved)
        assert torch.equal(saved, torch.stack(want))
    _lib.check_status(status, "bp_propagate")


@pytest.mark.parametrize("stride", [1, 3, 7])
@pytest.mark.parametrize("begin", [0, 2])
def test_strided_states_over_several_launches(stride, begin, monkeypatch):
    """The state at every few windows' start, from a forward in one launch and from one whose workspace divides it."""
    n = 300
    ph, seq = _phantom(n, 3), _sequence((95, 64, 33, 200, 31, 95) * 3, 4)
    pk, win, wdev, state0 = _packed(ph, seq, bpb.birdcage_sensitivities(ph.pos, 2))
    W = win.shape[0]
    status = torch.zeros(1, dtype=torch.int32, device=pk.device)
    out = []
    for room in (None, 1):
        if room:
            monkeypatch.setattr(engine, "Z_BYTES", 8 * n * room)
            assert engine._window_step(pk, W - begin)[0] < W - begin
        saved = torch.full((-(-(W - begin) // stride), 6, n), -1.0, device=pk.device)
        raw = torch.zeros(pk.n_adc, 4, dtype=F64, device=pk.device)
        engine.run_forward(pk, state0.clone(), wdev, begin, W, raw, status, wstates=saved, wstate_stride=stride)
        out.append(saved)
    assert torch.equal(out[0], out[1]) and not (out[0] == -1.0).all(2).any()
    _lib.check_status(status, "bp_propagate")


def test_first_forward_in_a_graph():
    """A packed case's first forward can be captured: no copy from the host is left for it."""
    ph, seq = _phantom(500, 3), _sequence((95, 64), 4)
    pk, win, wdev, state0 = _packed(ph, seq, bpb.birdcage_sensitivities(ph.pos, 4))
    status = torch.zeros(1, dtype=torch.int32, device=pk.device)
    state, raw = state0.clone(), torch.zeros(pk.n_adc, 8, dtype=F64, device=pk.device)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        engine.run_forward(pk, state, wdev, 0, win.shape[0], raw, status)
    assert torch.equal(state, state0) and not raw.any()
    graph.replay()
    want_state, want = state0.clone(), torch.zeros_like(raw)
    engine.run_forward(pk, want_state, wdev, 0, win.shape[0], want, status)
    torch.cuda.synchronize()
    assert torch.equal(state, want_state) and float((raw - want).abs().max()) <= 1e-13 * float(want.abs().max())
    _lib.check_status(status, "bp_propagate")
