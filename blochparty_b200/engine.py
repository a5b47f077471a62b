"""Host driver of the b200 engine: inputs into device buffers, the window plan, the launches, the results.

Replaces blochparty's GPU driver for static spins (``engines/gpu/driver.py:_forward``, :197-756): the same
float64-on-host preparation (positions, rates 1/T1 and 1/T2, per-segment quantities, the state split into a
float32 high part and its float32 remainder) feeding the C ABI of ``libblochparty_b200.so``.

Device buffers (float32 unless stated; N spins, S segments, C coils, A ADC samples):

* ``spins`` [8][N]: x, y, z, pd, r1, r2, dB0, b1 (structure of arrays: one coalesced row per field);
* ``sens`` [16 ceil(C/8)][N]: coil c real at row 2c, imaginary at 2c+1, zero padding rows;
* ``segs`` [S] 32-byte records: dt, -2 pi dt rf_x, -2 pi dt rf_y, g dt (3), b0_offset dt, flags (int32);
* ``seg64`` [S][4] float64: g dt (3), b0_offset dt: the free segments' phase is evaluated in float64;
* ``windows`` [W][4] int32: first segment, end segment, first ADC row, samples (``bp_plan_windows``);
* ``state`` [6][N]: mx, my, mz and their compensation parts;
* ``raw`` [A][2C] float64: the coil sums before demodulation; ``signal`` (C, A) complex64.
"""

from __future__ import annotations

import ctypes
import math
from dataclasses import dataclass

import numpy as np
import torch

from . import _lib
from ._lib import ptr

TWO_PI = 2.0 * math.pi
F32, F64 = torch.float32, torch.float64

RF, ADC, SPOIL, SAME_FREE, SAME_RFDT, SAME_OFF, SMALL = 1, 2, 4, 8, 16, 32, 64


Z_BYTES = 1 << 30  # the forward's workspace at most: the first samples of the runs of one launch
RUN_MAX = 256  # samples per run
# A run of samples costs bp_readout its factor and a table of powers, up to about 40 ps a spin and group of eight coils
# whatever its samples; bp_forward pays per sample. The lines between them: samples per 32-sample block (of the sequence),
# and spins, more of them the more samples. 1,600 samples, 8 coils, bp_propagate + bp_readout against bp_forward [ms]:
#   samples per run  4,096 spins   20,000        40,000        262,144
#   1 (on RF)        0.90 / 0.43   1.69 / 0.51   2.68 / 0.61   15.1 / 2.5
#   2                0.57 / 0.85   1.14 / 1.00   2.01 / 1.20   10.4 / 5.2
#   4                0.30 / 0.53   0.61 / 0.64   1.04 / 0.76   5.1 / 3.3
#   8                0.19 / 0.37   0.35 / 0.45   0.56 / 0.54   2.63 / 2.28
#   16               0.13 / 0.29   0.24 / 0.36   0.33 / 0.43   1.40 / 1.82
# and with gradients of the T1 map (8 coils), the sweep over runs against bp_adjoint:
#   2                2.2 / 4.3     3.7 / 4.8     (100,000 spins) 12.7 / 10.6
#   4                1.0 / 2.7     1.9 / 2.9     6.5 / 6.6, of the RF waveform 4.3 / 3.7
#   8                0.55 / 1.9    1.1 / 2.1     3.3 / 4.5
#   4 at 40,000 spins, of the T1 map 2.9 / 3.3, of the RF waveform 2.4 / 1.9
ONE_SAMPLE, FEW_SAMPLES, FEW_SAMPLES_GRAD = 1.5, 10.0, 6.0
SPINS_PER_SAMPLE, SPINS_GRAD = 5000, 15000


def sample_runs(flags: np.ndarray):
    """(runs (R, 4), subs (B, 2)) int32: the runs of samples (``bp_propagate`` in the header: first segment, the segment
    after it or -1, samples, ADC row of the first) and their 32-sample blocks. A sample joins the run before it when it
    follows it on a free segment, unspoiled, with the factors of the run's samples (a run of one sample takes any: a
    readout's first sample half a dwell in, then the dwells). A run that would pass ``RUN_MAX`` samples ends at a
    multiple of 32 segments."""
    fl = np.ascontiguousarray(flags, dtype=np.int32)
    n_adc = int(np.count_nonzero(fl & ADC))
    runs, subs = np.empty((n_adc, 4), dtype=np.int32), np.empty((n_adc, 2), dtype=np.int32)
    n = np.zeros(2, dtype=np.int64)
    code = _lib.lib().bp_sample_runs(fl.ctypes.data, fl.shape[0], RUN_MAX, runs.ctypes.data, n_adc, n[:1].ctypes.data,
                                     subs.ctypes.data, n_adc, n[1:].ctypes.data)
    _lib.check(code, "bp_sample_runs")
    return runs[: n[0]], subs[: n[1]]


class SampleRuns:
    """The runs of samples of a sequence and their blocks of 32, on the device for ``bp_propagate`` and
    ``bp_readout``."""

    def __init__(self, flags: np.ndarray, device):
        runs, subs = sample_runs(flags)
        both = torch.from_numpy(np.concatenate([runs.reshape(-1), subs.reshape(-1)])).to(device)
        self.n_runs, self.n_subs = runs.shape[0], subs.shape[0]
        self.runs, self.subs = both[: runs.size], both[runs.size:]
        self.starts, self.lengths = runs[:, 0], runs[:, 2]

    def most_blocks(self, runs: int) -> int:
        """The most 32-sample blocks that ``runs`` runs in a row have."""
        if runs >= self.n_runs:
            return self.n_subs
        before = np.concatenate([[0], np.cumsum((self.lengths + 31) // 32)])
        return int((before[runs:] - before[:-runs]).max()) if runs else 0

    def most_in(self, segments: int) -> int:
        """The most runs that start within any stretch of ``segments`` segments."""
        if self.n_runs == 0:
            return 0
        return int((np.searchsorted(self.starts, self.starts + segments) - np.arange(self.n_runs)).max())


@dataclass
class Packed:
    """A case's device buffers (see module docstring) and sizes."""

    n: int
    n_coils: int
    n_adc: int
    spins: torch.Tensor
    sens: torch.Tensor
    segs: torch.Tensor  # (S, 8) float32 view of the records (the flags column holds int32 bits)
    seg64: torch.Tensor
    psi: torch.Tensor  # (A,) float64 receiver phase of every sample
    flags: np.ndarray  # (S,) int32 on the host
    device: torch.device
    runs: SampleRuns | None = None  # the runs of samples (sample_runs)
    dt: np.ndarray | None = None  # the segments' durations (float32) and the spins' largest relaxation rate, on the host
    rate: float | None = None

    def sample_runs(self) -> SampleRuns:
        if self.runs is None:
            self.runs = SampleRuns(self.flags, self.device)
        return self.runs

    def windowed(self, grad: bool = False) -> bool:
        """``short_runs`` of this case."""
        return self.n_adc > 0 and short_runs(self.n_adc, self.sample_runs().n_subs, self.n, grad)


def short_runs(n_adc: int, n_blocks: int, n: int, grad: bool = False) -> bool:
    """Whether a forward of ``n`` spins (with gradients: and its backward) takes ``bp_forward``'s windows instead of
    ``bp_propagate`` and ``bp_readout``: where the runs of samples are short (the lines above)."""
    if n_blocks == 0:
        return False
    mean = n_adc / n_blocks
    few, spins = (FEW_SAMPLES_GRAD, SPINS_GRAD) if grad else (FEW_SAMPLES, 0)
    return mean < ONE_SAMPLE or (mean < few and n > spins + SPINS_PER_SAMPLE * mean)


def _bools(flags, n: int) -> np.ndarray:
    """A sequence of n truth values (Python bools or ints, as blochparty's Sequence holds them) as a bool array:
    through bytes() when every item is a small int (four times faster on a million items), else item by item."""
    if isinstance(flags, (list, tuple)):
        try:
            out = np.frombuffer(bytes(flags), dtype=np.uint8).astype(bool)
            if out.shape[0] == n:
                return out
        except (TypeError, ValueError):
            pass
    return np.fromiter((bool(x) for x in flags), dtype=bool, count=n)


def _np64(t) -> np.ndarray:
    return t.detach().to(F64).cpu().numpy()


def _host(t: torch.Tensor) -> torch.Tensor:
    """``t`` as a contiguous host tensor of float32, float64, complex64 or complex128."""
    t = t.detach().cpu().resolve_conj().resolve_neg()
    if t.dtype not in (F32, F64, torch.complex64, torch.complex128):
        t = t.to(F64)
    return t.contiguous()


def _upload_spins(pos, pd, t1, t2, db0, b1, coils, m_init, device, want_state: bool):
    """(spins [8][N], sens [16 ceil(C/8)][N], state [6][N] or None, extent): every value rounded once to float32 from
    its float64 value (the rates 1/T1, 1/T2 formed in float64), by the native packer through page-locked staging;
    extent: the largest magnitude of every row of ``spins`` (float32 on the host)."""
    n, n_coils = pd.shape[0], coils.shape[1]
    rows = [_host(t.expand(n)) for t in (pd, t1, t2, db0)]
    pos = _host(pos.expand(n, 3))
    b1 = None if b1 is None else _host(b1.expand(n))
    if coils.shape != (n, n_coils):
        coils = coils.reshape(n, n_coils)  # (raises where it has other than n rows: the packer reads n of them)
    coils = _host(coils if coils.dtype in (torch.complex64, torch.complex128) else coils.to(torch.complex128))
    m0 = None if m_init is None else _host(m_init.expand(n, 3))
    spins = torch.empty(8, n, dtype=F32, device=device)
    sens = torch.empty(16 * ((n_coils + 7) // 8), n, dtype=F32, device=device)
    state = torch.empty(6, n, dtype=F32, device=device) if want_state else None
    extent = np.zeros(8, dtype=np.float32)
    arrays = [pos, *rows, b1, coils, m0]
    src = _lib.BpHostSpins(*(ptr(t) for t in arrays))
    for i, t in enumerate(arrays):
        src.wide[i] = int(t is not None and t.dtype in (F64, torch.complex128))
    lib = _lib.lib()
    staging = torch.empty(lib.bp_pack_spins_staging(n, n_coils), dtype=torch.uint8, pin_memory=True)
    with torch.cuda.device(device):
        code = lib.bp_pack_spins(ctypes.addressof(src), n, n_coils, ptr(spins), ptr(sens), ptr(state),
                                 extent.ctypes.data, ptr(staging), staging.numel(), _lib.stream_ptr())
    _lib.check(code, "bp_pack_spins")
    return spins, sens, state, extent


def pack_spins(pos, pd, t1, t2, db0, b1, coils, device):
    """spins [8][N] and sens [16 ceil(C/8)][N] float32 on ``device`` (``_upload_spins``; on the CPU row by row in
    torch)."""
    n = pd.shape[0]
    if torch.device(device).type == "cuda" and 0 < n and 0 < coils.shape[1] <= _lib.BP_MAX_COILS:
        return _upload_spins(pos, pd, t1, t2, db0, b1, coils, None, device, False)[:2]
    d64 = lambda t: t.detach().cpu().to(F64)
    spins = torch.empty(8, n, dtype=F32)
    spins[0:3] = d64(pos).T
    spins[3] = d64(pd)
    spins[4] = 1.0 / d64(t1)
    spins[5] = 1.0 / d64(t2)
    spins[6] = d64(db0)
    if b1 is None:
        spins[7] = 1.0
    else:
        spins[7] = d64(b1)
    n_coils = coils.shape[1]
    ncg = (n_coils + 7) // 8
    c = torch.view_as_real(coils.detach().cpu().to(torch.complex128).contiguous()).reshape(n, 2 * n_coils).to(F32)
    sens = torch.zeros(16 * ncg, n, dtype=F32, device=device)
    sens[0:2 * n_coils] = c.to(device).T
    return spins.to(device).contiguous(), sens.contiguous()


def pack_segments(dt, rf, grad, b0_offset, adc_phase, is_rf, adc, spoil, device, extent: np.ndarray | None = None):
    """Segment records (float64 arithmetic, one rounding to float32), the float64 moments, psi, the flags (host) and
    the number of samples, by the native packer into one buffer and, on a GPU, one copy from page-locked memory.
    ``extent``: the spins' extents (``_upload_spins``), to set SMALL as ``mark_small_rf`` does. The RF, the gradient and
    the offset are broadcast over the segments (one offset for all of them, say); the RF's first two columns count."""
    dt, rf = _np64(dt), _np64(rf)
    S = dt.shape[0]
    if rf.ndim != 2 or rf.shape[1] < 2:
        raise ValueError(f"the RF takes two columns, got {rf.shape}")

    def rows(t, *shape):
        if t.shape != shape:
            t = np.broadcast_to(t, shape)  # (raises where it cannot)
        return np.ascontiguousarray(t)

    phase = _np64(adc_phase)
    if phase.shape == (S, 1):
        phase = phase[:, 0]
    if dt.shape != (S,) or phase.shape != (S,):
        raise ValueError(f"a sequence of {S} segments takes a duration and a phase for each, got {dt.shape}, {phase.shape}")
    dt, rf, grad, phase = rows(dt, S), rows(rf[:, :2], S, 2), rows(_np64(grad), S, 3), rows(phase, S)
    b0 = None if b0_offset is None else rows(_np64(b0_offset), S)
    marks = [np.ascontiguousarray(_bools(f, S)).view(np.uint8) for f in (is_rf, adc, spoil)]
    n_adc = int(np.count_nonzero(marks[1]))
    flags = np.empty(S, dtype=np.int32)
    gpu = torch.device(device).type == "cuda"
    host = torch.empty(64 * S + 8 * n_adc, dtype=torch.uint8, pin_memory=gpu and S > 0)
    base = host.data_ptr()
    count = np.zeros(1, dtype=np.int64)
    code = _lib.lib().bp_pack_segments(dt.ctypes.data, rf.ctypes.data, grad.ctypes.data,
                                       None if b0 is None else b0.ctypes.data, phase.ctypes.data,
                                       *(m.ctypes.data for m in marks), S,
                                       None if extent is None else extent.ctypes.data, base, base + 32 * S,
                                       flags.ctypes.data, base + 64 * S, count.ctypes.data)
    _lib.check(code, "bp_pack_segments")
    dev = host.to(device, non_blocking=True) if gpu else host
    return (dev[: 32 * S].view(F32).view(S, 8), dev[32 * S: 64 * S].view(F64).view(S, 4), dev[64 * S:].view(F64), flags,
            n_adc)


def plan_windows(flags: np.ndarray, samp_max: int, seg_max: int = _lib.BP_SEG_MAX, breaks: np.ndarray | None = None):
    """(W, 4) int32 windows from the native planner (``bp_plan_windows``)."""
    S = flags.shape[0]
    n_adc = int(((flags & ADC) != 0).sum())
    n_breaks = 0 if breaks is None else int(breaks.sum())
    cap = 2 * (S // seg_max + n_adc // samp_max + n_breaks) + 2  # (grown below if the aligned cuts need more)
    nw = np.zeros(1, dtype=np.int64)
    fl = np.ascontiguousarray(flags, dtype=np.int32)
    br = None if breaks is None else np.ascontiguousarray(breaks, dtype=np.uint8)
    while True:
        out = np.zeros((cap, 4), dtype=np.int32)
        code = _lib.lib().bp_plan_windows(fl.ctypes.data, S, seg_max, samp_max,
                                          None if br is None else br.ctypes.data, out.ctypes.data, cap, nw.ctypes.data)
        if code != _lib.BP_E_SIZE or cap >= S + 1:
            break
        cap = min(2 * cap, S + 1)
    _lib.check(code, "bp_plan_windows")
    return out[: int(nw[0])].copy()


def initial_state(pd, m_init, device):
    """[6][N] float32: m0 split exactly from float64 into a float32 high part and its float32 remainder."""
    n = pd.shape[0]
    out = torch.zeros(6, n, dtype=F32)
    if m_init is None:  # (0, 0, pd): only the z rows are nonzero
        z = pd.detach().cpu().to(F64)
        out[2] = z
        out[5] = z - out[2].to(F64)
    else:
        m64 = m_init.detach().cpu().to(F64).T
        out[0:3] = m64
        out[3:6] = m64 - out[0:3].to(F64)
    return out.to(device).contiguous()


def final_m(state: torch.Tensor) -> torch.Tensor:
    if state.is_cuda and state.is_contiguous():
        m = torch.empty(state.shape[1], 3, dtype=F32, device=state.device)
        _lib.check(_lib.lib().bp_final_m(ptr(state), state.shape[1], ptr(m), _lib.stream_ptr()), "bp_final_m")
        return m.cpu()
    s = state.to(F64)
    return (s[0:3] + s[3:6]).to(F32).T.contiguous().cpu()


def mark_small_rf(spins: torch.Tensor, segs: torch.Tensor, flags: np.ndarray) -> None:
    """Set SMALL on the RF segments whose rotation |w|^2 = b1^2 (wx0^2 + wy0^2) + wz^2 stays below 0.0624 (under
    the first tier's 1/16) for every spin, bounding |wz| = 2 pi |k.r + dt dB0 + beta| by the spins' extents (in the
    device records and the host flags). The kernels then take the first-tier factors without tests: the same
    arithmetic the tests would choose. (The reference tests phi per spin and step, switching to its two-term
    series below phi = 1e-3: blochparty ``engines/gpu/shaders/common.metal:57-72``.)"""
    if spins.shape[1] == 0 or segs.shape[0] == 0:
        return
    ext = spins.abs().amax(dim=1).to(F64)  # |x|, |y|, |z|, pd, r1, r2, |dB0|, |b1| maxima
    rec = segs.to(F64)
    wz = TWO_PI * (rec[:, 3].abs() * ext[0] + rec[:, 4].abs() * ext[1] + rec[:, 5].abs() * ext[2]
                   + rec[:, 0].abs() * ext[6] + rec[:, 6].abs())
    p2 = ext[7] ** 2 * (rec[:, 1] ** 2 + rec[:, 2] ** 2) + wz ** 2
    bits = segs.view(torch.int32)[:, 7]
    small = ((bits & RF) != 0) & (p2 < 0.0624)
    bits |= small.to(torch.int32) * SMALL
    flags |= small.cpu().numpy().astype(np.int32) * SMALL


def pack_with_state(case, device):
    """(``pack(case, device)``, its start state [6][N] on ``device``)."""
    n, n_coils = case.pd.shape[0], case.coils.shape[1]
    extent = None
    if torch.device(device).type == "cuda" and 0 < n and 0 < n_coils <= _lib.BP_MAX_COILS:
        spins, sens, state, extent = _upload_spins(case.pos, case.pd, case.t1, case.t2, case.db0, case.b1, case.coils,
                                                   case.m_init, device, True)
    else:
        spins, sens = pack_spins(case.pos, case.pd, case.t1, case.t2, case.db0, case.b1, case.coils, device)
        state = initial_state(case.pd, case.m_init, device)
    segs, seg64, psi, flags, n_adc = pack_segments(case.dt, case.rf, case.grad, case.b0_offset, case.adc_phase,
                                                   case.is_rf, case.adc, case.spoil, device, extent)
    if extent is None:
        mark_small_rf(spins, segs, flags)
    pk = Packed(n, n_coils, n_adc, spins, sens, segs, seg64, psi, flags, device)
    if extent is not None:
        pk.dt, pk.rate = _np64(case.dt).astype(np.float32), float(np.maximum(extent[4], extent[5]))
    if segs.is_cuda and n_adc:
        pk.sample_runs()  # (a forward is then launches alone: it can be the first thing in a captured graph)
    return pk, state


def pack(case, device) -> Packed:
    return pack_with_state(case, device)[0]


def _window_step(pk: Packed, windows: int) -> tuple[int, int]:
    """(windows per launch, runs the workspace holds) of a forward with a readout over ``windows`` windows: all of them
    where the runs' first samples fit ``Z_BYTES``, else as many as keep any launch's runs under it."""
    runs, step = pk.sample_runs(), max(windows, 1)
    cap, room = runs.n_runs, max(Z_BYTES // (8 * max(pk.n, 1)), 1)
    if step * _lib.BP_SEG_MAX < pk.flags.shape[0]:  # (some of the sequence's windows: not all of its runs)
        cap = min(cap, runs.most_in(step * _lib.BP_SEG_MAX) + 1)
    if cap > room:
        step = max(1, step * room // cap)
        while step > 1 and runs.most_in(step * _lib.BP_SEG_MAX) + 1 > room:
            step = (step + 1) // 2
        cap = min(cap, runs.most_in(step * _lib.BP_SEG_MAX) + 1)
    return step, cap


def forward_launches(pk: Packed, windows: int) -> int:
    """Kernel launches of ``run_forward`` with a readout over ``windows`` windows."""
    if pk.windowed():
        return 1
    step, cap = _window_step(pk, windows)
    return -(-windows // step) * (2 if cap else 1)


def run_forward(pk: Packed, state: torch.Tensor, windows_dev: torch.Tensor, w_begin: int, w_end: int,
                raw: torch.Tensor | None, status: torch.Tensor, wstates: torch.Tensor | None = None,
                wstate_stride: int = 1, max_ctas: int = 0, wslot: torch.Tensor | None = None,
                whole_runs: bool = False, windowed: bool | None = None) -> torch.Tensor | None:
    """The forward over windows [w_begin, w_end) from ``state``, advanced in place. With ``windowed`` (``pk.windowed()``
    unless given): one launch of ``bp_forward``, the samples formed window by window. Else: ``bp_propagate``, then with
    ``raw`` (the coil sums, added to) ``bp_readout``, over as many windows at a time as keep the workspace between
    them under ``Z_BYTES``. ``wstates``: states at window starts, every ``wstate_stride``-th or by slot (``wslot``).
    ``whole_runs``: a run of samples is formed whole by the call whose windows it starts in (calls over consecutive
    windows then give the same bits wherever they are divided); else the windows' samples alone. Returns the workspace
    (the runs' first samples, [run][N] pairs) when one launch took all windows."""
    lib, stream = _lib.lib(), _lib.stream_ptr()
    if pk.windowed() if windowed is None else windowed:
        case = (ptr(pk.spins), ptr(pk.sens), pk.n, pk.n_coils, ptr(pk.segs), ptr(pk.seg64), ptr(windows_dev), w_begin, w_end,
                ptr(state), ptr(raw))
        if wslot is None:
            code = lib.bp_forward(*case, ptr(wstates), wstate_stride, max_ctas, ptr(status), stream)
        else:
            code = lib.bp_forward_saving(*case, ptr(wslot), ptr(wstates), max_ctas, ptr(status), stream)
        _lib.check(code, "bp_forward")
        return None
    runs = pk.sample_runs() if raw is not None else None
    step, cap = _window_step(pk, w_end - w_begin) if runs is not None else (max(w_end - w_begin, 1), 0)
    z = torch.empty(cap, pk.n, 2, dtype=F32, device=pk.device) if cap else None
    most_subs = 0 if z is None else runs.most_blocks(cap)
    if wstates is not None and wslot is None and step < w_end - w_begin:  # every few windows' states over several launches
        wslot = torch.full((w_end,), -1, dtype=torch.int32, device=pk.device)
        at = wslot[w_begin::wstate_stride]
        at.copy_(torch.arange(at.shape[0], dtype=torch.int32, device=pk.device))
    for wa in range(w_begin, w_end, step):
        wb = min(wa + step, w_end)
        clip = 0 if whole_runs else ((_lib.BP_CLIP_BEGIN if wa == w_begin else 0)
                                     | (_lib.BP_CLIP_END if wb == w_end else 0))
        code = lib.bp_propagate(ptr(pk.spins), pk.n, ptr(pk.segs), ptr(pk.seg64), ptr(windows_dev), wa, wb, ptr(state),
                                ptr(wstates), wstate_stride, ptr(wslot), ptr(runs.runs) if z is not None else None,
                                runs.n_runs if z is not None else 0, ptr(z), cap, clip, max_ctas, ptr(status), stream)
        _lib.check(code, "bp_propagate")
        if z is not None:
            code = lib.bp_readout(ptr(pk.spins), ptr(pk.sens), pk.n, pk.n_coils, ptr(pk.segs), ptr(pk.seg64),
                                  ptr(windows_dev), wa, wb, ptr(runs.runs), runs.n_runs, ptr(runs.subs), runs.n_subs,
                                  most_subs, ptr(z), cap, clip, ptr(raw), stream)
            _lib.check(code, "bp_readout")
    return z if step >= w_end - w_begin else None


def finish_signal(pk: Packed, raw: torch.Tensor) -> torch.Tensor:
    """(C, A) complex64 on the device: the float64 sums demodulated by exp(-i psi)."""
    out = torch.empty(pk.n_coils, max(pk.n_adc, 1), dtype=torch.complex64, device=pk.device)
    code = _lib.lib().bp_signal_finish(ptr(raw), ptr(pk.psi), pk.n_adc, pk.n_coils, ptr(out), _lib.stream_ptr())
    _lib.check(code, "bp_signal_finish")
    return out[:, : pk.n_adc]


def plan_replacing(pk: Packed, spans):
    """Windows (host array and device copy) with breaks at every span's start and end, and the window ranges
    [(w_begin, w_end)] stepped before each span and after the last, for ``forward_replacing``."""
    S = pk.flags.shape[0]
    breaks = np.zeros(S, dtype=np.uint8)
    for s, k in spans:
        breaks[s] = 1
        if s + k < S:
            breaks[s + k] = 1
    samp = _lib.lib().bp_forward_samp_max(pk.n_coils)
    windows = plan_windows(pk.flags, samp, breaks=breaks)
    starts = windows[:, 0]
    ranges, w = [], 0
    for s, k in spans:
        wa = int(np.searchsorted(starts, s))
        ranges.append((w, wa))
        w = int(np.searchsorted(starts, s + k))
    ranges.append((w, windows.shape[0]))
    return windows, torch.from_numpy(windows).to(pk.device), ranges


def forward_replacing(pk: Packed, state: torch.Tensor, spans, apply, raw: torch.Tensor | None,
                      status: torch.Tensor, max_ctas: int = 0, plan=None, events=None) -> None:
    """The forward over all segments, where each span ``(start, length)`` of ``spans`` (sorted, disjoint, no ADC
    inside) is not stepped but replaced by ``apply(i)`` (launching the replacement of span i on the state).
    Windows are planned with breaks at every span's start and end (``plan_replacing``, or ``plan`` when given), so
    a span is a whole run of windows. ``events``: a list that receives a (start, end) pair of recorded CUDA events
    around every forward launch (the stepped part's device time)."""
    _, wdev, ranges = plan or plan_replacing(pk, spans)

    def step(wa, wb):
        if wb <= wa:
            return
        if events is not None:
            e = (torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
            e[0].record()
        run_forward(pk, state, wdev, wa, wb, raw, status, max_ctas=max_ctas)
        if events is not None:
            e[1].record()
            events.append(e)

    for i in range(len(spans)):
        step(*ranges[i])
        apply(i)
    step(*ranges[-1])


def forward_spans(pk: Packed, state: torch.Tensor, plan, spans, raw: torch.Tensor | None, status: torch.Tensor,
                  max_ctas: int = 0) -> None:
    """``forward_replacing`` in one native call: ``spans`` is a ctypes array of ``_lib.BpSpan`` (one per span of
    ``plan``, from ``plan_replacing``), launched in order by ``bp_forward_spans``."""
    _, wdev, ranges = plan
    if len(ranges) == 1:  # nothing is replaced: the stepped forward
        run_forward(pk, state, wdev, *ranges[0], raw, status, max_ctas=max_ctas)
        return
    rng = np.ascontiguousarray(np.asarray(ranges, dtype=np.int32).reshape(-1, 2))
    n_spans = rng.shape[0] - 1
    # the first sample of every run of samples, of as many ranges at a time as Z_BYTES holds
    runs, z, run_at, cap = None, None, None, 0
    if raw is not None:
        runs = pk.sample_runs()
        starts = plan[0][:, 0]
        first = [int(starts[wa]) if wa < len(starts) else pk.flags.shape[0] for wa, _ in ranges] + [pk.flags.shape[0]]
        run_at = np.ascontiguousarray(np.searchsorted(runs.starts, first), dtype=np.int32)
        cap = min(runs.n_runs, max(Z_BYTES // (8 * max(pk.n, 1)), 1))
        if not pk.windowed() and 0 < int(np.diff(run_at).max()) <= cap:
            z = torch.empty(cap, pk.n, 2, dtype=F32, device=pk.device)
    args = (ptr(pk.spins), ptr(pk.sens), pk.n, pk.n_coils, ptr(pk.segs), ptr(pk.seg64), ptr(wdev), rng.ctypes.data, n_spans,
            ctypes.addressof(spans) if n_spans else None, ptr(state), ptr(raw), max_ctas)
    if z is None:
        code = _lib.lib().bp_forward_spans(*args, ptr(status), _lib.stream_ptr())
    else:
        code = _lib.lib().bp_forward_spans_readout(*args, ptr(runs.runs), runs.n_runs, ptr(runs.subs), runs.n_subs,
                                                   runs.most_blocks(cap), run_at.ctypes.data, ptr(z), cap, ptr(status),
                                                   _lib.stream_ptr())
    _lib.check(code, "bp_forward_spans")


def forward(case, device, max_ctas: int = 0):
    """Signal (C, A) complex64 and m (N, 3) float32, both on the CPU, of a case (``oracle.bloch.Case``-like)."""
    samp = _lib.lib().bp_forward_samp_max(case.coils.shape[1])
    if samp <= 0:
        raise ValueError(f"at most {_lib.BP_MAX_COILS} coils, got {case.coils.shape[1]}")
    pk, state = pack_with_state(case, device)
    windows = plan_windows(pk.flags, samp)
    wdev = torch.from_numpy(windows).to(device).contiguous()
    raw = torch.zeros(max(pk.n_adc, 1), 2 * pk.n_coils, dtype=F64, device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    run_forward(pk, state, wdev, 0, windows.shape[0], raw if pk.n_adc else None, status, max_ctas=max_ctas)
    sig = finish_signal(pk, raw)
    _lib.check_status(status, "bp_forward")  # (waits for the kernels)
    return sig.cpu(), final_m(state)
