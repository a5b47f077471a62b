"""The native packing of a case against the same arithmetic in torch: bit for bit (one rounding from float64)."""

import numpy as np
import pytest
import torch

from blochparty_b200 import _lib, engine

pytestmark = pytest.mark.gpu
F32, F64 = torch.float32, torch.float64


@pytest.mark.parametrize("n", [1, 127, _lib.BP_PACK_BLOCK, 4 * _lib.BP_PACK_BLOCK, 4 * _lib.BP_PACK_BLOCK + 1,
                               70 * _lib.BP_PACK_BLOCK + 77])
@pytest.mark.parametrize("dtype,coils,m0", [(F64, 8, False), (F32, 3, True), (F64, 13, True), (torch.float16, 1, False)])
def test_spins(n, dtype, coils, m0):
    """Blocks of spins, one thread and several, float32, float64 and other inputs, strided and conjugated ones."""
    g = torch.Generator().manual_seed(n)
    rnd = lambda *s: (torch.rand(*s, generator=g, dtype=F64) + 0.1).to(dtype)
    pos, pd, t1, t2, db0, b1 = rnd(3, n).T, rnd(n), rnd(n, 2)[:, 0], rnd(n), -rnd(n), rnd(n)
    c = torch.complex(rnd(coils, n).double(), rnd(coils, n).double()).T
    c = (c.to(torch.complex64) if dtype == F32 else c).conj()
    m = rnd(n, 3) if m0 else None
    dev = torch.device("cuda", 0)
    spins, sens, state, extent = engine._upload_spins(pos, pd, t1, t2, db0, b1, c, m, dev, True)
    want_spins, want_sens = engine.pack_spins(pos, pd, t1, t2, db0, b1, c.resolve_conj(), "cpu")
    assert torch.equal(spins.cpu(), want_spins) and torch.equal(sens.cpu(), want_sens)
    assert torch.equal(state.cpu(), engine.initial_state(pd, m, "cpu"))
    assert np.array_equal(extent, want_spins.abs().amax(1).numpy())
    m_dev = engine.final_m(state)
    assert torch.equal(m_dev, engine.final_m(state.cpu()))


def test_extent_keeps_a_nan():
    n = engine._lib.BP_PACK_BLOCK * 12
    v = torch.ones(n, dtype=F64)
    b1 = v.clone()
    b1[7] = float("nan")
    out = engine._upload_spins(torch.ones(n, 3, dtype=F64), v, v, v, v, b1, torch.ones(n, 1, dtype=torch.complex64), None,
                               torch.device("cuda", 0), False)
    assert np.isnan(out[3][7]) and (out[3][:7] == 1).all()
