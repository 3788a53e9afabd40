"""The fixed-point kinetics at the last numbers below powers of two, where the seed of
1/T is taken from an all-ones significand, and reactors whose temperature crosses the
upper end of the range (one cell on both paths in turn), against the oracle.  Bars as
in test_gpu_parity.py."""
import os

import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry
from flint_gb300.mech import Mechanism
from flint_gb300.native import reactor_opts
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


@pytest.mark.parametrize("repeat", [9, 1400])      # a warp per cell, a thread per cell
def test_temperatures_below_powers_of_two(repeat):
    m = mechgen.load("c2")
    T = np.concatenate([2.0 ** k * (1.0 - 2.0 ** -53 * np.array([1, 2, 3, 2 ** 28, 2 ** 29, 2 ** 29 + 1, 2 ** 30]))
                        for k in (8, 9, 10, 11, 12)])
    T = np.repeat(T, repeat)[:24000 if repeat > 9 else None]
    n = T.size
    rng = np.random.default_rng(8)
    p, Y = rng.uniform(1.0, 40.0, n) * 101325.0, rng.dirichlet(np.full(m.ns, 0.3), size=n)
    w_o, ws_o, cp_o, h_o = Oracle(m).wdot_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    cp, h = torch.empty_like(Tt), torch.empty_like(Tt)
    w = Chemistry(m).wdot(Tt, pt, Yt, cp=cp, h=h)[0].cpu().numpy()
    assert (np.abs(w - w_o.reshape(n, -1)) / (ws_o.reshape(n, -1) + 1e-300)).max() < 1e-12
    np.testing.assert_allclose(cp.cpu().numpy(), cp_o, rtol=1e-13)
    assert np.max(np.abs(h.cpu().numpy() - h_o) / (np.abs(h_o) + cp_o * T)) < 1e-13


@pytest.mark.parametrize("volume", [False, True])
@pytest.mark.parametrize("n", [60, 4000])          # blocks of few cells, 12 warps a block
def test_reactor_across_the_end_of_the_range(volume, n):
    """The mechanism's range ends at 5,000 K; the gas passes it upwards."""
    m = Mechanism.load(os.path.join(GOLDEN, "mech_pelucchi.json"))
    rng = np.random.default_rng(9)
    T = rng.uniform(4900.0, 5700.0, n)
    p = rng.uniform(5.0, 40.0, n) * 101325.0
    Y = rng.dirichlet(np.full(m.ns, 1.0), size=n)
    dt = 10.0 ** rng.uniform(-9.0, -8.0, n)
    few = slice(0, 60)
    opts = dict(rtol=1e-12, atol=1e-18, max_steps=400000, tmin=200.0, tmax=9000.0, constant_volume=volume)
    T_x, Y_x, st_x, _ = Oracle(m).reactor_advance(T[few], p[few], Y[few], dt[few], reactor_opts(**opts))
    assert (st_x == 0).all()
    assert ((T[few] > 5000.0) & (T_x < 5000.0)).sum() > 5 or ((T[few] < 5000.0) & (T_x > 5000.0)).sum() > 5
    Tt, pt, Yt, dtt = (torch.from_numpy(a.copy()).cuda() for a in (T, p, Y, dt))
    st, _ = Chemistry(m).reactor_advance(Tt, pt, Yt, dtt, tmin=200.0, tmax=9000.0, constant_volume=volume)
    assert (st == 0).all()
    assert (np.abs(Tt.cpu().numpy()[few] - T_x) / T_x).max() < 1e-5
    assert np.abs(Yt.cpu().numpy()[few] - Y_x.reshape(60, -1)).max() < 1e-6
