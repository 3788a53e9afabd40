"""Warp sums whose value lies just below a power of two.

sum Y/W of a pure gas of molar mass 32 with a tiny undershoot of another species
is 2^-5 less a fraction of its last place: the conversion of the integer sum to a
double rounds up to the next power of two.  Rates, cp, h and the right-hand side
against the oracle, bars as in test_gpu_parity.py.
"""
import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", ["c2", "c5"])
def test_sum_below_a_power_of_two(name):
    m = mechgen.load(name)
    o2, n2 = m.index("O2"), m.index("N2")
    m.species[o2].mw = 32.0
    n = 256
    rng = np.random.default_rng(5)
    T, p = rng.uniform(1000.0, 2500.0, n), rng.uniform(1.0, 20.0, n) * 101325.0
    Y = np.zeros((n, m.ns))
    Y[:] = rng.uniform(0.0, 1e-21, (n, m.ns))
    Y[:, o2] = 1.0
    Y[:, n2] = -10.0 ** rng.uniform(-18.5, -16.5, n)
    chem, orc = Chemistry(m), Oracle(m)
    w_o, ws_o, cp_o, h_o = orc.wdot_batch(T, p, Y)
    _, J_o, Js_o = orc.wdot_jac_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    cp, h = torch.empty_like(Tt), torch.empty_like(Tt)
    w = chem.wdot(Tt, pt, Yt, cp=cp, h=h)[0]
    _, J = chem.wdot_jac(Tt, pt, Yt, wdot=torch.empty_like(Yt))
    f = chem.rhs(Tt, pt, Yt)
    torch.cuda.synchronize()
    w_o, ws_o = w_o.reshape(n, -1), ws_o.reshape(n, -1)
    assert (np.abs(w.cpu().numpy() - w_o) / (ws_o + 1e-300)).max() < 1e-12
    assert (np.abs(J.cpu().numpy().reshape(n, -1) - J_o.reshape(n, -1)) / (Js_o.reshape(n, -1) + 1e-300)).max() < 1e-12
    np.testing.assert_allclose(cp.cpu().numpy(), cp_o, rtol=1e-13)
    np.testing.assert_allclose(h.cpu().numpy(), h_o, rtol=1e-13, atol=1e-13 * np.abs(cp_o * T).max())
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    assert (np.abs(f.cpu().numpy()[:, :-1] - w_o / rho[:, None]) / (ws_o / rho[:, None] + 1e-300)).max() < 1e-12
