"""Mechanisms with three-body reactions and no falloff reaction.

The third-body sums are handed from lane to lane through shared memory; without a
falloff reaction no other step lies between.  Their number is such that a sum is
formed on another lane than its reaction's: source terms, right-hand side,
Jacobian and reactor of many cells against the oracle, and repeated calls bit for
bit.  Bars as in test_gpu_parity.py."""
import os

import numpy as np
import pytest

from flint_gb300.api import Chemistry
from flint_gb300.mech import Mechanism
from flint_gb300.native import reactor_opts
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def cells(m, n, seed):
    rng = np.random.default_rng(seed)
    T = rng.uniform(900.0, 2600.0, n)
    p = rng.uniform(1.0, 30.0, n) * 101325.0
    return T, p, rng.dirichlet(np.full(m.ns, 0.4), size=n)


@pytest.mark.parametrize("name", ["smooke", "troyes", "ecker"])
def test_kinetics(name):
    m = Mechanism.load(os.path.join(GOLDEN, f"mech_{name}.json"))
    tb = sum(r.rtype != 0 for r in m.reactions)
    assert tb and all(r.rtype < 2 for r in m.reactions) and (m.nr - tb) % 32
    n = 5000
    T, p, Y = cells(m, n, 3)
    chem, orc = Chemistry(m), Oracle(m)
    w_o, ws_o, _, _ = orc.wdot_batch(T, p, Y)
    _, J_o, Js_o = orc.wdot_jac_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    for i in range(4):
        w2 = torch.empty_like(Yt)
        w = chem.wdot(Tt, pt, Yt)[0].cpu().numpy()
        _, J = chem.wdot_jac(Tt, pt, Yt, wdot=w2)
        f = chem.rhs(Tt, pt, Yt).cpu().numpy()
        J, w2 = J.cpu().numpy(), w2.cpu().numpy()
        scale = ws_o.reshape(n, -1) + 1e-300
        assert (np.abs(w - w_o.reshape(n, -1)) / scale).max() < 1e-12
        assert (np.abs(w2 - w_o.reshape(n, -1)) / scale).max() < 1e-12
        assert (np.abs(f[:, :-1] * rho[:, None] - w_o.reshape(n, -1)) / scale).max() < 1e-12
        assert (np.abs(J.reshape(n, -1) - J_o.reshape(n, -1)) / (Js_o.reshape(n, -1) + 1e-300)).max() < 1e-12
        if i == 0:
            first = (w, w2, f, J)
        assert all(np.array_equal(a, b) for a, b in zip(first, (w, w2, f, J)))


@pytest.mark.parametrize("name", ["smooke", "troyes", "ecker"])
@pytest.mark.parametrize("n", [100, 4000])
def test_reactor(name, n):
    """Every cell over its own dt, against the oracle's solution at 1e-12 (the bounds of
    test_gpu_parity.py's reactor tests), and twice bit for bit."""
    m = Mechanism.load(os.path.join(GOLDEN, f"mech_{name}.json"))
    T, p, Y = cells(m, n, 4)
    dt = 10.0 ** np.random.default_rng(5).uniform(-7.5, -5.5, n)
    few = slice(0, 100)
    T_x, Y_x, st_x, _ = Oracle(m).reactor_advance(T[few], p[few], Y[few], dt[few],
                                                  reactor_opts(rtol=1e-12, atol=1e-18, max_steps=400000))
    assert (st_x == 0).all()
    chem = Chemistry(m)
    pt, dtt = torch.from_numpy(p).cuda(), torch.from_numpy(dt).cuda()
    out = []
    for _ in range(2):
        Tt, Yt = torch.from_numpy(T).cuda(), torch.from_numpy(Y).cuda()
        st, ns = chem.reactor_advance(Tt, pt, Yt, dtt)
        assert (st == 0).all()
        out.append((Tt.cpu().numpy(), Yt.cpu().numpy(), ns.cpu().numpy()))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    assert (np.abs(out[0][0][few] - T_x) / T_x).max() < 1e-5
    assert np.abs(out[0][1][few] - Y_x.reshape(100, -1)).max() < 1e-6
