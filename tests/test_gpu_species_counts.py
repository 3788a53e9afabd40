"""Species counts around the width of a warp: ns + 1 unknowns take one slot a lane up
to 31 species and two beyond.  The 31-species mechanism with one, two and three inert
species added: source terms, right-hand sides of small and large batches, Jacobian and
reactor against the oracle (bars as in test_gpu_parity.py)."""
import copy

import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry
from flint_gb300.native import reactor_opts
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def widened(extra):
    m = mechgen.load("c2")
    for i in range(extra):
        s = copy.deepcopy(m.species[m.index("N2")])
        s.name, s.mw = f"INERT{i}", 40.0 + i
        m.species.append(s)
    return m


@pytest.mark.parametrize("extra", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [64, 33333])
def test_kinetics(extra, n):
    m = widened(extra)
    T, p, Y = mechgen.c2_states(n, m, seed=7)
    chem, orc = Chemistry(m), Oracle(m)
    w_o, ws_o, cp_o, _ = orc.wdot_batch(T, p, Y)
    w_o, ws_o = w_o.reshape(n, -1), ws_o.reshape(n, -1) + 1e-300
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    cp = torch.empty_like(Tt)
    w = chem.wdot(Tt, pt, Yt, cp=cp)[0].cpu().numpy()
    assert (np.abs(w - w_o) / ws_o).max() < 1e-12
    np.testing.assert_allclose(cp.cpu().numpy(), cp_o, rtol=1e-13)
    few = min(n, 64)
    f_o = np.array([orc.rhs(T[i], p[i], Y[i]) for i in range(few)])
    W = np.array([s.mw for s in m.species])
    rho = (p / (m.r_eos * T * (Y / W).sum(1)))[:few]
    # dT/dt on the scale of its absolute terms (|h_k/RT| < 400, cp/R > 2 per mole)
    scale = np.concatenate([ws_o[:few] / rho[:, None],
                            (T[:few] * 400.0 * (ws_o[:few] / W).sum(1) / (2.0 * rho * (Y[:few] / W).sum(1)))[:, None]], 1)
    f = torch.full((n, m.ns + 1), float("nan"), dtype=torch.float64, device="cuda")
    chem.rhs(Tt, pt, Yt, f=f)
    assert (np.abs(f.cpu().numpy()[:few] - f_o) / scale).max() < 1e-12
    rt = torch.from_numpy(rho).cuda()
    fv_o = np.array([orc.rhs_constv(T[i], rho[i], Y[i]) for i in range(few)])
    fv = torch.full((few, m.ns + 1), float("nan"), dtype=torch.float64, device="cuda")
    chem.rhs_constv(Tt[:few].contiguous(), rt, Yt[:few].contiguous(), f=fv)
    assert (np.abs(fv.cpu().numpy() - fv_o) / (1.5 * scale)).max() < 1e-12


@pytest.mark.parametrize("extra", [0, 1, 2])
def test_jacobian(extra):
    m = widened(extra)
    n = 200
    T, p, Y = mechgen.c2_states(n, m, seed=8)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    _, J_o, Js_o = Oracle(m).wdot_jac_batch(T, p, Y)
    J = torch.full((n, m.ns + 1, m.ns + 1), float("nan"), dtype=torch.float64, device="cuda")
    Chemistry(m).wdot_jac(Tt, pt, Yt, jac=J)
    err = np.abs(J.cpu().numpy().reshape(n, -1) - J_o.reshape(n, -1)) / (Js_o.reshape(n, -1) + 1e-300)
    assert err.max() < 1e-12


@pytest.mark.parametrize("extra", [0, 1, 2])
def test_reactor(extra):
    m = widened(extra)
    n = 128
    T, p, Y, dt = mechgen.c3_states(n, m, seed=9)
    T_x, Y_x, st_x, _ = Oracle(m).reactor_advance(T, p, Y, dt, reactor_opts(rtol=1e-12, atol=1e-18, max_steps=400000))
    Tt, pt, Yt, dtt = (torch.from_numpy(a).cuda() for a in (T, p, Y, dt))
    st, _ = Chemistry(m).reactor_advance(Tt, pt, Yt, dtt)
    assert (st == 0).all() and (st_x == 0).all()
    assert (np.abs(Tt.cpu().numpy() - T_x) / T_x).max() < 1e-5
    assert np.abs(Yt.cpu().numpy() - Y_x.reshape(n, -1)).max() < 1e-6
