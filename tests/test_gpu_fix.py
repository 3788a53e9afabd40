"""The fixed-point kinetics against the oracle at the edges of its ranges.

Temperatures at the ends of the fixed-point range, at the polynomials' middle
temperatures, at powers of two and outside the range (the FP64 path), for
mechanisms with and without the fixed-point image.  Bars as in
test_gpu_parity.py: 1e-12 of the sum of absolute terms for rates and Jacobian.
"""
import os

import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry, SPECIES_MAJOR
from flint_gb300.mech import Mechanism
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")

EDGES = [250.0, 255.9, 256.0, 300.0, 512.0, 999.9999999, 1000.0, 1000.0000001, 1024.0, 1390.0, 1690.0, 1710.0, 1999.9, 2000.1,
         2034.9, 2035.1, 2047.9999, 2048.0, 3500.0, 4095.9, 4096.0, 4999.9, 5000.0, 5000.1, 6000.0, 8191.9, 8192.0, 9000.0]


def load(name):
    return mechgen.load(name) if name in ("c2", "c5") else Mechanism.load(os.path.join(GOLDEN, f"mech_{name}.json"))


@pytest.mark.parametrize("name", ["c2", "c5", "tsr_rich_31", "pelucchi", "coria", "smooke", "troyes", "cross", "negative_A"])
def test_edges(name):
    mech = load("c2" if name == "negative_A" else name)
    if name == "negative_A":
        # duplicate reactions may carry a negative A; an elementary and a three-body one
        for j in (3, [r.rtype for r in mech.reactions].index(1)):
            mech.reactions[j].A = -mech.reactions[j].A
    rng = np.random.default_rng(41)
    T = np.repeat(EDGES, 9)
    n = T.size
    p = rng.uniform(1.0, 40.0, n) * 101325.0
    Y = rng.dirichlet(np.full(mech.ns, 0.3), size=n)
    chem, orc = Chemistry(mech), Oracle(mech)
    w_o, ws_o, cp_o, h_o = orc.wdot_batch(T, p, Y)
    _, J_o, Js_o = orc.wdot_jac_batch(T, p, Y)
    Tt, pt, Yt, Ys = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, p, Y, Y.T))
    cp, h, w2 = torch.empty_like(Tt), torch.empty_like(Tt), torch.empty_like(Yt)
    w, _, _ = chem.wdot(Tt, pt, Yt, cp=cp, h=h)
    ws, _, _ = chem.wdot(Tt, pt, Ys, layout=SPECIES_MAJOR)
    _, J = chem.wdot_jac(Tt, pt, Yt, wdot=w2)
    f = chem.rhs(Tt, pt, Yt)
    torch.cuda.synchronize()
    fine = np.isfinite(ws_o.reshape(n, -1)).all(1) & (ws_o.reshape(n, -1) < 1e280).all(1)
    assert fine.sum() > 0.9 * n

    def off(x, ref, scale):
        e = np.abs(x.cpu().numpy().reshape(n, -1) - ref.reshape(n, -1)) / (scale.reshape(n, -1) + 1e-300)
        return e[fine].max()

    assert off(w, w_o, ws_o) < 1e-12
    assert off(ws.t(), w_o, ws_o) < 1e-12
    assert off(w2, w_o, ws_o) < 1e-12
    assert off(J, J_o, Js_o) < 1e-12
    np.testing.assert_allclose(cp.cpu().numpy(), cp_o, rtol=1e-13)
    assert np.max(np.abs(h.cpu().numpy() - h_o) / (np.abs(h_o) + cp_o * T)) < 1e-13
    # dY/dt of the right-hand side is the rate over the density
    W = np.array([s.mw for s in mech.species])
    rho = p / (mech.r_eos * T * (Y / W).sum(1))
    assert off(f[:, :-1], w_o.reshape(n, -1) / rho[:, None], ws_o.reshape(n, -1) / rho[:, None]) < 1e-12


@pytest.mark.parametrize("bad", [np.nan, np.inf, -300.0, 0.0])
def test_bad_temperature_takes_the_general_path(bad):
    """A cell whose T is no temperature leaves its neighbours as they are."""
    mech = load("c2")
    chem = Chemistry(mech)
    T, p, Y = mechgen.c2_states(64, mech, seed=3)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    w0 = chem.wdot(Tt, pt, Yt)[0].cpu().numpy()
    Tb = Tt.clone()
    Tb[5] = bad
    w1 = chem.wdot(Tb, pt, Yt)[0].cpu().numpy()
    keep = np.arange(64) != 5
    assert np.array_equal(w0[keep], w1[keep])


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e6])
def test_unnormalised_mass_fractions(scale):
    """Mass fractions of any common scale: the concentrations depend on their
    ratios alone (bar: two roundings of the scaled inputs)."""
    mech = load("c2")
    chem = Chemistry(mech)
    T, p, Y = mechgen.c2_states(128, mech, seed=4)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    w0 = chem.wdot(Tt, pt, Yt)[0]
    w1 = chem.wdot(Tt, pt, Yt * scale)[0]
    _, ws_o, _, _ = Oracle(mech).wdot_batch(T, p, Y)
    assert (np.abs((w1 - w0).cpu().numpy()) / (ws_o.reshape(128, -1) + 1e-300)).max() < 1e-13


@pytest.mark.parametrize("name", ["c2", "c5", "tsr_rich_31", "pelucchi", "coria"])
@pytest.mark.parametrize("n", [22039, 22040, 22073])
def test_thread_per_cell(name, n):
    """Batches large enough for the thread-per-cell kernel, a ragged last warp and
    cells outside the fixed-point range among them, in both storage orders and as
    right-hand sides; constant volume against the warp kernel (a small batch)."""
    mech = load(name)
    rng = np.random.default_rng(n)
    T = rng.uniform(300.0, 4500.0, n)
    T[::37] = 8500.0
    T[n - 1] = 9000.0
    p = rng.uniform(1.0, 40.0, n) * 101325.0
    Y = rng.dirichlet(np.full(mech.ns, 0.3), size=n)
    chem, orc = Chemistry(mech), Oracle(mech)
    w_o, ws_o, cp_o, h_o = orc.wdot_batch(T, p, Y)
    w_o, ws_o = w_o.reshape(n, -1), ws_o.reshape(n, -1)
    Tt, pt, Yt, Ys = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, p, Y, Y.T))
    cp, h = torch.empty_like(Tt), torch.empty_like(Tt)
    w = chem.wdot(Tt, pt, Yt, cp=cp, h=h)[0].cpu().numpy()
    ws = chem.wdot(Tt, pt, Ys, layout=SPECIES_MAJOR)[0].cpu().numpy().T
    f = chem.rhs(Tt, pt, Yt)
    W = np.array([s.mw for s in mech.species])
    rho = p / (mech.r_eos * T * (Y / W).sum(1))
    rt = torch.from_numpy(rho).cuda()
    fv = chem.rhs_constv(Tt, rt, Yt)
    few = slice(n - 500, n)
    args = [a[few].contiguous() for a in (Tt, pt, rt, Yt)]
    f0, fv0 = chem.rhs(args[0], args[1], args[3]), chem.rhs_constv(args[0], args[2], args[3])
    torch.cuda.synchronize()
    assert (np.abs(w - w_o) / (ws_o + 1e-300)).max() < 1e-12
    assert (np.abs(ws - w_o) / (ws_o + 1e-300)).max() < 1e-12
    # cp and h on the scale of their absolute terms (a polynomial beyond its range
    # may pass through zero)
    tmid = np.array([s.tmid for s in mech.species])
    a = np.where((T[:, None] <= tmid)[:, :, None], np.array([s.low for s in mech.species]),
                 np.array([s.high for s in mech.species]))
    powers = T[:, None, None] ** np.arange(5)
    cps = mech.r_thermo * (Y / W * (np.abs(a[:, :, :5]) * powers).sum(2)).sum(1)
    hs = T * cps + mech.r_thermo * (Y / W * np.abs(a[:, :, 5])).sum(1)
    assert np.max(np.abs(cp.cpu().numpy() - cp_o) / cps) < 1e-13
    assert np.max(np.abs(h.cpu().numpy() - h_o) / hs) < 1e-13
    scale = ws_o / rho[:, None]
    f, fv = f.cpu().numpy(), fv.cpu().numpy()
    assert (np.abs(f[:, :-1] - w_o / rho[:, None]) / (scale + 1e-300)).max() < 1e-12
    # dT/dt: a sum over the species of h_k w_k, on the scale of its absolute terms
    # (|h_k/RT| < 400, cp/R > 2 per mole)
    tscale = T * 400.0 * (ws_o / W).sum(1) / (2.0 * rho * (Y / W).sum(1))
    for a, b in ((f, f0.cpu().numpy()), (fv, fv0.cpu().numpy())):
        assert (np.abs(a[few, :-1] - b[:, :-1]) / (scale[few] + 1e-300)).max() < 1e-12
        assert (np.abs(a[few, -1] - b[:, -1]) / tscale[few]).max() < 1e-12
