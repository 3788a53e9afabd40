"""Orders in power form (small mechanisms, fixed-point image) against the oracle.

An irreversible reaction whose orders are not 0 to 3 is evaluated as one
exponential of log2 k + sum of order x log2 c, for orders up to 16.  Falloff and
three-body reactions in that form, also with the reactant absent, and orders with
concentrations so small that the sum leaves the format's 2^11 octaves.

Bar as in test_gpu_parity.py: 1e-12 of the sum of absolute terms; an exponent's
error is at most 16 x 2^-52 (three roundings of a concentration times the order),
which leaves two decades.
"""
import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BAR = 1e-12
N = 700


def states(m, seed):
    rng = np.random.default_rng(seed)
    T = rng.uniform(600.0, 2500.0, N)
    p = rng.uniform(1.0, 20.0, N) * 101325.0
    Y = rng.dirichlet(np.full(m.ns, 0.5), size=N)
    return T, p, np.ascontiguousarray(Y)


def compare(m, T, p, Y):
    """wdot and chemistry_source against the oracle."""
    chem, orc = Chemistry(m), Oracle(m)
    w_o, ws_o, _, _ = orc.wdot_batch(T, p, Y)
    w_o, ws_o = w_o.reshape(N, -1), ws_o.reshape(N, -1)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    w = chem.wdot(Tt, pt, Yt)[0].cpu().numpy()
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    s = chem.chemistry_source(torch.from_numpy(rho[:, None] * Y).cuda(), Tt).cpu().numpy()
    assert np.isfinite(w_o).all()
    assert (np.abs(w - w_o) / (ws_o + 1e-300)).max() < BAR
    # (a concentration formed from rho Y differs by two roundings from the oracle's)
    assert (np.abs(s - w_o) / (ws_o + 1e-300)).max() < 1e-11
    return w


@pytest.mark.parametrize("order", [0.5, 7.9, 8.0, 8.5, 12.5, 15.9, 16.0, 20.0])
def test_orders(order):
    m = mechgen.load("c1")
    m.reactions[0].orders = {"CH4": 1.0, "O2": order}
    T, p, Y = states(m, 11)
    compare(m, T, p, Y)


@pytest.mark.parametrize("rtype", [1, 2, 3])
def test_absent_reactant(rtype):
    m = mechgen.load("c1")
    r = m.reactions[0]
    r.rtype, r.efficiencies, r.default_eff = rtype, {"H2O": 6.0}, 1.0
    r.A0, r.b0, r.EaR0 = r.A * 50.0, r.b, r.EaR * 0.9
    r.troe = [0.6, 100.0, 2000.0, 5000.0] if rtype == 3 else None
    T, p, Y = states(m, 12)
    Y[::3, m.index("CH4")] = 0.0
    w = compare(m, T, p, Y)
    # CH4 takes part in the first reaction alone
    assert (w[::3, m.index("CH4")] == 0.0).all() and (w[1::3, m.index("CH4")] != 0.0).any()


@pytest.mark.parametrize("order,trace", [(15.0, 1e-17), (15.9, 1e-16), (11.0, 1e-17), (4.5, 1e-17)])
def test_exponent_beyond_the_format(order, trace):
    """Three factors of large order at trace concentrations: the rate vanishes."""
    m = mechgen.load("c1")
    m.reactions[0].orders = {"CH4": order, "O2": order, "N2": order}
    T, p, Y = states(m, 13)
    for s in ("CH4", "O2", "N2"):
        Y[::2, m.index(s)] = trace * (1.0 + np.arange(Y[::2].shape[0]) / N)
    compare(m, T, p, Y)


@pytest.mark.parametrize("value", [1e-18, 1e-25, 1e-120, 3e-300, -1e-12, -1e-25, 0.0])
@pytest.mark.parametrize("orders", [None, {"CH4": 1.0, "O2": 0.5}, {"CH4": 3.0, "O2": 7.5}, {"CH4": 2.0, "N2": -0.0, "O2": 0.25},
                                    {"CH4": 4.0, "O2": 1.0}])
def test_trace_and_undershoot(value, orders):
    """Trace species and the small negative mass fractions a flow solver leaves."""
    m = mechgen.load("c1")
    if orders:
        m.reactions[0].orders = orders
    chem, orc = Chemistry(m), Oracle(m)
    T, p, Y = states(m, 14)
    Y[::2, m.index("CH4")] = value
    Y[::3, m.index("CO")] = value
    w_o, ws_o, _, _ = orc.wdot_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    w = chem.wdot(Tt, pt, Yt)[0].cpu().numpy()
    err = np.abs(w - w_o.reshape(N, -1)) / (ws_o.reshape(N, -1) + 1e-290)
    if value < 0.0 and orders and orders["CH4"] == 4.0:
        # the kernels take a negative concentration to any order but 1, 2 and 3 as
        # absent, the oracle multiplies up to order 4; CH4 is in this reaction alone
        assert (w[::2, m.index("CH4")] == 0.0).all()
        err[::2, m.index("CH4")] = 0.0
    assert err.max() < BAR


@pytest.mark.parametrize("value", [1e-25, -1e-12])
def test_trace_and_undershoot_cost_no_second_path(value):
    """A million cells with such a reactant take the time of a million without (the
    FP64 path took five times as long; the bar is twice)."""
    m = mechgen.load("c1")
    chem = Chemistry(m)
    T, p, Y = (torch.from_numpy(a).cuda() for a in mechgen.c1_states(1000000))
    w = torch.empty_like(Y)

    def time_of(Y):
        times = []
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            chem.wdot(T, p, Y, wdot=w)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return sorted(times)[4]

    plain = time_of(Y)
    Yv = Y.clone()
    Yv[:, m.index("CH4")] = value
    assert time_of(Yv) < 2.0 * plain
