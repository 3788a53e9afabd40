"""The thread-per-cell kernels of the tabulated path at the edges of their ranges.

Batches on both sides of the size where the general loop changes kernels and
ragged last warps, against the same cells in small batches (the warp kernel):
equal bit for bit where every operation is an IEEE one, 1e-12 of the cell's
largest rate where falloff reactions take powers and logarithms.  Non-finite
concentrations give the same non-finite rates on both."""
import copy
import os

import numpy as np
import pytest

from flint_gb300 import mechgen, tables
from flint_gb300.mech import Mechanism
from oracle.oracle import TableOracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def mechanism(name):
    if name == "c2_no_falloff":
        m = copy.deepcopy(mechgen.load("c2"))
        m.reactions = [r for r in m.reactions if r.rtype < 2]
        # an explicit collider: every other species has efficiency zero
        tb = [r for r in m.reactions if r.rtype == 1]
        tb[0].collider, tb[0].efficiencies = "CO", None
        return m
    return mechgen.load("c2") if name == "c2" else Mechanism.load(os.path.join(GOLD, f"mech_{name}.json"))


def states(m, n, seed):
    T, p, Y = mechgen.c2_states(n, m, seed=seed)
    T = np.clip(T, 300.0, 2990.0)
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    return torch.from_numpy(T).cuda(), torch.from_numpy(np.ascontiguousarray(rho[:, None] * Y)).cuda()


def small_batches(f, *arrays, size=1000):
    return torch.cat([f(*[a[i:i + size].contiguous() for a in arrays]) for i in range(0, arrays[0].shape[0], size)])


@pytest.mark.parametrize("name", ["c2_no_falloff", "c2", "pelucchi", "tsr_rich_31"])
@pytest.mark.parametrize("n", [3647, 3648, 3649, 5003])
def test_general_loop(name, n):
    m = mechanism(name)
    gpu = tables.Tables(tables.generate(m, 1, 3000))
    T, roi = states(m, n, n)
    w = gpu.chemistry_source(roi, T)
    w0 = small_batches(lambda r, t: gpu.chemistry_source(r, t), roi, T)
    if name == "c2_no_falloff":
        assert torch.equal(w, w0)
        assert np.array_equal(w.cpu().numpy(), TableOracle(gpu.t).general(roi.cpu().numpy(), T.cpu().numpy()))
    else:
        assert ((w - w0).abs().amax(1) / (w0.abs().amax(1) + 1e-300)).max() < 1e-12
    Z = torch.cat([roi, T[:, None]], 1).contiguous()
    F, F0 = gpu.rhs_native(Z), small_batches(lambda z: gpu.rhs_native(z), Z)
    assert ((F - F0)[:, :-1].abs().amax(1) / (F0[:, :-1].abs().amax(1) + 1e-300)).max() < 1e-12
    # dT/dt: a sum over the species, on the scale of its absolute terms (|e_k| < 5e8
    # J/kg, cv > 300 J/kg/K)
    scale = 5e8 * F0[:, :-1].abs().sum(1) / (300.0 * roi.sum(1))
    assert ((F - F0)[:, -1].abs() / (scale + 1e-300)).max() < 1e-12


@pytest.mark.parametrize("value", [float("inf"), float("nan"), -1e-3, 0.0, 1e-310])
def test_odd_concentrations(value):
    m = mechanism("c2_no_falloff")
    gpu = tables.Tables(tables.generate(m, 1, 3000))
    T, roi = states(m, 3700, 5)
    for i in range(m.ns):
        roi[7 * i, i] = value
    w = gpu.chemistry_source(roi, T)
    w0 = small_batches(lambda r, t: gpu.chemistry_source(r, t), roi, T)
    assert torch.equal(w.isnan(), w0.isnan())
    assert torch.equal(w.nan_to_num(), w0.nan_to_num())


@pytest.mark.parametrize("ndim", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 31, 33, 5003])
def test_cons2prim(n, ndim):
    m = mechanism("c2")
    t = tables.generate(m, 1, 3000)
    gpu = tables.Tables(t)
    T, roi = states(m, n, 9 + n)
    rng = np.random.default_rng(n)
    rho = roi.sum(1)
    u = torch.from_numpy(rng.normal(0.0, 200.0, (n, ndim))).cuda()
    E = torch.from_numpy(rng.uniform(1e5, 4e6, n)).cuda()
    cons = torch.cat([roi, rho[:, None] * u, (rho * E)[:, None]], 1).contiguous()
    prim, T1 = gpu.cons2prim(cons, T)
    ref, Tref = TableOracle(t).cons2prim(cons.cpu().numpy(), T.cpu().numpy())
    assert np.array_equal(prim.cpu().numpy(), ref) and np.array_equal(T1.cpu().numpy(), Tref)
