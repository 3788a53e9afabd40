"""The small-mechanism kernel on the fixed-point image against the oracle.

chemistry_source (up to 16 species) and wdot (up to 8), with orders in power
form, reversible, third-body and falloff reactions; absent, trace and negative
species and temperatures outside the range (both take the FP64 path).  Bars as in
test_gpu_parity.py."""
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


def load(name):
    return mechgen.load(name) if name == "c1" else Mechanism.load(os.path.join(GOLDEN, f"mech_{name}.json"))


def cells(m, n, seed):
    rng = np.random.default_rng(seed)
    T = rng.uniform(300.0, 3000.0, n)
    p = rng.uniform(1.0, 20.0, n) * 101325.0
    Y = rng.dirichlet(np.full(m.ns, 0.5), size=n)
    Y[::5, 0] = 0.0
    Y[1::7, 1] = 1e-25
    Y[2::11, m.ns - 1] = 1e-290
    T[3::13] = 120.0
    T[4::17] = 8192.0
    return T, p, np.ascontiguousarray(Y)


@pytest.mark.parametrize("name", ["c1", "smooke", "troyes", "ecker", "tsr_cdf_13", "wd"])
@pytest.mark.parametrize("n", [1, 33, 4865, 9729, 40001])
def test_chemistry_source(name, n):
    m = load(name)
    T, p, Y = cells(m, n, n)
    chem, orc = Chemistry(m), Oracle(m)
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    roi = rho[:, None] * Y
    roi[5::19, 2] *= -1.0
    roi_t, Tt = torch.from_numpy(roi.copy()).cuda(), torch.from_numpy(T).cuda()
    w = chem.chemistry_source(roi_t, Tt).cpu().numpy()
    assert (roi_t.cpu().numpy() == np.clip(roi, 0.0, None)).all()
    c = np.clip(roi, 0.0, None)
    Yc = c / c.sum(1, keepdims=True)
    pc = c.sum(1) * m.r_eos * T * (Yc / W).sum(1)
    w_o, ws_o, _, _ = orc.wdot_batch(T, pc, Yc)
    fine = np.isfinite(ws_o.reshape(n, -1)).all(1)
    # (1e-11: the oracle is given a pressure and mass fractions formed from c, as in
    # test_c1_chemistry_source_clamps)
    assert (np.abs(w - w_o.reshape(n, -1)) / (ws_o.reshape(n, -1) + 1e-300))[fine].max() < 1e-11


@pytest.mark.parametrize("name", ["c1", "wd"])
@pytest.mark.parametrize("major", [False, True])
@pytest.mark.parametrize("n", [1, 4864, 9727, 30000])
def test_wdot(name, major, n):
    m = load(name)
    T, p, Y = cells(m, n, n + 1)
    Y[5::19, 2] *= -1e-3
    chem, orc = Chemistry(m), Oracle(m)
    w_o, ws_o, cp_o, h_o = orc.wdot_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, p, Y.T if major else Y))
    cp, h = torch.empty_like(Tt), torch.empty_like(Tt)
    w = chem.wdot(Tt, pt, Yt, layout=SPECIES_MAJOR if major else 0, cp=cp, h=h)[0].cpu().numpy()
    w = w.T if major else w
    assert (np.abs(w - w_o.reshape(n, -1)) / (ws_o.reshape(n, -1) + 1e-300)).max() < 1e-12
    hs = np.abs(h_o) + np.abs(cp_o) * T
    assert np.max(np.abs(cp.cpu().numpy() - cp_o) / (np.abs(cp_o) + 1000.0)) < 1e-13
    assert np.max(np.abs(h.cpu().numpy() - h_o) / hs) < 1e-13
