"""Mechanisms near the shared memory of a block: what the kernels accepted with the
FP64 image staged they accept with the fixed-point one.

* 255 three-body reactions with 20 efficiencies each: the Jacobian's term lists grow
  with reactions x species x efficiencies and leave no room in a block;
* an FP64 image that leaves its block next to nothing.
"""
import copy

import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def many_third_bodies(per_reaction, name="c2"):
    m = mechgen.load(name)
    rng = np.random.default_rng(3)
    names = [s.name for s in m.species]
    plain = [r for r in m.reactions if r.rtype == 0]
    own = [r for r in m.reactions if r.rtype != 0]
    m.reactions = plain[:10] + own
    for i in range(255 - len(own)):
        r = copy.deepcopy(plain[i % len(plain)])
        r.rtype, r.default_eff = 1, 1.0
        r.efficiencies = {names[k]: float(e) for k, e in zip(rng.permutation(m.ns)[:per_reaction],
                                                             rng.uniform(1.5, 6.0, per_reaction))}
        m.reactions.append(r)
    return m


@pytest.mark.parametrize("per_reaction", [4, 20])
def test_jacobian_of_many_third_bodies(per_reaction):
    m = many_third_bodies(per_reaction)
    n = 300
    T, p, Y = mechgen.c2_states(n, m, seed=21)
    w_o, J_o, Js_o = Oracle(m).wdot_jac_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    chem = Chemistry(m)
    w = torch.empty_like(Yt)
    _, J = chem.wdot_jac(Tt, pt, Yt, wdot=w)
    # the scale of a sum of absolute terms; the error grows with the number of terms
    # (256 reactions a species at most: 2^-53 x 256 < 3e-14)
    assert (np.abs(J.cpu().numpy().reshape(n, -1) - J_o.reshape(n, -1)) / (Js_o.reshape(n, -1) + 1e-300)).max() < 1e-12
    _, ws_o, _, _ = Oracle(m).wdot_batch(T, p, Y)
    assert (np.abs(w.cpu().numpy().reshape(n, -1) - w_o.reshape(n, -1)) / (ws_o.reshape(n, -1) + 1e-300)).max() < 1e-12


def test_fp64_image_at_the_limit():
    """608 reactions on NASA-9 thermo: image and scratch fill a block's 227 KB but for
    less than 384 bytes."""
    m = mechgen.load("c2")
    for s in m.species:
        s.nasa9 = [[s.tlow, s.tmid, 0.0, 0.0] + list(s.low), [s.tmid, s.thigh, 0.0, 0.0] + list(s.high)]
    plain = [r for r in m.reactions if r.rtype == 0]
    while m.nr < 608:
        m.reactions.append(copy.deepcopy(plain[m.nr % len(plain)]))
    three = [r for r in m.reactions if r.rtype == 1]
    for r in three:
        r.efficiencies = {}
    for i in range(298):
        three[i // 30].efficiencies[m.species[i % 30].name] = 1.5 + i
    n = 200
    T, p, Y = mechgen.c2_states(n, m, seed=22)
    w_o, ws_o, _, _ = Oracle(m).wdot_batch(T, p, Y)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    chem = Chemistry(m)
    w = chem.wdot(Tt, pt, Yt)[0].cpu().numpy()
    f = chem.rhs(Tt, pt, Yt).cpu().numpy()
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    scale = ws_o.reshape(n, -1) + 1e-300
    assert (np.abs(w - w_o.reshape(n, -1)) / scale).max() < 1e-12
    assert (np.abs(f[:, :-1] * rho[:, None] - w_o.reshape(n, -1)) / scale).max() < 1e-12
