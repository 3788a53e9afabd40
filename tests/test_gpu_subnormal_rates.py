"""Rate constants below the normal range (2^-1022) are not lost.

One irreversible reaction of high activation temperature, cold; at a pressure that
makes its rate a normal number, or (power form) at one that leaves it subnormal.  The
reference is in extended precision (the oracle
forms A exp(-E/T) of an exponential that is itself subnormal).  A mechanism's
fixed-point range ends where its constants do; colder cells take the FP64 path, whose
exponential is cut at a unit of 2^-1074 before it is multiplied by A.  The power form
of small mechanisms goes on, and cuts the rate itself."""
import copy

import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name,n", [("c2", 400), ("c2", 23000), ("c1", 400)])
def test_subnormal_constants(name, n):
    m = copy.deepcopy(mechgen.load(name))
    r = m.reactions[0]
    m.reactions = [r]
    r.reversible, r.b, r.EaR = False, 0.0, 150000.0
    r.orders = {k: 1.5 for k in r.reactants} if name == "c1" else r.orders
    octaves = np.log2(r.A)
    # log2 k = octaves - EaR log2(e) / T between -1032 and -1010 in equal steps
    T = r.EaR / np.log(2.0) / (octaves + np.linspace(1010.0, 1032.0, n))
    rng = np.random.default_rng(1)
    Y = rng.dirichlet(np.full(m.ns, 3.0), size=n)
    p = np.full(n, 1e13 if name == "c2" else 1e5)
    Tt, pt, Yt = (torch.from_numpy(a).cuda() for a in (T, p, Y))
    w = Chemistry(m).wdot(Tt, pt, Yt)[0].cpu().numpy()
    ld = np.longdouble
    W = np.array([s.mw for s in m.species])
    k = ld(r.A) * np.exp(-ld(r.EaR) / T.astype(ld))
    c = (p / (m.r_eos * T * (Y / W).sum(1)))[:, None] * Y / W
    powers = np.ones(n, dtype=ld)
    for s, o in (r.orders or r.reactants).items():
        powers *= c[:, m.index(s)].astype(ld) ** ld(o)
    rate = k * powers
    unit = ld(2.0) ** -1074 * (ld(r.A) * powers if name == "c2" else 1)
    for s in list(r.reactants) + list(r.products):
        nu, mw = r.products.get(s, 0.0) - r.reactants.get(s, 0.0), W[m.index(s)]
        x = w[:, m.index(s)].astype(ld)
        # 2^-40: two roundings of a concentration and the exponent's 2^-44 octaves
        # (FP64); each product of a subnormal number is cut too
        bar = (ld(2.0) ** -40 * rate + unit) * abs(nu) * mw + ld(2.0) ** -1073 * mw
        assert (np.abs(x - rate * nu * mw) <= bar).all()
        assert (x != 0).all()
