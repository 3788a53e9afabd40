"""Surrogate's conservative projection for every number of elements (one build each).

The element rows are synthetic: row e holds the species e, e + ne, ... once and those of
row e - 1 1.2 times, so that the pivot search swaps rows, and the last of two or more
rows is empty.  B's smallest singular value is above 1.2^-8 of its largest, so G = B B^T
has a condition below 1e3 and one solve leaves 1e3 x 2^-52 = 2e-13 of the removed
residual, itself far below the amounts: bound 1e-12 of the largest amount.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _rows(ne, W):
    E = np.zeros((ne, W.size))
    for e in range(ne):
        if ne > 1 and e == ne - 1:
            break
        E[e, e::ne] += 1.0
        if e:
            E[e, e - 1::ne] += 1.2
    return E * W / 30.0


@pytest.mark.parametrize("ne", range(9))
def test_projection_conserves_every_element(ne):
    from flint_gb300 import mechgen
    from flint_gb300.api import Chemistry
    from flint_gb300.surrogate import Surrogate
    chem = Chemistry.from_config("c2")
    W = np.array([s.mw for s in chem.mech.species])
    E = _rows(ne, W)
    chem.mech.element_matrix = lambda: E
    one = lambda k, v: np.full(chem.ns + k, v, np.float32)  # noqa: E731
    sur = Surrogate(chem, {"x_mean": one(2, 0.0), "x_std": one(2, 1.0), "y_mean": one(1, 0.0), "y_std": one(1, 1e-4),
                           "bath": chem.mech.index("N2"), "domain": {}}, hidden=64, n_layers=3, seed=3)
    T0, p0, _, dt0 = mechgen.c3_states(256, chem.mech, seed=43)
    Y0 = np.random.default_rng(44).uniform(0.5, 1.0, (256, chem.ns))
    Y0[128:, ::5] = 1e-9     # these species are clipped where their increment is negative
    Y0 /= Y0.sum(1, keepdims=True)
    T, p, Y, dt = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T0, p0, Y0, dt0))
    sur.gate.update({"max_dT_resid": 1e30, "max_elem_resid": 1e30, "min_Y": -1e30, "T_lo": 0.0, "T_hi": 1e9,
                     "log10p_lo": -1e9, "log10p_hi": 1e9, "log10dt_lo": -1e9, "log10dt_hi": 1e9})
    st, ns, (acc, rej) = sur.advance(T, p, Y, dt)
    torch.cuda.synchronize()
    ok = (st.cpu().numpy() == 0) & (ns.cpu().numpy() == 0)
    Y1 = Y.cpu().numpy()
    assert ok.sum() == acc and ok[:128].all()
    assert (Y1[ok] >= 0.0).all()
    assert not np.array_equal(Y1[ok], Y0[ok])
    if ne:
        a0, a1 = (Y0 / W) @ E.T, (Y1 / W) @ E.T
        assert np.abs(a1[ok] - a0[ok]).max() <= 1e-12 * np.abs(a0).max()
