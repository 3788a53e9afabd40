"""Production rates written over the mass fractions (wdot = Y): the rates are those
of separate arrays, bit for bit, in every kernel and also for the cells outside the
fixed-point range, which their kernels evaluate on another path."""
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry, SPECIES_MAJOR

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name,n", [("c1", 3000), ("c2", 500), ("c2", 22073), ("c5", 500)])
@pytest.mark.parametrize("major", [False, True])
def test_rates_over_mass_fractions(name, n, major):
    m = mechgen.load(name)
    chem = Chemistry(m)
    T, p, Y = (torch.from_numpy(a).cuda() for a in (mechgen.c1_states(n) if name == "c1" else
                                                     mechgen.c2_states(n, m, seed=n)))
    T[::29] = 9000.0
    T[n - 1] = 100.0
    layout = SPECIES_MAJOR if major else 0
    Y = Y.t().contiguous() if major else Y
    ref = chem.wdot(T, p, Y, layout=layout)[0]
    own = Y.clone()
    chem.wdot(T, p, own, layout=layout, wdot=own)
    assert torch.equal(own, ref)
