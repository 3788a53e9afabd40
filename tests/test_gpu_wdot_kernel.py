"""Which kernel serves a batch, as the library tells it, and what the block-size tuning
leaves where it is not the warp-per-cell one: its default, not the noise of timing one
launch three times."""
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_kernel_of_a_batch():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    c1, c2, c5 = (Chemistry.from_config(c) for c in ("c1", "c2", "c5"))
    assert {c1.wdot_kernel(n) for n in (0, 1, 1000, 10**6)} == {"small"}
    assert {c5.wdot_kernel(n) for n in (0, 1, 1000, 10**6)} == {"warp"}      # too few warps fit an SM
    assert [c2.wdot_kernel(n) for n in (1, 145 * sms - 1, 145 * sms, 256 * sms, 256 * sms + 1, 290 * sms, 10**6)] == \
        ["warp", "warp", "cell", "cell", "warp", "cell", "cell"]


@pytest.mark.parametrize("name,n", [("c2", 2000), ("c2", 30000), ("c5", 2000), ("c1", 2000)])
def test_block_size_of_a_sample(name, n):
    chem = Chemistry.from_config(name)
    T, p, Y = (torch.from_numpy(a).cuda() for a in (mechgen.c1_states(n) if name == "c1" else
                                                     mechgen.c2_states(n, chem.mech, seed=1)))
    t = chem.wdot_autotune(T, p, Y)
    assert t["wdot_threads"] in ((64, 128, 256) if chem.wdot_kernel(n) == "warp" else (0,))
    assert t["jac_threads"] in (64, 128, 256)
