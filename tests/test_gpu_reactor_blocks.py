"""Reactor, matrices in shared memory: the block sizes that follow from the cell count.

Fewer cells than warps run in smaller blocks, two or more rounds of 12 warps on every
multiprocessor in blocks of 12.  The cells are independent and the arithmetic is that of
the layout with 8 warps and global matrices, which keeps its block size: every result has
the same bits (tolerance none).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GLOBAL = 2


def _count(where):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return {"one": 1, "below_a_warp_each": sms - 1, "two_warps": sms + 1, "seven_warps": 7 * sms - 3,
            "below_wide": 24 * sms - 1, "wide": 24 * sms, "wide_ragged": 36 * sms + 5}[where]


@pytest.mark.parametrize("where", ["one", "below_a_warp_each", "two_warps", "seven_warps", "below_wide", "wide",
                                   "wide_ragged"])
def test_block_sizes_compute_the_same_bits(where):
    from flint_gb300 import mechgen
    from flint_gb300.api import Chemistry
    chem = Chemistry.from_config("c2")
    T0, p, Y0, dt = mechgen.c3_states(_count(where), chem.mech, seed=47)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    pd, dtd = cuda(p), cuda(dt)
    out = []
    for lay in (0, GLOBAL):
        chem.set_tuning(lay, 0, 0)
        T, Y = cuda(T0), cuda(Y0)
        st, ns = chem.reactor_advance(T, pd, Y, dtd, max_steps=200000)
        torch.cuda.synchronize()
        out.append([a.cpu().numpy() for a in (T, Y, st, ns)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert (out[0][2] == 0).all()
