"""bench.py's roofline names the kernel that the library says serves the batch, with that
kernel's operation count (host only: the library's answer is given)."""
import os
import sys

import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), ".."))
import bench  # noqa: E402


class Chem:
    def __init__(self, name, cell_from):
        self.mech = type("M", (), {"name": name})
        self.cell_from = cell_from

    def wdot_kernel(self, n):
        return "cell" if n >= self.cell_from else "warp"


C2, C5 = "synthetic-31sp-160r", "synthetic-54sp-320r"


@pytest.mark.parametrize("n,kernel,count", [(22039, "k_wdot_warp<0>", "rhs"), (22040, "k_wdot_cell", "cell"),
                                            (32767, "k_wdot_cell", "cell")])
def test_source_terms(n, kernel, count):
    assert bench.kernel_and_flops(Chem(C2, 22040), n, False, False) == (kernel, bench.KINETICS_FLOPS[C2][count])


def test_others():
    never = Chem(C5, 1 << 62)
    assert bench.kernel_and_flops(never, 10**6, False, False) == ("k_wdot_warp<0>", bench.KINETICS_FLOPS[C5]["rhs"])
    assert bench.kernel_and_flops(Chem(C2, 1), 10**6, True, False) == ("k_wdot_warp<1>", bench.KINETICS_FLOPS[C2]["jac"])
    assert bench.kernel_and_flops(Chem(C2, 1), 10**6, False, True) == ("ytf_<mech>_kernel", bench.GENERATED_FLOPS[C2]["rhs"])
    assert bench.kernel_and_flops(Chem("unknown", 1), 10, False, False) is None
