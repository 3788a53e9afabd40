"""Where the tabulated loop changes from a warp to a thread per cell: both sides of each
mechanism's own line give the same rates, and no batch just above a line takes much
longer than one just below."""
import copy
import os

import numpy as np
import pytest

from flint_gb300 import mechgen, tables
from flint_gb300.mech import Mechanism

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
GOLD = os.path.join(os.path.dirname(__file__), "golden")
NAMES = ["c2", "c2_no_falloff", "tsr_rich_31", "tsr_rich_31_no_falloff", "ecker", "troyes"]


def mechanism(name):
    base = name.replace("_no_falloff", "")
    m = copy.deepcopy(mechgen.load("c2") if base == "c2" else Mechanism.load(os.path.join(GOLD, f"mech_{base}.json")))
    if base != name:
        m.reactions = [r for r in m.reactions if r.rtype < 2]
    return m


def states(m, n, seed):
    T, p, Y = mechgen.c2_states(n, m, seed=seed)
    T = np.clip(T, 400.0, 2800.0)
    W = np.array([s.mw for s in m.species])
    rho = p / (m.r_eos * T * (Y / W).sum(1))
    return torch.from_numpy(T).cuda(), torch.from_numpy(np.ascontiguousarray(rho[:, None] * Y)).cuda()


@pytest.mark.parametrize("name", NAMES)
def test_same_rates_on_both_sides(name):
    m = mechanism(name)
    gpu = tables.Tables(tables.generate(m))
    T, roi = states(m, 12200, 3)
    whole = gpu.chemistry_source(roi, T)
    F = gpu.rhs_native(torch.cat([roi, T[:, None]], 1).contiguous())
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for rounds in (1, 4, 5, 6, 8, 9):
        n = min(8 * sms * rounds, 12200)
        w = gpu.chemistry_source(roi[:n].contiguous(), T[:n].contiguous())
        f = gpu.rhs_native(torch.cat([roi[:n], T[:n, None]], 1).contiguous())
        scale = whole[:n].abs().amax(1, keepdim=True) + 1e-300
        if "no_falloff" in name or name in ("ecker", "troyes"):
            assert torch.equal(w, whole[:n])
        assert ((w - whole[:n]).abs() / scale).max() < 1e-12
        assert ((f - F[:n])[:, :-1].abs() / scale).max() < 1e-12


@pytest.mark.parametrize("name", NAMES)
def test_no_step_in_the_time(name):
    """From three rounds of 8 cells on every multiprocessor to four, five, ... at most the
    round's share longer (4/3 at most; the bar leaves a fifth for the fit and the clock)."""
    m = mechanism(name)
    gpu = tables.Tables(tables.generate(m))
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def time_of(rounds):
        T, roi = states(m, 8 * sms * rounds - 3, 5)
        out = torch.empty_like(roi)
        for _ in range(3):
            gpu.chemistry_source(roi, T, omegadot=out)
        times = []
        for _ in range(7):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(10):
                gpu.chemistry_source(roi, T, omegadot=out)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return sorted(times)[3]

    t = [time_of(r) for r in range(3, 11)]
    for i in range(len(t) - 1):
        assert t[i + 1] < 1.2 * (i + 4) / (i + 3) * t[i], (i + 4, t)


@pytest.mark.parametrize("value", [float("inf"), float("nan"), -1e-3, 0.0, 1e-310])
def test_odd_concentrations_beyond_the_line(value):
    """Non-finite, negative and subnormal concentrations, with an explicit collider (every
    other species has efficiency zero): the thread-per-cell kernel as the other one."""
    m = mechanism("c2_no_falloff")
    three = [r for r in m.reactions if r.rtype == 1]
    three[0].collider, three[0].efficiencies = "CO", None
    gpu = tables.Tables(tables.generate(m, 1, 3000))
    T, roi = states(m, 12200, 5)
    for i in range(m.ns):
        roi[7 * i, i] = value
    w = gpu.chemistry_source(roi, T)
    w0 = torch.cat([gpu.chemistry_source(roi[i:i + 1000].contiguous(), T[i:i + 1000].contiguous())
                    for i in range(0, 12200, 1000)])
    assert torch.equal(w.isnan(), w0.isnan())
    assert torch.equal(w.nan_to_num(), w0.nan_to_num())
