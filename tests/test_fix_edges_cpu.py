"""The fixed-point primitives of the kinetics (csrc/flint_fix.cuh) on the host, at the
arguments where their rounding carries: a conversion to double is a single rounding
everywhere (2^-53), also where it rounds up to a power of two."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def values(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_edges")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(CUDA, "include"), "-I",
                    os.path.join(HERE, "..", "flint_gb300", "csrc"), "-o", exe,
                    os.path.join(HERE, "fix_edges_host.cpp")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {k.strip(): float(v) for k, v in (line.split("=") for line in out.splitlines())}


def test_conversion_that_rounds_up_to_a_power_of_two(values):
    assert values["fix2d_carry"] <= 2.0 ** -53
    assert (values["fix2d_one"], values["fix2d_four"], values["fix2d_minus"]) == (1.0, 4.0, -1.0)


def test_exp2_below_the_normal_range(values):
    """Cut to a subnormal number: less than one unit (and 2^-5 of the evaluation's)."""
    assert values["exp2_subnormal"] <= 1.0 + 2.0 ** -5
