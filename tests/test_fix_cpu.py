"""The fixed-point primitives of the kinetics (csrc/flint_fix.cuh) on the host.

The bars follow from the formats: exp2 rounds a 62-bit significand whose error
is below 2^-57, so the double is within 1/2 ulp + 2^-5; log2 keeps 62 bits with
three floored products (2^-59); log2 T in Q61 and 1/T in Q70 add their own last
place; a conversion to double is a single rounding, one to Q52 drops below 2^-52.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(CUDA, "include"), "-I",
                    os.path.join(HERE, "..", "flint_gb300", "csrc"), "-o", exe, os.path.join(HERE, "fix_host.cpp")],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {k.strip(): float(v) for k, v in (line.split("=") for line in out.splitlines())}


@pytest.mark.parametrize("key,bar", [("exp_ulp", 0.5 + 2.0 ** -5), ("log2", 2.0 ** -59), ("L", 2.0 ** -59),
                                     ("v", 2.0 ** -69), ("fix2d", 2.0 ** -53), ("d2fix", 2.0 ** -52)])
def test_error(errors, key, bar):
    assert errors[key] <= bar


def test_exact_values(errors):
    assert errors["exact"] == 1
