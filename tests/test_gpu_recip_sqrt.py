"""The kernels' 1/x and sqrt(x) (csrc/flint_fix.cuh) against extended precision.

Both end in one rounding (half a unit of the result) of a third-order step whose own
error follows from the 2^-20 of the SM's approximations: e^3 = 2^-60 of 1/x, 2^-7 of a
unit at most; 5/16 (2^-19)^3 = 2^-58.7 of sqrt(x), 2^-5 of a unit at most.  At the ends
of the fast range, and beyond it, where the library's operations take over: zero,
subnormal, huge, inf and NaN give CUDA's own results."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def run(x):
    from flint_gb300 import native
    xt = torch.from_numpy(x).cuda()
    y = torch.empty(x.size, 4, dtype=torch.float64, device="cuda")
    assert native.lib().flint_selftest_recip(x.size, C.c_void_p(xt.data_ptr()), C.c_void_p(y.data_ptr()), None) == 0
    torch.cuda.synchronize()
    return y.cpu().numpy()


def units(got, exact):
    """The error in units of the last place of the exact value (both normal)."""
    ld = np.longdouble
    return np.abs((got.astype(ld) - exact) / ld(2.0) ** (np.floor(np.log2(np.abs(exact))).astype(int) - 52))


def arguments():
    rng = np.random.default_rng(6)
    # bit patterns 0x030.. and 0x7c0.. are the ends of the fast range
    ends = np.array([0x03000000, 0x7c000000], dtype=np.uint64) << np.uint64(32)
    near = np.concatenate([e + np.arange(-300, 300).astype(np.int64).view(np.uint64) for e in ends]).view(np.float64)
    pow2 = 2.0 ** np.arange(-970, 960, dtype=np.float64)
    return np.concatenate([rng.uniform(1.0, 4.0, 300000), 2.0 ** rng.uniform(-960, 950, 200000), near, pow2,
                           np.nextafter(pow2, 0.0), np.nextafter(pow2, np.inf),
                           2.0 - 2.0 ** -52 * np.arange(1, 2000), 1.0 + 2.0 ** -52 * np.arange(0, 2000)])


def test_reciprocal():
    x = arguments()
    x = np.concatenate([x, -x])
    y = run(x)
    assert units(y[:, 0], 1 / x.astype(np.longdouble)).max() <= 0.5 + 2.0 ** -7


def test_square_root():
    x = arguments()
    y = run(x)
    assert units(y[:, 2], np.sqrt(x.astype(np.longdouble))).max() <= 0.5 + 2.0 ** -5


def test_arguments_of_the_library_path():
    tiny = np.finfo(float).tiny
    x = np.array([0.0, -0.0, 5e-324, 1e-310, tiny, tiny / 2, 1e300, 1.7e308, np.finfo(float).max, np.inf, -np.inf, np.nan,
                  -1e-310, -1e300, -np.nan])
    y = run(x)
    np.testing.assert_array_equal(y[:, 0], y[:, 1])
    positive = ~(x < 0)
    np.testing.assert_array_equal(y[positive, 2], y[positive, 3])
    assert np.isnan(run(np.array([-1.0, -1e-3, -1e300]))[:, 2]).all()
