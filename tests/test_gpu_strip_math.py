"""The FP64 strip walk's reciprocal and exponential against 80-bit values, beside
CUDA's division and exp().

Bounds, in units of the last place (ulp): the reciprocal is one rounding (0.5) of
a value good to the cube of its seed's error (a seed of 19 bits leaves 2^-57, a
sixteenth of the smallest ulp).  The exponential is one rounding (0.5) of
h (1 + q), q below 6.8e-4: the table's low part and the roundings inside q give
0.005 together, the polynomial's rounded 1/6 (2.4e-7 of r^3/6) 0.115 and its
remainder 0.012; beyond t = 50 the rounded step lets r grow to 8.6e-4 and those
two to 0.23 and 0.04."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from slsimlib_b200.build import NVCC_FLAGS, nvcc

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "strip_math_test.cu")


@pytest.fixture(scope="module")
def strip_math(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("strip_math") / "strip_math.so")
    subprocess.run([nvcc(), *NVCC_FLAGS, "-shared", SRC, "-o", lib], check=True, timeout=300)
    f = C.CDLL(lib).strip_math
    f.argtypes = [C.c_void_p, C.c_size_t, C.c_void_p]

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.zeros((4, len(x)))
        assert f(x.ctypes.data, len(x), out.ctypes.data) == 0
        return out

    return run


def _ulps(got, exact):
    near = exact.astype(np.float64)
    return np.abs((got.astype(np.longdouble) - exact) / np.spacing(np.abs(near))).astype(np.float64)


@pytest.mark.gpu
def test_reciprocal(strip_math):
    r = np.random.default_rng(1)
    x = np.concatenate([10 ** r.uniform(-20, 12, 1 << 20), 2.0 ** np.arange(-66, 41), r.uniform(1, 2, 1 << 18),
                        np.nextafter(2.0 ** np.arange(-66, 41), 0), np.nextafter(2.0 ** np.arange(-66, 41), 1e300)])
    rcp, div, _, _ = strip_math(x)
    exact = 1 / x.astype(np.longdouble)
    assert _ulps(rcp, exact).max() <= 0.5 + 1 / 16
    assert np.mean(rcp != div) < 1 / 16


@pytest.mark.gpu
def test_exponential(strip_math):
    r = np.random.default_rng(2)
    step = np.log(2.0) / 512
    k = np.arange(0, 36000)
    x = np.concatenate([[0.0, 2.0 ** -60, 1e-300, 5e-324, 50.0], r.uniform(0, 1, 1 << 19), r.uniform(0, 50, 1 << 20),
                        10 ** r.uniform(-12, 1.6, 1 << 19), k * step, (k + 0.5) * step,
                        np.nextafter((k + 0.5) * step, 0), np.nextafter((k + 0.5) * step, 100)])
    x = x[x <= 50]
    _, _, mine, cuda = strip_math(x)
    exact = np.exp(-x.astype(np.longdouble))
    assert mine[0] == 1.0
    assert _ulps(mine, exact).max() <= 0.65
    assert _ulps(mine, exact).max() <= _ulps(cuda, exact).max()
    assert _ulps(mine, exact).mean() <= _ulps(cuda, exact).mean()
    x = r.uniform(50, 700, 1 << 20)
    _, _, mine, _ = strip_math(x)
    assert _ulps(mine, np.exp(-x.astype(np.longdouble))).max() <= 0.8
    far = np.array([700.0, 701.0, 745.2, 1e6, 1e300, np.inf])
    _, _, mine, _ = strip_math(far)
    assert np.all((mine >= 0) & (mine < 1e-303))


@pytest.mark.gpu
def test_exponential_of_nans(strip_math):
    bits = np.array([0x7FF8000000000000, 0xFFF8000000000000, 0xFFFFFFFFE0000000, 0xFFFFFFFFFFFFFFFF, 0x7FF0000000000001,
                     0xFFF0000080000000], dtype=np.uint64)
    rcp, _, mine, _ = strip_math(bits.view(np.float64))
    assert np.all(np.isnan(rcp))
    neg = bits >> np.uint64(63) == 1  # (a positive NaN is held at 700, as a large number is)
    assert np.all(np.isnan(mine[neg]))
    assert np.all((mine[~neg] >= 0) & (mine[~neg] < 1e-303) | np.isnan(mine[~neg]))
