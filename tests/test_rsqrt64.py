"""The FP64 reciprocal square root of the far-field kernels (an FP32 seed and
one step of Householder's third-order iteration where the argument's leading
part is a normal float, the library's square root and division elsewhere)
against 1 / sqrt(x) in extended precision: mantissas all over, every exponent,
both ends of the seed's range, denormals, zeros, infinities, NaN and negative
arguments.

Five rounded operations, of which the products' errors enter halved: below 2
units in the last place."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fastercap_gb300 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rsqrt64(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rsqrt") / "librsqrt.so")
    subprocess.check_call([build.NVCC] + build.ARCH + ["-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                           os.path.join(HERE, "native", "rsqrt_check.cu"), "-o", out])
    lib = C.CDLL(out)
    lib.rsqrt64_all.argtypes = [C.c_int64, C.c_void_p, C.c_void_p]

    def run(x):
        x = np.ascontiguousarray(x, np.float64)
        y = np.empty_like(x)
        assert lib.rsqrt64_all(x.size, x.ctypes.data, y.ctypes.data) == 0
        return y

    return run


def ulps(x, y):
    want = 1 / np.sqrt(x.astype(np.longdouble))
    return np.abs(y.astype(np.longdouble) - want) / np.spacing(want.astype(np.float64)).astype(np.longdouble)


def test_mantissas(rsqrt64):
    x = np.concatenate([np.random.default_rng(1).uniform(1, 4, 1 << 20), np.linspace(1, 4, 1 << 16),
                        np.nextafter(2.0 ** np.arange(-30.0, 30.0), 0), np.nextafter(2.0 ** np.arange(-30.0, 30.0), 9e99)])
    assert ulps(x, rsqrt64(x)).max() < 2.0


def test_every_exponent(rsqrt64):
    e = np.arange(-1074, 1024)
    m = np.random.default_rng(2).uniform(1, 2, (64, e.size))
    m[0], m[1] = 1.0, 2 - 2.0**-52
    x = np.ldexp(m, e).ravel()  # denormals among them, rounded
    x = x[(x > 0) & np.isfinite(x)]
    assert ulps(x, rsqrt64(x)).max() < 2.0


@pytest.mark.parametrize("edge", [2.0**-125, 2.0**127])
def test_ends_of_the_seed_range(rsqrt64, edge):
    steps = np.arange(-1000, 1001)
    x = np.concatenate([(np.float64(edge).view(np.int64) + steps * s).view(np.float64) for s in (1, 1 << 29, 1 << 40)])
    assert ulps(x, rsqrt64(x)).max() < 2.0


def test_special_values(rsqrt64):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, -5e-324, 5e-324, 2.0**-1022, np.finfo(np.float64).max])
    with np.errstate(all="ignore"):
        want = 1 / np.sqrt(x)
    got = rsqrt64(x)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~np.isfinite(x) | (x == 0)], want[~np.isfinite(x) | (x == 0)], equal_nan=True)
    assert np.all(np.signbit(got[:3]) == np.signbit(want[:3]))
    assert ulps(x[7:], got[7:]).max() < 2.0
