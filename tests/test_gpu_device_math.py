"""Device functions that no entry point returns by themselves (tests/cpp/device_math_check.cu), against exact values."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from pdds_gb300 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("math") / "device_math_check.so")
    src = [os.path.join(HERE, "cpp", "device_math_check.cu")]
    subprocess.run([build.nvcc()] + build.ARCH + build.CU_FLAGS + ["-shared", "-o", so] + src, check=True)
    return C.CDLL(so)


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("length", [1, 2, 21, 64, 200])
def test_pair_sums_are_not_less_exact_than_fp64(lib, length):
    """The contraction's sums over a side's bins: what FP64 additions would give, or closer to the exact sum."""
    rng = np.random.default_rng(length)
    n = 512
    x = (rng.standard_normal((n, length)) * 2.0 ** rng.integers(-30, 10, (n, length))).astype(np.float32)
    x[::3] = -np.abs(x[::3])
    x[1::7, length // 2:] *= np.float32(1e-6)
    x[4:8] = np.array([0.0, np.inf, -np.inf, np.nan], np.float32)[:, None]
    out = np.zeros(n)
    assert lib.check_pair_sum(ptr(x), n, length, ptr(out)) == 0
    assert out[4] == 0.0 and out[5] == np.inf and out[6] == -np.inf and np.isnan(out[7])
    for i in [i for i in range(n) if not 4 <= i < 8]:
        exact = math.fsum(x[i].astype(np.float64))
        largest = np.max(np.abs(np.cumsum(x[i].astype(np.float64))))
        # the last addition's rounding, and length^2 2^-72 of the largest partial sum in the third float
        assert abs(out[i] - exact) <= 2.0 ** -53 * abs(exact) + 2.0 ** -56 * largest


LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288419716939937510582")


def arguments(fn):
    rng = np.random.default_rng(fn + 1)
    edge = np.array([0.0, -0.0, 1e-300, -1e-300, 5e-324, 1e-60, -1e-40, 1e-20])
    if fn == 2:
        x = [rng.uniform(-745.0, 709.7, 40_000), rng.uniform(-2, 2, 40_000), rng.uniform(-708.5, -707.5, 20_000),
             rng.uniform(707.5, 708.5, 4000), rng.integers(-4096 * 12, 4096 * 12, 20_000) * (math.log(2.0) / 4096)]
    else:
        unit = 0.5 if fn == 0 else math.pi / 2  # a right angle
        near = rng.integers(-9, 10, 20_000) * unit  # of a zero of either
        node = rng.integers(-4 * 65536, 4 * 65536, 40_000) * (unit / 65536)
        far = 4096.0 if fn == 0 else 16.0  # from here on the math library's
        x = [rng.uniform(-2.5, 2.5, 60_000), near * (1 + rng.integers(-8, 9, 20_000) * 2.0 ** -52),
             near + rng.choice([-1, 1], 20_000) * 2.0 ** rng.uniform(-60, -10, 20_000), node,
             np.nextafter(node, 9), node + unit / 131072, rng.uniform(-1.01 * far, 1.01 * far, 20_000),
             np.nextafter(far, [0.0, 1e9]), -np.nextafter(far, [0.0, 1e9])]
    return np.concatenate([edge] + x)


def exact(fn, x):
    if fn == 2:
        return [np.exp(x.astype(LD))]
    if fn == 1:
        return [np.sin(x.astype(LD)), np.cos(x.astype(LD))]
    k = np.rint(2 * x)
    r = (x.astype(LD) - k.astype(LD) / 2) * PI
    s, c, q = np.sin(r), np.cos(r), k.astype(np.int64) % 4
    return [np.choose(q, [s, c, -s, -c]), np.choose(q, [c, -s, -c, s])]


# the documented largest errors of the CUDA functions that these stand in for, in units of the last place
@pytest.mark.parametrize("fn,ulps", [(0, 2), (1, 2), (2, 1)])
def test_table_functions(lib, fn, ulps):
    x = arguments(fn)
    got = {}
    for tab in (0, 1):
        out = np.zeros((len(x), 2))
        assert lib.check_math(ptr(x), len(x), fn, tab, ptr(out)) == 0
        got[tab] = out
    for j, ref in enumerate(exact(fn, x)):
        unit = np.spacing(np.maximum(np.abs(ref), LD(2.0) ** -1022).astype(np.float64))
        err = {tab: (np.abs(got[tab][:, j].astype(LD) - ref) / unit).astype(np.float64) for tab in got}
        assert err[1].max() <= min(ulps, err[0].max())
        assert np.sqrt(np.mean(err[1] ** 2)) <= np.sqrt(np.mean(err[0] ** 2)) * 1.001 + 1e-3


def test_table_functions_without_a_number(lib):
    x = np.array([np.inf, -np.inf, np.nan])
    for fn in (0, 1, 2):
        out = np.zeros((3, 2))
        assert lib.check_math(ptr(x), 3, fn, 1, ptr(out)) == 0
        want = [np.inf, 0.0, np.nan] if fn == 2 else [np.nan] * 3
        assert np.array_equal(out[:, 0], want, equal_nan=True)
