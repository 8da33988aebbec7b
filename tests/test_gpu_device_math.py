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
