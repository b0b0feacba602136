"""The FP64 kernels' division by a tabulated divisor (div_by, csrc/dfdm_common.cuh): product with the rounded reciprocal
and one fused remainder correction.  Its three operations, restated with the C library's fma, against the divide."""
import ctypes

import numpy as np
import pytest

_libm = ctypes.CDLL("libm.so.6")
_libm.fma.restype = ctypes.c_double
_libm.fma.argtypes = [ctypes.c_double] * 3
fma = _libm.fma


def div_by(x, d):
    r = 1.0 / d
    q = x * r
    return fma(fma(-q, d, x), r, q)


@pytest.mark.parametrize("lo,hi", [(0, 1), (-30, 30), (-300, 300)], ids=["one-binade", "fields", "wide"])
def test_equals_the_divide(lo, hi):
    rng = np.random.default_rng(7)
    n = 100000
    x = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n) * rng.choice([-1.0, 1.0], n)
    d = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n)
    for a, b in zip(x.tolist(), d.tolist()):
        assert div_by(a, b) == a / b


@pytest.mark.parametrize("d", [1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 3.0, 65536.0, 49152.0, 0.1, 1e-3, 1.5])
def test_divisors_at_the_ends_of_a_binade(d):
    rng = np.random.default_rng(8)
    for a in [0.0, d, -d, 1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52] + rng.uniform(-2.0, 2.0, 20000).tolist():
        assert div_by(a, d) == a / d
