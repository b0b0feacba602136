"""The FP64 kernels' division by a divisor whose reciprocal is at hand (div_by, csrc/div_by.h), compiled here with g++, against
the divide: quotients of normal numbers, and every operand or quotient that is zero, infinite or not a number."""
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dopamine-fdm_b200", "csrc")

# pairs (x, d) of doubles from standard input to quotients on standard output, the reciprocal formed as the kernels form it
HARNESS = r"""
#include "div_by.h"
#include <cstdio>
int main() {
    double v[2];
    while (std::fread(v, sizeof(double), 2, stdin) == 2) {
        const double q = dfdm::div_by(v[0], v[1], 1.0 / v[1]);
        std::fwrite(&q, sizeof(double), 1, stdout);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def div_by(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("div")
    src = d / "div.cpp"
    src.write_text(HARNESS)
    exe = d / "div"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)

    def run(x, d):
        pairs = np.ascontiguousarray(np.stack(np.broadcast_arrays(np.float64(x), np.float64(d)), axis=-1))
        return np.frombuffer(subprocess.run([str(exe)], input=pairs.tobytes(), capture_output=True, check=True).stdout)
    return run


def divide(x, d):
    with np.errstate(all="ignore"):
        return np.float64(x) / np.float64(d)


@pytest.mark.parametrize("lo,hi", [(0, 1), (-30, 30), (-300, 300)], ids=["one-binade", "fields", "wide"])
def test_equals_the_divide(div_by, lo, hi):
    rng = np.random.default_rng(7)
    n = 100000
    x = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n) * rng.choice([-1.0, 1.0], n)
    d = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n)
    assert np.array_equal(div_by(x, d), divide(x, d))


@pytest.mark.parametrize("d", [1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 3.0, 65536.0, 49152.0, 0.1, 1e-3, 1.5, 0.41, 0.75 * 2e-3])
def test_divisors_at_the_ends_of_a_binade(div_by, d):
    rng = np.random.default_rng(8)
    x = np.array([0.0, d, -d, 1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52] + rng.uniform(-2.0, 2.0, 20000).tolist())
    assert np.array_equal(div_by(x, d), divide(x, d))


def test_zeros_infinities_and_nans(div_by):
    """A field that overflows, a quotient that does, and the divisors 0 (a viscosity of zero is accepted) and infinity; the
    sign of a zero for positive divisors (the negative ones are wave numbers, whose quotients go into a transform)."""
    big = np.finfo(np.float64).max
    x = [0.0, -0.0, 1.0, -3.0, big, -big, np.inf, -np.inf, np.nan]
    d = [0.0, 1e-3, 0.41, 3.0, -7.0, 65536.0, np.inf, -np.inf, np.nan]
    x, d = np.array(list(itertools.product(x, d))).T
    got, want = div_by(x, d), divide(x, d)
    assert np.array_equal(got, want, equal_nan=True)
    signed = ~np.isnan(want) & ~((want == 0.0) & (d < 0.0))
    assert np.array_equal(np.signbit(got[signed]), np.signbit(want[signed]))
