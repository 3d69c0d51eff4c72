"""The quotients written for the kernels against the compiler's division on the GPU (tests/quotient_harness.cu).

co_quot, for a divisor whose magnitude and reciprocal are normal numbers (2^-1022 <= |d| <= 2^1022) or zero, infinite or
NaN: within one unit in the last place of the rounded quotient where that is a normal number (the correction by the
residual leaves a relative error below 2^-53 + 2^-100 before its rounding, so the result is one of the two neighbours
of the exact quotient), and the same infinity, NaN or zero elsewhere: overflowing quotients among them.

over_t: within one unit for operands as the rate kernel has them (activation temperatures over T)."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    from unicorn_b200.build import NVCC_FLAGS, nvcc
    so = tmp_path_factory.mktemp("q") / "quotient_harness.so"
    subprocess.run([nvcc(), *NVCC_FLAGS, "-o", str(so), str(ROOT / "tests" / "quotient_harness.cu")], check=True)
    lib = ctypes.CDLL(str(so))

    def run(num, den):
        num, den = np.ascontiguousarray(num, np.float64), np.ascontiguousarray(den, np.float64)
        out = [np.empty_like(num) for _ in range(3)]
        p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
        assert lib.harness_quotients(len(num), p(num), p(den), *[p(a) for a in out]) == 0
        return out
    return run


def _ulps(a, b):
    """Distance in representable numbers of two arrays of finite numbers of one sign each."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def _random(rng, n, lo, hi):
    return rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))


def test_co_quot_within_a_unit_of_the_division(quotients):
    rng = np.random.default_rng(5)
    n = 1 << 20
    d = np.concatenate([_random(rng, n, -60, 60), _random(rng, n, -1022, 1022)])
    q = np.concatenate([_random(rng, n, -200, 200), _random(rng, n, -900, 1000)])
    with np.errstate(over="ignore", under="ignore"):
        num = q * d
    keep = np.isfinite(num) & (np.abs(num) >= 2.0 ** -960)      # residuals are then normal numbers
    num, d = num[keep], d[keep]
    co, _, div = quotients(num, d)
    assert len(num) > n and np.isfinite(div).all() and (np.sign(co) == np.sign(div)).all()
    u = _ulps(co, div)
    print(f"\nco_quot: {(u > 0).mean():.2e} of {len(u)} quotients differ from the division, by {u.max()} at most")
    assert u.max() <= 1


def test_co_quot_at_the_edges(quotients):
    rng = np.random.default_rng(6)
    inf, nan = np.inf, np.nan
    edge = [(1e300, 3e-10), (-1e300, 3e-10), (1e300, -3e-10), (1.0, 0.0), (-1.0, 0.0), (1.0, -0.0), (0.0, 0.0), (0.0, 3.0),
            (-0.0, 3.0), (inf, 2.0), (-inf, 2.0), (inf, -2.0), (1.0, inf), (1.0, -inf), (inf, inf), (inf, 0.0), (nan, 2.0),
            (2.0, nan), (nan, nan), (0.0, inf), (0.0, nan), (1.7e308, 0.5), (1.7e308, 2.0 ** -1022)]
    num, den = (np.array(x, float) for x in zip(*edge))
    n = 1 << 18                                                  # overflowing by a factor of two and more
    d = _random(rng, n, -1000, -300)
    e = np.frexp(d)[1]
    num2 = rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(1.0, 2.0, n), np.minimum(e + 1025 + rng.integers(0, 40, n), 1023))
    co, _, div = quotients(np.concatenate([num, num2]), np.concatenate([den, d]))
    assert np.isinf(div[len(edge):]).all()
    assert np.array_equal(co, div, equal_nan=True), [(x, y, a, b) for x, y, a, b in zip(num, den, co, div)
                                                   if not (a == b or (a != a and b != b))]


def test_over_t_within_a_unit_of_the_division(quotients):
    rng = np.random.default_rng(7)
    n = 1 << 20
    x = rng.uniform(-1.0e5, 1.0e5, n)
    x[::7] = np.ldexp(rng.uniform(1.0, 2.0, x[::7].size), rng.integers(-20, 30, x[::7].size))
    x[::1001] = 0.0
    T = np.concatenate([rng.uniform(50.0, 6000.0, n // 2), np.exp(rng.uniform(0.0, np.log(1e5), n - n // 2))])
    _, over, div = quotients(x, T)
    u = _ulps(over, div)
    print(f"\nover_t: {(u > 0).mean():.2e} of {n} quotients differ from the division, by {u.max()} at most")
    assert u.max() <= 1
