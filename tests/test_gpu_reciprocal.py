"""Reciprocals of the pivots in the dense LDL^T: against 1 / d over signs, exponents and mantissas, and a block
whose pivots grow out of the fast reciprocal's range during the elimination."""
import ctypes as C
import math
from fractions import Fraction

import numpy as np
import pytest
import scipy.sparse as sp

from inla_b200 import GpuSolver, _lib

pytestmark = pytest.mark.gpu


def reciprocal(x):
    y = np.empty_like(x)
    _lib.check(_lib.lib().inla_reciprocal_selftest(C.c_int64(len(x)), _lib.dptr(x), _lib.dptr(y)))
    return y


def test_within_one_unit_of_the_rounded_reciprocal():
    rng = np.random.default_rng(0)
    edges = np.concatenate([1.0 + 2.0 ** -np.arange(1, 53), [1.0, np.nextafter(2.0, 1.0)]])
    m = np.concatenate([rng.uniform(1.0, 2.0, 400_000), np.tile(edges, 200)])
    e = rng.integers(-1000, 1000, len(m))
    x = np.ldexp(m, e) * rng.choice([-1.0, 1.0], len(m))
    got, want = reciprocal(x), 1.0 / x
    # the approximation is within 2^-18, the step's error below half a unit, its rounding and that of 1 / x half
    # a unit each: fewer than two units apart, hence at most one
    assert np.array_equal(np.sign(got), np.sign(want))
    assert np.max(np.abs(got.view(np.int64) - want.view(np.int64))) <= 1


def test_error_of_the_reciprocal():
    x = np.random.default_rng(1).uniform(1.0, 2.0, 20_000)
    got = reciprocal(x)
    ulp = np.spacing(1.0 / x)
    worst = max(abs(Fraction(float(y)) - 1 / Fraction(float(d))) / Fraction(float(u)) for d, y, u in zip(x, got, ulp))
    assert worst <= 1


def test_special_values_divide():
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 2.0 ** 1023, -1.5 * 2.0 ** 1023, 2.0 ** -1001, 2.0 ** 1000])
    with np.errstate(divide="ignore", over="ignore"):
        want = 1.0 / x
    assert np.array_equal(reciprocal(x).view(np.int64)[~np.isnan(x)], want.view(np.int64)[~np.isnan(x)])
    assert np.isnan(reciprocal(x)[np.isnan(x)]).all()


@pytest.mark.parametrize("n", [40, 80, 130])
@pytest.mark.parametrize("at", [0, 5, 6])
def test_pivots_that_grow_out_of_range(n, at):
    """Diagonal entries of ordinary size; pivot at + 1 is beyond 2^1022, so its reciprocal is subnormal, and the
    entry below it is large enough for the product with that reciprocal to decide the next pivot."""
    rng = np.random.default_rng(n + at)
    a = np.tril(rng.uniform(-1.0, 1.0, (n, n)), -1) * 2.0 ** -600
    a += a.T
    np.fill_diagonal(a, rng.uniform(3.0, 5.0, n))
    a[at, at], a[at + 1, at + 1] = 2.0 ** -40, 1.0
    a[at, at + 1] = a[at + 1, at] = 1.25 * 2.0 ** 491
    a[at + 1, at + 2] = a[at + 2, at + 1] = 2.0 ** 1000
    # the couplings of 2^-600 change no other pivot by more than 2^-60 of itself
    d1 = Fraction(a[at + 1, at + 1]) - Fraction(a[at, at + 1]) ** 2 / Fraction(a[at, at])
    d2 = Fraction(a[at + 2, at + 2]) - Fraction(a[at + 1, at + 2]) ** 2 / d1
    assert abs(d1) > 2 ** 1022 and abs(d2) > 2 ** 900
    pivots = [d1, d2] + [Fraction(a[i, i]) for i in range(n) if i not in (at + 1, at + 2)]
    want = sum(math.log2(abs(d.numerator)) - math.log2(d.denominator) for d in pivots) * math.log(2.0)
    sv = GpuSolver(_lib.ORDER_NATURAL)
    sv.factorize(sp.csc_matrix(a))
    # a sum of n logarithms of up to 710, each rounded
    assert abs(sv.log_abs_det() - want) <= 4.0 * n * 710.0 * np.finfo(float).eps
