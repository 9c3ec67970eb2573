"""FP64 unit products and inverses whose operands are graded along the contraction index, which
shared row and column exponents cannot absorb.

Products: every element is within K 2^-50 sum_k |x_ik|_1 |y_kj|_1 of the exact one (|.|_1 =
|re| + |im|).  A split product's bound: both operands rounded to 2^-54 of their row's or column's
leading binary digit, two real products a term, K 2^-51 in these units where the terms reach the
scales; an FP64 product's: (2 K + 1) 2^-53.

Inverses: with X = A D, D powers of two, X^-1 = D^-1 A^-1 exactly, row by row; each row of the
inverse is within 8 N 2^-53 cond_1(A) of LAPACK's A^-1, a pivoted elimination's normwise bound for
both (partial pivoting ignores column scales), whatever D is."""
import numpy as np
import pytest

from wannier_tools_gb300 import api
from wannier_tools_gb300._lib import PREC_FP64

pytestmark = pytest.mark.gpu


def _c(rng, n):
    return rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))


def _check_product(x, y):
    got = api.mat_mul(x, y, PREC_FP64)
    xr, xi, yr, yi = [v.astype(np.longdouble) for v in (x.real, x.imag, y.real, y.imag)]
    cr, ci = xr @ yr - xi @ yi, xr @ yi + xi @ yr
    err = np.hypot((got.real - cr).astype(float), (got.imag - ci).astype(float))
    terms = ((abs(xr) + abs(xi)) @ (abs(yr) + abs(yi))).astype(float)
    assert np.all(err <= len(x) * 2.0 ** -50 * terms), float(np.max(err / np.maximum(terms, 1e-300)))


@pytest.mark.parametrize("n", [24, 25, 40, 65, 130, 264])
def test_products_graded_along_k(built_lib, n):
    rng = np.random.default_rng(n)
    x, y = _c(rng, n), _c(rng, n)
    for r in (2, 4, 8, 30) if n < 264 else (4,):
        d = 10.0 ** rng.uniform(-r, r, n)
        _check_product(x * d[None, :], y / d[:, None])
        _check_product(x * d[:, None], y / d[None, :])        # rows and columns: absorbed
    if n == 264:                                              # (the exact products take seconds)
        return
    for v in (1e6, 1e12, 1e200):
        d = np.ones(n)
        d[n // 3] = v
        _check_product(x * d[None, :], y / d[:, None])
    # graded rows of one operand only, permutations and diagonals (few terms an element)
    g = y * 10.0 ** rng.uniform(-12, 0, (n, 1))
    for s in (np.eye(n), np.eye(n)[rng.permutation(n)], np.diag(10.0 ** rng.uniform(-9, 9, n))):
        _check_product(s.astype(complex), g)
        _check_product(g.T.copy(), s.astype(complex))
    _check_product(x * 1e-300, y)                             # below the smallest shared exponent


@pytest.mark.parametrize("n", [24, 40, 130])
def test_products_with_infinities(built_lib, n):
    """Only the row (column) of an Inf in the left (right) factor is not finite, and not all NaN."""
    rng = np.random.default_rng(n)
    x, y = rng.normal(size=(n, n)) + 0j, rng.normal(size=(n, n)) + 0j
    a = x.copy()
    a[3, 5] = np.inf
    got = api.mat_mul(a, y, PREC_FP64)
    assert np.isfinite(np.delete(got, 3, 0)).all() and np.isinf(got[3].real).all()
    b = y.copy()
    b[5, 7] = np.inf
    got = api.mat_mul(x, b, PREC_FP64)
    assert np.isfinite(np.delete(got, 7, 1)).all() and np.isinf(got[:, 7].real).all()


@pytest.mark.parametrize("n", [24, 25, 40, 112, 113, 161, 264])
@pytest.mark.parametrize("r", [3, 7, 10, 16, 20, 60])
def test_inverses_of_graded_columns(built_lib, n, r):
    rng = np.random.default_rng(100 * n + r)
    a = _c(rng, n) + 2.0 * np.sqrt(n) * np.eye(n)
    d = 2.0 ** rng.integers(-r, r + 1, n)
    one = np.ones(n)
    one[n // 2] = 2.0 ** r
    ai = np.linalg.inv(a)
    bar = 8 * n * 2.0 ** -53 * np.linalg.norm(a, 1) * np.linalg.norm(ai, 1)
    for dd in (d, one):
        for left in (one * 0 + 1, d):                          # rows graded too
            g, st = api.inv(a * dd[None, :] * left[:, None], PREC_FP64)
            assert st == 0
            got = g * dd[:, None] * left[None, :]
            rows = np.linalg.norm(got - ai, axis=1) / np.linalg.norm(ai, axis=1)
            assert rows.max() <= bar, rows.max()
