"""FP64 unit products, inverses and spectra whose operands are graded along the contraction index, which
shared row and column exponents cannot absorb.

Products: every element is within K 2^-50 sum_k |x_ik|_1 |y_kj|_1 of the exact one (|.|_1 =
|re| + |im|).  A split product's bound: both operands rounded to 2^-54 of their row's or column's
leading binary digit, two real products a term, K 2^-51 in these units where the terms reach the
scales; an FP64 product's: (2 K + 1) 2^-53.

Inverses: with X = A D, D powers of two, X^-1 = D^-1 A^-1 exactly, row by row; each row of the
inverse is within 8 N 2^-53 cond_1(A) of LAPACK's A^-1, a pivoted elimination's normwise bound for
both (partial pivoting ignores column scales), whatever D is.

Spectra: the FP64 form's 1e-9 against the oracle, for orbitals of very different scales (one orbital
far away with a strong hopping, or a ramp of scales) on both sides of the rule's line, and off the
bands of a real Hamiltonian at an eta far below it, where FP64 arithmetic keeps every digit of the
imaginary parts."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import _lib, api, synthetic
from wannier_tools_gb300._lib import PREC_FP64

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE
NAMES = ("dos_l", "dos_r", "dos_bulk")


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


def _scaled(m, d, onsite=None):
    """The model with orbital i scaled by d[i] (H_ij d_i d_j) and orbital 0 at `onsite` eV."""
    h = m.hmnr * d[None, :, None] * d[None, None, :]
    if onsite is not None:
        h[np.flatnonzero((m.irvec == 0).all(1))[0], 0, 0] = onsite * EV
    return h


def _check(h, m, kp, om, eta, lib):
    """Per-model (both variants of the fallback inverse) and engine spectra against the oracle."""
    top, bot = list(range(1, m.nw + 1)), list(range(2, m.nw + 1, 2))
    ref = O.surface_spectrum(h, m.irvec, m.ndegen, m.nw, m.np_, kp, om, eta, top, bot)
    with api.Model(h, m.irvec, m.ndegen, m.np_) as g:
        got = []
        for forced in (0, 1):
            assert lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, forced) == 0
            try:
                got.append(g.surface_spectrum(kp, om, eta, top, bot))
            finally:
                lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, 0)
        n = len(kp) * len(om)
        with api.Engine([g], [top], [bot], max_points=64) as e:
            b = e.run(np.zeros(n, np.int32), np.repeat(kp, len(om), 0), np.tile(om, len(kp)), np.full(n, eta))
    for name in NAMES + ("iters", "status"):
        assert np.array_equal(got[0][name], got[1][name]), name
        if m.nw * m.np_ >= 25:                                 # the same kernel code
            assert np.array_equal(got[0][name].ravel(), b[name]), name
    assert (got[0]["status"] == 0).all()
    for name in NAMES:
        for r in (got[0][name], b[name].reshape(ref[name].shape)):
            err = np.max(np.abs(r - ref[name]) / np.abs(ref[name]))
            assert err <= 1e-9, (name, err)


@pytest.mark.parametrize("nw,np_", [(12, 2), (25, 1), (20, 2), (56, 2), (57, 2), (128, 2)])
@pytest.mark.parametrize("onsite,hop", [(30, 5), (1e3, 30), (3e3, 50), (1e8, 1e4), (1e12, 1e6), (1e12, 1)])
def test_spectra_with_a_far_orbital(built_lib, nw, np_, onsite, hop):
    if nw == 128 and onsite != 1e12:                           # (the oracle takes seconds)
        return
    m = synthetic.make_model(nw, np_, seed=nw)
    d = np.ones(nw)
    d[0] = hop
    _check(_scaled(m, d, onsite), m, synthetic.random_kpoints(2 if nw < 100 else 1, seed=nw),
           np.array([-0.2, 0.1]) * EV, 1e-2 * EV, built_lib)


@pytest.mark.parametrize("nw,np_", [(12, 2), (20, 2), (14, 3), (56, 2)])
@pytest.mark.parametrize("decades", [0.5, 1.0, 2, 4, 8])
def test_spectra_with_a_ramp_of_scales(built_lib, nw, np_, decades):
    m = synthetic.make_model(nw, np_, seed=nw + 1)
    for d in (10.0 ** np.linspace(0, decades, nw), 10.0 ** -np.linspace(0, decades, nw)):
        _check(_scaled(m, d), m, synthetic.random_kpoints(2, seed=nw), np.array([0.1]) * EV, 1e-2 * EV, built_lib)


@pytest.mark.parametrize("nw,np_", [(12, 2), (25, 1), (20, 2), (56, 2), (57, 2)])
@pytest.mark.parametrize("eta_ev", [1e-2, 1e-5, 1e-8, 1e-12])
def test_spectra_off_the_bands_at_small_eta(built_lib, nw, np_, eta_ev):
    m = synthetic.make_model(nw, np_, seed=nw + 2)
    m.hmnr = m.hmnr.real.astype(complex)                       # H(-R) = H(R)^T: real at k = 0
    _check(m.hmnr, m, np.zeros((1, 2)), np.array([-25.0, 25.0]) * EV, eta_ev * EV, built_lib)


def test_surfgreen_1985_of_graded_layers(built_lib):
    n = 40
    m = synthetic.make_model(20, 2, seed=9)
    d = np.tile(10.0 ** np.linspace(0, 6, 20), 2)
    h00, h01 = O.ham_qlayer2qlayer([0.21, -0.4], m.hmnr, m.irvec, m.ndegen, 20, 2)
    h00, h01 = h00 * d[:, None] * d[None], h01 * d[:, None] * d[None]
    ref = O.surfgreen_1985(0.03 * EV, h00, h01, 1e-2 * EV)
    got = api.surfgreen_1985(0.03 * EV, h00, h01, 1e-2 * EV)
    for a, b in zip(got[:3], ref[:3]):
        s = np.sqrt(np.abs(np.diag(b)))
        assert np.max(np.abs(a - b) / (s[:, None] * s[None])) <= 1e-9
    assert abs(got[3] - ref[3]) <= 1 and got[4] == 0
