"""The FP64 form's split kernels (products on the tensor cores, Ndim 25..256; unit
products and inverses up to 320): products and
inverses at the edges of their tiles, passes and K parts.

Tolerances.  A product's operands are rounded to 2^-55 of their row or column maximum (3-5 times
the rms of normal data): 2 sqrt(1/3) 2^-55 x 5 = 1.6e-16 of the result, plus the result's own
rounding (at most 1.1e-16): 5e-16 normwise bounds both with a factor of two to spare.  An inverse's
right residual |I - M G|_F of a backward-stable FP64 inverse is at most about N eps cond(M):
checked at 4 N eps cond, on both sides of the condition (about 1e7) where the refinement hands over
to the FP64 Gauss-Jordan."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import api, synthetic
from wannier_tools_gb300._lib import PREC_FP64, PT_NONFINITE, PT_NOT_CONVERGED

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE


def _product(a, b):
    ar, ai, br, bi = [x.astype(np.longdouble) for x in (a.real, a.imag, b.real, b.imag)]
    return ar @ br - ai @ bi, ar @ bi + ai @ br


# 24: the FP64 pipe; 25: the first split size; 64 / 65: one and two row tiles of a stacked pair;
# 128 / 129: row blocks; 160 / 161: one and two K parts; 320: the largest
@pytest.mark.parametrize("n", [24, 25, 40, 64, 65, 96, 97, 112, 128, 129, 160, 161, 255, 320])
def test_products(built_lib, n):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    b = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    # every entry equal: all digit products of one sign, the largest partial sums
    v = 1 - 2.0 ** -9 - 2.0 ** -17 - 2.0 ** -25
    rows = 10.0 ** rng.uniform(-8, 8, n)
    for x, y in ((a, b), (np.full((n, n), v + 1j * v), np.full((n, n), v - 1j * v)),
                 (a * rows[:, None], b / rows[None, :]), (np.zeros((n, n)), b)):
        got = api.mat_mul(x, y, PREC_FP64)
        cr, ci = _product(x.astype(complex), y.astype(complex))
        err = np.hypot((got.real - cr).astype(float), (got.imag - ci).astype(float))
        scale = np.sqrt(float((cr ** 2 + ci ** 2).sum()))
        bar = 5e-16 if n > 24 else 4e-16 * np.sqrt(n)      # FP64 sums round K times
        assert np.linalg.norm(err) <= bar * max(scale, 1e-300)


@pytest.mark.parametrize("n", [25, 64, 112, 113, 161, 264])
@pytest.mark.parametrize("cond", [1e1, 1e4, 1e6, 1e8, 1e11])
def test_inverses(built_lib, n, cond):
    rng = np.random.default_rng(n)
    q = [np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))[0] for _ in range(2)]
    m = (q[0] * np.logspace(0, -np.log10(cond), n)) @ q[1]
    g, st = api.inv(m, PREC_FP64)
    assert st == 0
    assert np.linalg.norm(np.eye(n) - m @ g) <= 4 * n * 1.1e-16 * cond


def test_nonfinite_hamiltonian_is_flagged(built_lib):
    """An Inf in H(R): no point converges and the sums are not finite, in the split kernel (Ndim
    40) as on the FP64 pipe (Ndim 16)."""
    for nw in (8, 20):
        m = synthetic.make_model(nw, 2, seed=5)
        h = m.hmnr.copy()
        h[len(h) // 2, 1, 1] = np.inf
        with api.Model(h, m.irvec, m.ndegen, 2) as g:
            r = g.surface_spectrum([[0.1, 0.2]], [0.0], 1e-2 * EV, [1, 2], [1, 2], itermax=5)
        assert (r["status"] & PT_NONFINITE).all() and (r["status"] & PT_NOT_CONVERGED).all()
        assert (r["iters"] == 5).all()


# columns of NaN alone: no row is a pivot candidate, at instance numbers above Ndim too
@pytest.mark.parametrize("nw,np_,nk", [(2, 2, 300), (8, 2, 300), (20, 2, 200), (56, 2, 160), (88, 3, 3)])
def test_nonfinite_instances(built_lib, nw, np_, nk):
    m = synthetic.make_model(nw, np_, seed=6)
    h = np.full_like(m.hmnr, np.nan)
    with api.Model(h, m.irvec, m.ndegen, np_) as g:
        r = g.surface_spectrum(np.zeros((nk, 2)), [0.0], 1e-2 * EV, [1], [1], itermax=2)
    assert (r["status"] & PT_NONFINITE).all() and (r["status"] & PT_NOT_CONVERGED).all()


@pytest.mark.parametrize("nw,np_", [(12, 2), (5, 5), (32, 2), (65, 1), (43, 3), (54, 3), (97, 2)])
def test_spectra_vs_oracle(built_lib, nw, np_):
    m = synthetic.make_model(nw, np_, seed=nw)
    kp = synthetic.random_kpoints(2, seed=nw)
    om = np.array([-0.1, 0.3]) * EV
    top, bot = list(range(1, nw + 1, 2)), list(range(2, nw + 1, 3))
    ref = O.surface_spectrum(m.hmnr, m.irvec, m.ndegen, nw, np_, kp, om, 5e-3 * EV, top, bot,
                             with_spin=True)
    with api.Model.from_surface_model(m) as g:
        got = g.surface_spectrum_spin(kp, om, 5e-3 * EV, top, bot)
    assert np.array_equal(got["iters"], ref["iters"]) and (got["status"] == 0).all()
    for name in ("dos_l", "dos_r", "dos_bulk"):
        assert np.max(np.abs(got[name] - ref[name]) / np.abs(ref[name])) <= 1e-9, name
    scale = np.abs(ref["dos_l"]).max()
    for name in ("sx_l", "sy_l", "sz_l", "sx_r", "sy_r", "sz_r"):
        assert np.max(np.abs(got[name] - ref[name])) <= 1e-9 * scale, name
