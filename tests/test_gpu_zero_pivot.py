"""Exact zero pivots of the FP32 Gauss-Jordan that starts the split forms' inverses (Ndim 25 and
above), at every place of a panel of pivot steps, and the FP64 Gauss-Jordan that takes over.

A zero column stays exactly zero through the elimination steps before it, so its step has no pivot:
the status says so and the FP64 form returns the identity, as zgesv + inv do.  A Hamiltonian of
2^-140 Hartree is regular in FP64 but zero in FP32: every inverse of its decimation falls back to
the FP64 Gauss-Jordan (in shared or, forced, in global memory: the same bits).  Scaling energies by a
power of two scales every FP64 result exactly, so the spectra are the unscaled oracle's, to the FP64
form's 1e-9."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import _lib, api, synthetic
from wannier_tools_gb300._lib import PREC_FP64, PREC_MIXED, PT_SINGULAR

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE


# 25..112: panels of 8 in shared memory; above: panels of 16 in global memory
@pytest.mark.parametrize("n", [25, 40, 64, 65, 112, 113, 161, 264])
def test_zero_column(built_lib, n):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    for c in sorted({0, 1, 6, 7, 8, 9, 15, 16, 17, 23, n - 2, n - 1}):
        m = a.copy()
        m[:, c] = 0.0
        g, st = api.inv(m, PREC_FP64)
        assert st == PT_SINGULAR, (n, c)
        assert np.array_equal(g, np.eye(n)), (n, c)
        _, st = api.inv(m, PREC_MIXED)
        assert st & PT_SINGULAR, (n, c)
    g, st = api.inv(a, PREC_FP64)                     # the same kernel afterwards
    assert st == 0 and np.linalg.norm(np.eye(n) - a @ g) <= 1e-9


@pytest.mark.parametrize("nw,np_", [(25, 1), (20, 2), (56, 2), (57, 2), (75, 2)])
def test_spectra_of_values_below_fp32(built_lib, nw, np_):
    m = synthetic.make_model(nw, np_, seed=300 + nw)
    kp = synthetic.random_kpoints(2, seed=nw)
    om = np.array([-0.2, 0.1]) * EV
    top, bot = list(range(1, nw + 1, 2)), list(range(2, nw + 1, 3))
    ref = O.surface_spectrum(m.hmnr, m.irvec, m.ndegen, nw, np_, kp, om, 5e-3 * EV, top, bot)
    s = 2.0 ** -140
    got = []
    with api.Model(m.hmnr * s, m.irvec, m.ndegen, np_) as g:
        for forced in (0, 1):
            assert built_lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, forced) == 0
            try:
                got.append(g.surface_spectrum(kp, om * s, 5e-3 * EV * s, top, bot,
                                              tol=O.ACCURACY_REF * s))
            finally:
                built_lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, 0)
    for name in ("dos_l", "dos_r", "dos_bulk", "iters", "status"):
        assert np.array_equal(got[0][name], got[1][name]), name
    assert (got[0]["status"] == 0).all() and np.array_equal(got[0]["iters"], ref["iters"])
    for name in ("dos_l", "dos_r", "dos_bulk"):
        assert np.max(np.abs(got[0][name] * s - ref[name]) / np.abs(ref[name])) <= 1e-9, name
