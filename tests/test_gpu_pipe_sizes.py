"""The CTA-wide kernel on the FP64 pipe at the sizes it runs (Ndim 9..24): its shared-memory and its
forced global-memory inverse agree bit for bit at sizes of several panels of 8 pivot steps and odd
remainders, and its CTA widths (256 threads for few instances, 64 or 128 for many) agree to the
norm's order (1e-12) with the oracle's 1e-9 held."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import _lib, api, synthetic

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE
NAMES = ("dos_l", "dos_r", "dos_bulk")


@pytest.mark.parametrize("nw,np_", [(9, 1), (5, 2), (15, 1), (8, 2), (17, 1), (7, 3), (23, 1), (12, 2)])
@pytest.mark.parametrize("arc", [False, True])
def test_inverses_bitwise(built_lib, nw, np_, arc):
    m = synthetic.make_model(nw, np_, seed=40 + nw)
    kp, om = synthetic.random_kpoints(5, seed=nw), np.array([-0.3, 0.0, 0.2]) * EV
    top, bot = [1, 2, 3], [1, nw]
    got = []
    with api.Model.from_surface_model(m) as g:
        for forced in (0, 1):
            assert built_lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, forced) == 0
            try:
                got.append(g.surface_spectrum_spin(kp, om, 1e-3 * EV, top, bot, arc=arc))
            finally:
                built_lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, 0)
    for name in NAMES + ("iters", "status", "sx_l", "sy_l", "sz_l", "sx_r", "sy_r", "sz_r"):
        assert np.array_equal(got[0][name], got[1][name]), name


@pytest.mark.parametrize("nw,np_", [(9, 1), (12, 1), (8, 2), (20, 1), (7, 3), (12, 2)])
def test_widths_agree(built_lib, nw, np_):
    m = synthetic.make_model(nw, np_, seed=70 + nw)
    n = 1300                                         # 8 instances an SM and more: the narrow CTAs
    kp, om = synthetic.random_kpoints(n, seed=nw), np.array([0.1]) * EV
    top, bot = list(range(1, nw + 1)), [1, nw]
    with api.Model.from_surface_model(m) as g:
        many = g.surface_spectrum(kp, om, 5e-3 * EV, top, bot)
        few = g.surface_spectrum(kp[:40], om, 5e-3 * EV, top, bot)
    ref = O.surface_spectrum(m.hmnr, m.irvec, m.ndegen, nw, np_, kp[:8], om, 5e-3 * EV, top, bot)
    assert (many["status"] == 0).all() and np.abs(many["iters"][:40] - few["iters"]).max() <= 1
    for name in NAMES:
        assert np.all(np.abs(many[name][:40] - few[name]) <= 1e-12 * np.abs(few[name])), name
        assert np.max(np.abs(many[name][:8] - ref[name]) / np.abs(ref[name])) <= 1e-9, name
