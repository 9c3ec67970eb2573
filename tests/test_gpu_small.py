"""The FP64 form's small kernel (Ndim <= 8: an instance per group of lanes of a warp).

Its operations and their order are those of the CTA-wide kernel, so it must reproduce that kernel
(the forced global-memory inverse still runs it) bit for bit at every size, with odd instance
counts (a warp's second group idle), and agree with the oracle to the FP64 form's 1e-9."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import _lib, api, synthetic

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE
NAMES = ("dos_l", "dos_r", "dos_bulk", "iters", "status")
SPIN = ("sx_l", "sy_l", "sz_l", "sx_r", "sy_r", "sz_r")


def _forced(lib, fn):
    assert lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, 1) == 0
    try:
        return fn()
    finally:
        lib.wtg_test_option(_lib.TEST_FP64_GLOBAL_INVERSE, 0)


@pytest.mark.parametrize("nw,np_", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 1), (6, 1), (7, 1), (8, 1),
                                    (1, 2), (2, 2), (3, 2), (4, 2), (1, 3), (2, 3), (2, 4), (9, 1)])
@pytest.mark.parametrize("spin", [None, False, True])
def test_small_kernel_bitwise_and_oracle(built_lib, nw, np_, spin):
    m = synthetic.make_model(nw, np_, seed=60 + 10 * nw + np_)
    kp = synthetic.random_kpoints(3, seed=nw)
    om = np.array([-0.4, 0.1, 0.5]) * EV
    top = [1 + q % nw for q in range(3 if nw < 8 else 40)]       # lists may repeat orbitals
    bot = [nw, 1]
    with api.Model.from_surface_model(m) as g:
        def run():
            if spin is None:
                return g.surface_spectrum(kp, om, 5e-3 * EV, top, bot, divide_by_pi=True)
            return g.surface_spectrum_spin(kp, om, 5e-3 * EV, top, bot, arc=spin)
        a = run()
        b = _forced(built_lib, run)
        with api.Engine([g], [top], [bot], max_points=64) as e:
            c = e.run(np.zeros(9, np.int32), np.repeat(kp, 3, 0), np.tile(om, 3),
                      np.full(9, 5e-3 * EV), divide_by_pi=spin is None or spin)
    for name in NAMES + (SPIN if spin is not None else ()):
        assert np.array_equal(a[name], b[name]), name
    if spin is not False:      # surfstat's spin sums take GRR from the full inverse, the engine a block
        for name in NAMES:
            assert np.array_equal(a[name].ravel(), c[name]), name
    ref = O.surface_spectrum(m.hmnr, m.irvec, m.ndegen, nw, np_, kp, om, 5e-3 * EV, top, bot,
                             scale=1.0 / O.PI_REF if spin is None or spin else 1.0)
    for name in NAMES[:3]:
        assert np.max(np.abs(a[name] - ref[name]) / np.abs(ref[name])) <= 1e-9, name


def test_small_kernel_edges(built_lib):
    """One instance, itermax 0 and 2, an exactly singular pivot and a NaN in the model."""
    m = synthetic.make_model(2, 2, seed=5)
    with api.Model.from_surface_model(m) as g:
        for itmax in (0, 2):
            a = g.surface_spectrum([[0.1, 0.3]], [0.0], 1e-2 * EV, [1], [2], itermax=itmax)
            b = _forced(built_lib, lambda: g.surface_spectrum([[0.1, 0.3]], [0.0], 1e-2 * EV, [1], [2],
                                                              itermax=itmax))
            for name in NAMES:
                assert np.array_equal(a[name], b[name]), (itmax, name)
    h = np.zeros((1, 2, 2), complex)
    irv = np.zeros((1, 3), np.int32)
    with api.Model(h, irv, None, 2) as g:              # w - H = 0 at omega = eta = 0
        a = g.surface_spectrum([[0.0, 0.0]], [0.0], 0.0, [1], [2])
        b = _forced(built_lib, lambda: g.surface_spectrum([[0.0, 0.0]], [0.0], 0.0, [1], [2]))
    assert (a["status"] & _lib.PT_SINGULAR).all()
    for name in NAMES:
        assert np.array_equal(a[name], b[name]), name
    h = m.hmnr.copy()
    h[len(h) // 2, 0, 1] = np.nan
    with api.Model(h, m.irvec, m.ndegen, 2) as g:
        a = g.surface_spectrum([[0.1, 0.3]] * 3, [0.0], 1e-2 * EV, [1], [2], itermax=4)
    assert (a["status"] == (_lib.PT_NONFINITE | _lib.PT_NOT_CONVERGED)).all() and (a["iters"] == 4).all()
