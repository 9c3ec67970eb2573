"""Bounded waits of the FP64 form's split kernels (Ndim 25..256) run out cleanly on the GPU, as those
of the mixed kernels do: with the test switch's one non-blocking poll a wait gives up while the
tensor cores are still busy, the CTA stops issuing work, frees its tensor memory and returns, its
points are marked, and the same context computes the same bits afterwards.  Points on the FP64 pipe
(Ndim 16 beside the others, or an eta far below the energies) have no such wait."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import _lib, api, synthetic
from wannier_tools_gb300._lib import PREC_FP64, PT_TIMEOUT

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE
NAMES = ("dos_l", "dos_r", "dos_bulk", "iters", "status")


def _short_waits(lib, fn):
    assert lib.wtg_test_option(_lib.TEST_MIXED_SPIN_LIMIT, 1) == _lib.WTG_OK
    try:
        return fn()
    finally:
        assert lib.wtg_test_option(_lib.TEST_MIXED_SPIN_LIMIT, 0) == _lib.WTG_OK


@pytest.mark.parametrize("nw,np_,nk", [(20, 2, 200), (56, 2, 4), (75, 2, 4)])
def test_spectrum_waits_run_out(built_lib, nw, np_, nk):
    m = synthetic.make_model(nw, np_, seed=900 + nw)
    kp = synthetic.random_kpoints(nk, seed=nw)       # 200: some CTAs pull again after they gave up
    om = np.array([-0.2, 0.1]) * EV
    top, bot = list(range(1, nw + 1, 2)), list(range(1, nw + 1, 3))
    with api.Model.from_surface_model(m) as g:
        def run(eta=1e-2):
            return g.surface_spectrum_spin(kp, om, eta * EV, top, bot)
        before, pipe = run(), run(1e-9)
        assert (before["status"] == 0).all()
        timed, pipe_timed = _short_waits(built_lib, lambda: (run(), run(1e-9)))
        assert ((timed["status"] & PT_TIMEOUT) != 0).all(), timed["status"]
        after = run()
    for name in NAMES + ("sx_l", "sz_r"):
        assert np.array_equal(after[name], before[name]), name
        assert np.array_equal(pipe_timed[name], pipe[name]), name


def test_batch_waits_run_out(built_lib):
    shapes = [(8, 2), (20, 2), (30, 2)]
    gs = [api.Model.from_surface_model(synthetic.make_model(nw, np_, seed=950 + i))
          for i, (nw, np_) in enumerate(shapes)]
    try:
        tops = [list(range(1, nw + 1)) for nw, _ in shapes]
        rng = np.random.default_rng(4)
        n = 600                                      # more points than CTAs
        pm = rng.integers(0, 3, n).astype(np.int32)
        k, om, eta = rng.uniform(-0.5, 0.5, (n, 2)), rng.uniform(-1, 1, n) * EV, np.full(n, 1e-2 * EV)

        def run():
            return api.batch_spectrum(gs, tops, tops, pm, k, om, eta, precision=PREC_FP64)
        before = run()
        assert (before["status"] == 0).all()
        timed = _short_waits(built_lib, run)
        assert ((timed["status"][pm > 0] & PT_TIMEOUT) != 0).all()
        ok = timed["status"] == 0                    # Ndim 16 points pulled before their CTA gave up
        after = run()
        for name in NAMES:
            assert np.array_equal(after[name], before[name]), name
            assert np.array_equal(timed[name][ok], before[name][ok]), name
    finally:
        for g in gs:
            g.close()
