"""FP64 engines of models with many R vectors: a point's table of Fourier phases shares the shared
memory of the split products' stages (12 864 vectors); engines with more run on the FP64 pipe.

968 vectors would fit behind the stages' layout too, 1 800 (a 15 x 15 mesh over the eight R3 layers
of Np = 3) only in the shared area, 13 065 only beside the FP64 pipe's smaller layout; Ndim 24 is the
FP64 pipe's own kernel.  Every point is compared with the per-model call (bit for bit where both run
the same kernel) and one with the oracle, to the forms' 1e-9 and 1e-5."""
import numpy as np
import pytest

from oracle import wt_oracle as O
from wannier_tools_gb300 import api
from wannier_tools_gb300._lib import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu

EV = O.EV2HARTREE


def _model(nw, r1, r2, r3, seed):
    """Hermitian H(R) on a (2 r1 + 1) x (2 r2 + 1) x (2 r3 + 1) mesh, decaying over one cell."""
    rng = np.random.default_rng(seed)
    g3, g2, g1 = np.meshgrid(*(np.arange(-r, r + 1) for r in (r3, r2, r1)), indexing="ij")
    irvec = np.stack([g1.ravel(), g2.ravel(), g3.ravel()], 1).astype(np.int32)
    h = rng.standard_normal((len(irvec), nw, nw, 2)).view(np.complex128)[..., 0]
    h *= (0.5 * np.exp(-np.linalg.norm(irvec, axis=1)))[:, None, None]
    return irvec, (h + h[::-1].conj().transpose(0, 2, 1)) * (EV / np.sqrt(2.0))


@pytest.mark.parametrize("nw,np_,mesh,used,prec", [
    (9, 3, (5, 5, 5), 121 * 8, PREC_FP64), (9, 3, (7, 7, 5), 225 * 8, PREC_FP64),
    (13, 2, (33, 32, 1), 67 * 65 * 3, PREC_FP64), (6, 4, (7, 7, 3), 225 * 7, PREC_FP64),
    (9, 3, (5, 5, 5), 121 * 8, PREC_MIXED)])
def test_engine_with_many_r_vectors(built_lib, nw, np_, mesh, used, prec):
    irvec, h = _model(nw, *mesh, seed=nw)
    lo = (irvec[:, 2] > -np_) & (irvec[:, 2] < 2 * np_)
    assert lo.sum() == used
    top, bot = list(range(1, nw + 1)), list(range(2, nw + 1))
    rng = np.random.default_rng(1)
    n = 6
    k, om, eta = rng.uniform(-0.5, 0.5, (n, 2)), rng.uniform(-1, 1, n) * EV, np.full(n, 5e-3 * EV)
    with api.Model(h, irvec, None, np_) as g:
        with api.Engine([g], [top], [bot], precision=prec, max_points=64) as e:
            got = e.run(np.zeros(n, np.int32), k, om, eta)
        assert (got["status"] == 0).all()
        ref = [g.surface_spectrum(k[p:p + 1], om[p:p + 1], eta[p], top, bot, precision=prec) for p in range(n)]
    for name in ("dos_l", "dos_r", "dos_bulk"):
        one = np.array([r[name][0, 0] for r in ref])
        if used <= 12864:
            assert np.array_equal(got[name], one), name
        else:
            assert np.max(np.abs(got[name] - one) / np.abs(one)) <= 1e-9, name
    want = O.surface_spectrum(h, irvec, np.ones(len(irvec), np.int32), nw, np_, k[:1], om[:1], eta[0], top, bot)
    bar = 1e-9 if prec == PREC_FP64 else 1e-5
    for name in ("dos_l", "dos_r", "dos_bulk"):
        assert abs(got[name][0] - want[name][0, 0]) <= bar * abs(want[name][0, 0]), name
