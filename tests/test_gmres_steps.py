"""Arnoldi cycles of the mixed GMRES past the 64 steps that its one-block
kernels keep on chip, and short ones, against the FP64 BiCG.

Bound: both stop at |r|^2 < 1e-12 |b|^2, a relative residual of 1e-6; the
condition of the system is below ten in the observables: 1e-5.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


def test_long_and_short_cycles():
    from mstm_b200 import api
    pos, _ = C.rsa_sphere(60, 1.5, 0.2, seed=3)
    args = (pos, np.full(60, 1.5), np.full(60, 3.0 + 0.0j))
    want = api.SphereCluster(*args, mie_epsilon=-7.0).fixedorsoln(eps=1e-12, niter=3000)
    for restart in (0, 20):
        g = api.SphereCluster(*args, mie_epsilon=-7.0, precision="mixed", gmres_restart=restart)
        r = g.fixedorsoln(eps=1e-12, niter=3000)
        assert r["istat"] == 0
        if restart == 0:   # iterations are pairs of steps: some cycle has more than 64
            assert 2 * max(r["iterations"]) > 64 * r["outer"]
        assert np.abs(r["qtot"][:, 0] - want["qtot"][:, 0]).max() <= 1e-5 * np.abs(want["qtot"]).max()
        g.close()
