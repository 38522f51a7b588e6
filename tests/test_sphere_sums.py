"""Incident-field coefficients, pair Hankel functions and efficiencies at the
edges of their kernels, against the CPU oracle's FP64 solve: arguments below
the real-Bessel range, pair distances below, at and above the order, the
smallest and the largest sphere order, oblique and backward incidence.

Bound: both sides iterate to the same criterion by the same recurrence, so the
solutions differ by the rounding of their operators and sums (1e-13 of the
largest value, times the condition of these dilute clusters, below 100): 1e-10.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,x,L,sinc,direction", [(3, 0.01, 1, 0.0, 1), (4, 0.02, 3, 0.6, 2), (5, 0.3, 3, 0.0, 2), (6, 1.0, 7, 0.35, 1),
                                                  (3, 4.0, 16, 0.8, 2), (2, 9.0, 12, 0.2, 1)])
def test_against_oracle(n, x, L, sinc, direction):
    from mstm_b200 import api
    from oracle import oracle as O
    pos, _ = C.rsa_sphere(n, x, 0.1, seed=L)
    args = (pos, np.full(n, x), np.full(n, 1.5 + 0.02j))
    kw = dict(eps=1e-24, niter=200, alpha=0.7, sinc=sinc, direction=direction)
    g = api.SphereCluster(*args, mie_epsilon=-float(L))
    r, ro = g.fixedorsoln(**kw), O.Oracle(*args, mie_eps=-float(L)).fixedorsoln(**kw)
    for k in ("amnp", "qeff", "qtot"):
        a, b = np.asarray(r[k]), np.asarray(ro[k])
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max(), k
    g.close()
