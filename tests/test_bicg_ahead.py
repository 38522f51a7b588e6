"""The FP64 BiCG with its next pass queued ahead of the stopping test: capped
after a few iterations and run to the end, against the oracle's iteration
(solution, count, error), and the passes it reports.

Bound: the same iteration in FP64; rounding grows by the condition of this
dilute cluster, below 100, over a few iterations: 1e-11 of the largest value.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,niter", [(5, 4, 1), (5, 4, 2), (9, 7, 3), (9, 7, 500), (3, 12, 500)])
def test_capped_and_converged(n, L, niter):
    from mstm_b200 import api
    from oracle import oracle as O
    x = 0.35 * L
    pos, _ = C.rsa_sphere(n, x, 0.1, seed=L)
    args = (pos, np.full(n, x), np.full(n, 1.5 + 0.02j))
    g = api.SphereCluster(*args, mie_epsilon=-float(L))
    r = g.fixedorsoln(eps=1e-14, niter=niter)
    o = O.Oracle(*args, mie_eps=-float(L)).fixedorsoln(eps=1e-14, niter=niter)
    assert r["maxiter"] == o["maxiter"] and list(r["iterations"]) == list(o["iterations"])
    assert np.abs(r["amnp"] - o["amnp"]).max() <= 1e-11 * np.abs(o["amnp"]).max()
    assert r["maxerr"] == pytest.approx(o["maxerr"], rel=1e-3)
    # one pass for each initial residual and one an iteration
    assert r["passes64"] == 2 + sum(min(k, niter) for k in r["iterations"])
    g.close()
