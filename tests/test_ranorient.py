"""Orientation average of T matrices of the smallest and the largest order, at
the edge of a 32-wide product tile (order 16, 32 rows) and with the item loop
in one and in several chunks, against the oracle.

Bound: FP64 sums of at most 5041 items times 73 values of u over the same
single-precision T on both sides, the vector-coupling rows by the same
recurrence: 1e-12 of the largest value for the sums and 1e-10 with the
recurrence's own growth at order 70.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 5, 16, 17, 22, 35])
def test_orders(T):
    from mstm_b200 import api
    from oracle import oracle as O
    rng = np.random.default_rng(T)
    nb = 2 * T * (T + 2)
    fall = 0.5 ** (np.repeat(np.concatenate([np.full(2 * k + 1, k) for k in range(1, T + 1)]), 2) / max(2.0, T / 3.0))
    tm = np.asfortranarray((rng.normal(size=(nb, nb)) + 1j * rng.normal(size=(nb, nb))) * fall[:, None] * fall)
    pos, _ = C.rsa_sphere(2, 1.0, 0.1, seed=1)
    g = api.SphereCluster(pos, np.ones(2), np.full(2, 1.5 + 0.0j))
    rg, ro = g.ranorientscatmatrix(tm, T), O.ranorientscatmatrix(T, tm)
    for k, s in (("sm", "sm"), ("smcf", "smcf"), ("smat", "smat")):
        a, b = np.asarray(rg[k]), np.asarray(ro[s])
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max(), k
    g.close()
