"""Operator records made pair by pair (few pairs) and, from about 4,700 pairs
on, for groups of four: groups of one order, of mixed orders and a last group
of one or three pairs, through the FP64 interaction product against the CPU
oracle.

Bound: the same sums of at most 33 coupling terms on both sides and the
rounding of the rotations (1e-13 at order 8): 1e-11 of the largest value.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mixed", [(2, False), (3, True), (4, False), (5, True), (7, True), (99, False), (98, True)])
def test_against_oracle(n, mixed):
    from mstm_b200 import api
    from oracle import oracle as O
    pos, _ = C.rsa_sphere(n, 1.2, 0.1, seed=n)
    rad = np.full(n, 1.2) * (np.linspace(0.3, 1.0, n) if mixed else 1.0)
    args = (pos, rad, np.full(n, 1.5 + 0.02j))
    eps = 1e-6 if mixed else (-8.0 if n < 50 else -4.0)
    g, o = api.SphereCluster(*args, mie_epsilon=eps), O.Oracle(*args, mie_eps=eps)
    rng = np.random.default_rng(n)
    x = rng.normal(size=(g.number_eqns, 2)) + 1j * rng.normal(size=(g.number_eqns, 2))
    yo = o.sphereinteraction(x, con_tran=[0, 1])
    assert np.abs(g.sphereinteraction(x, con_tran=[0, 1]) - yo).max() <= 1e-11 * np.abs(yo).max()
    g.close()
