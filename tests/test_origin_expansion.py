"""Translation orders, origin expansion and averaged scattering matrix against
the oracle for given sphere expansions: distances below the real-Bessel range,
a sphere at the origin, mixed and the largest sphere orders, orders past one
and several chunks of azimuthal orders (32 each way).

Bound: FP64 sums of the same terms on both sides (a few thousand a value),
coupling rows by the same recurrence, axial blocks by sums where the oracle
recurs: 1e-10 of the largest value.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,x,orders,spread", [(3, 0.005, (1, 2), 1.0), (1, 1.0, (5,), 1.0), (5, 1.0, (3, 6, 7), 1.0), (4, 5.0, (14, 16), 1.0),
                                               (7, 1.0, (4, 7), 6.0), (5, 2.0, (9,), 7.0)])
def test_against_oracle(n, x, orders, spread):
    from mstm_b200 import api
    from oracle import oracle as O
    rng = np.random.default_rng(n)
    pos = np.zeros((1, 3)) if n == 1 else C.rsa_sphere(n, x, 0.1, seed=n)[0] * spread
    want = np.array([orders[i % len(orders)] for i in range(n)], float)
    # radii whose convergence order is their own: fixed orders need one order for all
    eps = -want[0] if len(orders) == 1 else 1e-6
    rad = np.full(n, x) if len(orders) == 1 else x * (0.3 + 0.7 * want / want.max())
    args = (pos, rad, np.full(n, 1.5 + 0.02j))
    g, o = api.SphereCluster(*args, mie_epsilon=eps), O.Oracle(*args, mie_eps=eps)
    fall = np.concatenate([np.tile([2.0 ** -(row if row > col else col) for col in range(1, L + 1) for row in range(L + 2)], 2)
                           for L in g.sphere_order])
    a = np.asfortranarray((rng.normal(size=(len(fall), 2)) + 1j * rng.normal(size=(len(fall), 2))) * fall[:, None])
    sg, so = g.scattering(a), o.scattering(a)
    assert sg["t_matrix_order"] == so["t_matrix_order"]
    assert np.abs(sg["amnp0"] - so["amnp0"]).max() <= 1e-10 * np.abs(so["amnp0"]).max()
    assert np.abs(sg["smat"] - so["smat"]).max() <= 1e-10 * np.abs(so["smat"]).max()
    g.close()
