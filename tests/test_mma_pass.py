"""The FP64 tensor-core translation pass (translate_mma.cu) against the
order-generic kernel (translate.cu) at the edges of its tiles: every sphere
order with an instance of its own and the larger ones, mixed orders, partial
and single-sphere tiles, tile groups of 1, 2 and 4 spheres, odd column counts
and conjugate-transpose patterns.

Bounds: both kernels sum the same products in FP64 in different orders, at
most 2 L (L + 2) terms a value in each of three products; 600 terms of
relative rounding 1.1e-16 stay below 1e-12 of the largest output.  An FP32
pass rounds its columns to FP32 once on the way out: 2e-6 of it.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


def _pair(pos, rad, ri, eps):
    from mstm_b200 import api
    kw = dict(mie_epsilon=eps, precision="mixed")
    return api.SphereCluster(pos, rad, ri, **kw), api.SphereCluster(pos, rad, ri, generic_kernel=True, **kw)


def _compare(a, b, patterns, seed):
    rng = np.random.default_rng(seed)
    # values falling with the degree as a field's do, so that every degree counts
    fall = np.concatenate([np.tile([2.0 ** -(row if row > col else col) for col in range(1, L + 1) for row in range(L + 2)], 2)
                           for L in a.sphere_order])
    for ct in patterns:
        x = (rng.normal(size=(a.number_eqns, len(ct))) + 1j * rng.normal(size=(a.number_eqns, len(ct)))) * fall[:, None]
        y = b.translation_pass(x, ct, "fp64")
        s = np.abs(y).max()
        assert np.isfinite(s) and s > 0
        assert np.abs(a.translation_pass(x, ct, "fp64") - y).max() <= 1e-12 * s, ct
        assert np.abs(a.translation_pass(x, ct, "fp32") - y).max() <= 2e-6 * s, ct
    a.close()
    b.close()


@pytest.mark.parametrize("L", list(range(3, 17)))
def test_every_order(L):
    n = 5 if L > 10 else 9
    x = max(0.3, 0.35 * L)
    pos, _ = C.rsa_sphere(n, x, 0.15, seed=L)
    _compare(*_pair(pos, np.full(n, x), np.full(n, 1.4 + 0.01j), -float(L)), ([0, 1], [1], [0, 1, 1]), L)


@pytest.mark.parametrize("n,L", [(2, 7), (3, 9), (123, 6), (241, 4)])
def test_tile_edges(n, L):
    """One pair, one sphere left over, tiles of 2 x 2 and of 4 x 4 spheres with partial ones."""
    pos, _ = C.rsa_sphere(n, 1.0, 0.12, seed=n)
    _compare(*_pair(pos, np.full(n, 1.0), np.full(n, 1.4 + 0.01j), -float(L)), ([0], [1, 0, 1], [0, 1] * 2), n)


@pytest.mark.parametrize("n,spread", [(7, 2.5), (40, 2.0), (130, 1.6)])
def test_mixed_orders(n, spread):
    """Pairs of unequal orders in both directions, in one or several launch groups."""
    rng = np.random.default_rng(n)
    rad = np.exp(rng.uniform(-np.log(spread), np.log(spread), n))
    pos, _ = C.rsa_sphere(n, spread, 0.15, seed=n)
    a, b = _pair(pos, rad, np.full(n, 1.5 + 0.01j), 1e-6)
    assert len(set(a.sphere_order)) > 1
    _compare(a, b, ([0, 1], [1], [1, 0, 0, 1, 1]), n)
