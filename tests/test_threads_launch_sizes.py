"""Contexts of their own driven by threads at once, their launches of one kernel
with different amounts of shared memory: none is refused, and the results are
those of one thread.

Bounds: the same kernels on the same inputs, the order of FP64 sums apart: 1e-12
of the largest value.
"""
import threading

import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


def _cluster(n, order):
    from mstm_b200 import api
    pos, _ = C.rsa_sphere(n, 1.0, 0.12, seed=n)
    g = api.SphereCluster(pos, np.ones(n), np.full(n, 1.5 + 0.02j), mie_epsilon=-float(order))
    rng = np.random.default_rng(n)
    return g, np.asfortranarray(rng.normal(size=(g.number_eqns, 2)) + 1j * rng.normal(size=(g.number_eqns, 2)))


def _pass(n, order):
    g, x = _cluster(n, order)
    return g, lambda: g.translation_pass(x, [0, 1], "fp64")


def _scattering(n, order, most):
    g, x = _cluster(n, order)
    return g, lambda: g.scattering(x, max_t_order=most, nangles=5)["smat"]


@pytest.mark.parametrize("make", [
    # tiles of single spheres and of 2 x 2: accumulators of two sizes
    lambda: [_pass(5, 8), _pass(130, 8), _pass(5, 8)],
    # tables of the merge to the origin and of its expansion by the order
    lambda: [_scattering(6, 4, 6), _scattering(60, 4, 40), _scattering(8, 3, 4)],
], ids=["passes", "scattering"])
def test_launches_of_different_sizes(make):
    ctx = make()
    want = [f() for _, f in ctx]
    errors = []

    def run(f, y):
        try:
            for _ in range(150):
                assert np.abs(f() - y).max() <= 1e-12 * np.abs(y).max()
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=run, args=(f, y)) for (_, f), y in zip(ctx, want)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for g, _ in ctx:
        g.close()
