"""The workspace a context keeps for its post-processing calls: calls of
growing and shrinking sizes in turn, and from two threads at once (one works
in the kept blocks, the other in its own), give what a fresh context gives.

Bound: the same kernels on the same inputs; only the order of the FP64
atomics differs: 1e-12 of the largest value.
"""
import threading

import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


def _cluster(n, spread):
    from mstm_b200 import api
    pos, _ = C.rsa_sphere(n, 1.0, 0.1, seed=n)
    g = api.SphereCluster(pos * spread, np.ones(n), np.full(n, 1.5 + 0.02j), mie_epsilon=-5.0)
    rng = np.random.default_rng(n)
    a = np.asfortranarray(rng.normal(size=(g.number_eqns, 2)) + 1j * rng.normal(size=(g.number_eqns, 2)))
    return g, a


@pytest.mark.parametrize("n", [4, 30])
def test_repeated_and_concurrent_calls(n):
    g, a = _cluster(n, 1.5)
    f, _ = _cluster(n, 1.5)
    want = f.scattering(a)
    scale = np.abs(want["smat"]).max()
    rng = np.random.default_rng(1)
    T = 12
    tm = np.asfortranarray(rng.normal(size=(2 * T * (T + 2),) * 2) + 0.5j)
    ro = f.ranorientscatmatrix(tm, T)["smat"]

    def check():
        assert np.abs(g.scattering(a)["smat"] - want["smat"]).max() <= 1e-12 * scale

    check()
    assert np.abs(g.ranorientscatmatrix(tm, T)["smat"] - ro).max() <= 1e-12 * np.abs(ro).max()
    check()
    assert g.t_matrix_order() == f.t_matrix_order()
    errors = []

    def worker():
        try:
            for _ in range(8):
                check()
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=worker) for _ in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    g.close()
    f.close()
