"""Two threads in one context's calls that take their own inputs and results:
FP32 passes of different widths (their FP64 copies of the columns are one
buffer of the context) and T matrices (one call has the kept work, the other
its own) give what they give alone.

Bounds: FP64 sums in another order, 1e-12 of the largest value, rounded once
more to FP32 by a pass: 2e-7.  T matrices solved to 1e-10 of the right-hand
sides, times the inverse of I - M H, below 10 for these spheres: 1e-8.
"""
import threading

import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


def _together(*calls):
    errors = []

    def run(f):
        try:
            f()
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=run, args=(f,)) for f in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_fp32_passes():
    from mstm_b200 import api
    n = 60
    pos, _ = C.rsa_sphere(n, 1.0, 0.15, seed=n)
    g = api.SphereCluster(pos, np.ones(n), np.full(n, 1.5 + 0.02j), mie_epsilon=-6.0, precision="mixed", tensor_core=-1)
    rng = np.random.default_rng(1)

    def work(cols):
        x = rng.normal(size=(g.number_eqns, cols)) + 1j * rng.normal(size=(g.number_eqns, cols))
        y = g.translation_pass(x, None, "fp32")
        return x, y, np.abs(y).max()

    def repeat(x, y, s):
        for _ in range(40):
            assert np.abs(g.translation_pass(x, None, "fp32") - y).max() <= 2e-7 * s

    a, b = work(1), work(2)   # the wider buffers come while both threads run
    xw = [rng.normal(size=(g.number_eqns, w)) + 0j for w in range(3, 12)]

    def widen():
        for x in xw:
            g.translation_pass(x, None, "fp32")
            repeat(*b)

    _together(lambda: repeat(*a), lambda: repeat(*b), widen)
    g.close()


def test_t_matrices():
    from mstm_b200 import api
    n = 8
    pos, _ = C.rsa_sphere(n, 1.0, 0.1, seed=n)
    g = api.SphereCluster(pos, np.ones(n), np.full(n, 1.5 + 0.02j), mie_epsilon=-4.0)
    T = g.t_matrix_order()
    kw = dict(solution_eps=1e-20, convergence_eps=0.0)
    want = {t: g.tmatrix_solution(t, **kw)["tmat"] for t in (T, T - 2)}

    def check(t):
        for _ in range(4):
            got = g.tmatrix_solution(t, **kw)["tmat"]
            assert np.abs(got - want[t]).max() <= 1e-8 * np.abs(want[t]).max()

    _together(lambda: check(T), lambda: check(T - 2))
    g.close()
