"""The pair kernel's way out when a copy does not arrive in time: every warp of
a CTA leaves, the copies in flight are waited for, no unfinished sum reaches
the result, the status says so, and the context goes on working.

The copies themselves all complete; a wait at a CTA's first pair or a later one
is taken to have run out, for instances with orders at compile time, at run
time with two record buffers, and with one (order 16), with many pairs a CTA
and with few.

Bound of the passes that follow: the same kernel on the same inputs, the order
of FP64 sums apart: 1e-12 of the largest value.
"""
import ctypes

import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,order", [(120, 4), (90, 9), (60, 0), (12, 13), (6, 16), (40, 16)])
def test_waits_that_run_out(n, order):
    from mstm_b200 import _lib, api
    L = _lib.lib()
    rad = np.full(n, max(0.3, 0.35 * order))
    if order == 0:
        rad = np.exp(np.random.default_rng(n).uniform(-0.6, 0.6, n))
    pos, _ = C.rsa_sphere(n, rad.max(), 0.15, seed=n)
    g = api.SphereCluster(pos, rad, np.full(n, 1.4 + 0.01j), mie_epsilon=-float(order) if order else 1e-6)
    rng = np.random.default_rng(n)
    x = np.asfortranarray(rng.normal(size=(g.number_eqns, 3)) + 1j * rng.normal(size=(g.number_eqns, 3)))
    ct = np.array([0, 1, 0], np.int32)
    want = g.translation_pass(x, ct, "fp64")
    s = np.abs(want).max()
    for pair in (0, 1, 2, 3, 4, 5, 17, 1 << 30):
        y = np.full_like(x, np.nan)
        status = ctypes.c_int(1)
        assert L.mstmg_selftest_pass_wait(g.ctx, pair, 3, ct.ctypes.data, x.ctypes.data, y.ctypes.data, ctypes.byref(status)) == 0
        if pair == 0:
            assert status.value == -2   # MSTMG_ERR_CUDA
            assert np.abs(y).max() == 0.0
        assert status.value == -2 or np.abs(y - want).max() <= 1e-12 * s   # no CTA came that far
        if pair == 1 << 30:
            assert status.value == 0
        assert np.abs(g.translation_pass(x, ct, "fp64") - want).max() <= 1e-12 * s
    g.close()
