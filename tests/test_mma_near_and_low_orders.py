"""The pair kernel (translate_mma.cu) against the order-generic kernel
(translate.cu) where no other test puts them side by side: the near pairs of the
FFT path, grouped by cells, of one order and of several, and spheres of orders 1
and 2, which come to the tiles when translation_switch_order is lowered.

Bounds: both kernels sum the same products in FP64 in different orders, at most
600 terms a value in each of three products: 1e-12 of the largest output (the
far field is the same FP64 transforms on both sides).  An FP32 pass rounds its
columns to FP32 once: 2e-6 of it.
"""
import ctypes

import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread,order,n", [(1.0, 7, 260), (1.0, 4, 333), (1.6, 0, 240)])
def test_near_pairs_of_the_fft_path(spread, order, n):
    from mstm_b200 import api
    rng = np.random.default_rng(n)
    rad = np.exp(rng.uniform(-np.log(spread), np.log(spread), n)) if spread > 1 else np.ones(n)
    pos, _ = C.rsa_cylinder(n, spread, 0.2, 1.0, seed=3)
    rad = rad[:len(pos)]
    kw = dict(mie_epsilon=-float(order) if order else 1e-6, precision="mixed")
    a = api.SphereCluster(pos, rad, np.full(len(pos), 1.4 + 0.01j), **kw)
    b = api.SphereCluster(pos, rad, np.full(len(pos), 1.4 + 0.01j), generic_kernel=True, **kw)
    for g in (a, b):
        f = g.fft_setup(d_cell=4.5)
    assert f["near_pairs"] > len(pos)
    for ct in ([0, 1], [1], [0, 1, 1]):
        x = rng.normal(size=(a.number_eqns, len(ct))) + 1j * rng.normal(size=(a.number_eqns, len(ct)))
        want = b.translation_pass(x, ct, "fp64")
        s = np.abs(want).max()
        assert np.abs(a.translation_pass(x, ct, "fp64") - want).max() <= 1e-12 * s, ct
    a.close()
    b.close()


@pytest.mark.parametrize("orders", [(1,), (2,), (1, 2, 3, 5)])
def test_orders_below_the_usual_switch(orders):
    from mstm_b200 import _lib
    L = _lib.lib()
    n = 30
    pos, _ = C.rsa_sphere(n, 1.0, 0.1, seed=n)
    ri = np.tile([1.4, 0.01], (n, 1))
    rng = np.random.default_rng(n)
    # orders by convergence: radii that give the wanted ones at 1e-4
    pick = {1: 0.02, 2: 0.2, 3: 0.45, 5: 1.0}
    rad = np.array([pick[orders[i % len(orders)]] for i in range(n)])
    out, y = [], {}
    for generic in (0, 1):
        opts = _lib.MstmgOpts()
        L.mstmg_default_opts(ctypes.byref(opts))
        opts.precision, opts.translation_switch_order, opts.generic_kernel = 1, 1, generic
        ctx = ctypes.c_void_p()
        p = [np.ascontiguousarray(v, np.float64) for v in (pos, rad, ri)]
        assert L.mstmg_ctx_create(ctypes.byref(ctx), n, p[0].ctypes.data, p[1].ctypes.data, p[2].ctypes.data, 1e-4 if len(orders) > 1 else -float(orders[0]),
                                  ctypes.byref(opts)) == 0, L.mstmg_last_error()
        out.append(ctx)
    ne = L.mstmg_neqns(out[0])
    x = np.asfortranarray(rng.normal(size=(ne, 3)) + 1j * rng.normal(size=(ne, 3)))
    ct = np.array([0, 1, 0], np.int32)
    for generic, ctx in enumerate(out):
        for prec in (0, 1):
            r = np.zeros_like(x)
            assert L.mstmg_translation_pass(ctx, prec, 3, ct.ctypes.data, x.ctypes.data, r.ctypes.data) == 0
            y[generic, prec] = r
    so = np.zeros(n, np.int32)
    L.mstmg_sphere_orders(out[0], so.ctypes.data, None)
    assert min(so) < 3 and (len(set(so)) > 1) == (len(orders) > 1)
    s = np.abs(y[1, 0]).max()
    assert s > 0 and np.abs(y[0, 0] - y[1, 0]).max() <= 1e-12 * s
    assert np.abs(y[0, 1] - y[1, 0]).max() <= 2e-6 * s
    for ctx in out:
        L.mstmg_ctx_destroy(ctx)
