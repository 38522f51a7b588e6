"""The sphere-node and frequency kernels of the FFT translation at the edges of
their splits: node orders of fewer rows than a thread takes and with rows left
over, more sphere or node elements than a CTA has threads, one to five columns
(groups of four and the rest) with transposes among them.

Bounds: against the oracle the single precision of the stored spectra, 1e-5 of
the largest value as in the matvec test; column groups against single columns
the same sums in another order of the node atomics, 1e-12 (FP64) and 1e-5
(FP32) of it.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,x,L,d_cell,node_order", [(30, 0.6, 3, 2.2, 1), (40, 0.7, 3, 2.5, 2), (40, 1.0, 5, 4.0, 6), (10, 4.0, 11, 12.0, 11)])
def test_columns_and_orders(n, x, L, d_cell, node_order):
    from mstm_b200 import api
    from oracle import oracle as O
    pos, _ = C.rsa_sphere(n, x, 0.15, seed=L)
    args = (pos, np.full(n, x), np.full(n, 1.4 + 0.01j))
    g, o = api.SphereCluster(*args, mie_epsilon=-float(L), precision="mixed"), O.Oracle(*args, mie_eps=-float(L), nthreads=8)
    ig, io = g.fft_setup(d_cell=d_cell, node_order=node_order), o.fft_setup(d_cell=d_cell, node_order=node_order)
    assert ig["cell_dim"] == io["cell_dim"] and ig["node_order"] == io["node_order"] == node_order
    rng = np.random.default_rng(L)
    x5 = rng.normal(size=(g.number_eqns, 5)) + 1j * rng.normal(size=(g.number_eqns, 5))
    ct = [0, 1, 1, 0, 1]
    yo = o.sphereinteraction(x5[:, :2], con_tran=ct[:2])
    assert np.abs(g.sphereinteraction(x5[:, :2], con_tran=ct[:2]) - yo).max() <= 1e-5 * np.abs(yo).max()
    for precision, tol in (("fp64", 1e-12), ("fp32", 1e-5)):
        for w in range(1, 6):
            y = g.translation_pass(x5[:, :w], ct[:w], precision)
            for k in range(w):
                y1 = g.translation_pass(x5[:, k:k + 1], ct[k:k + 1], precision)
                assert np.abs(y[:, k:k + 1] - y1).max() <= tol * np.abs(y1).max(), (precision, w, k)
    g.close()
