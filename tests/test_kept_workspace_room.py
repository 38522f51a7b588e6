"""What a context keeps between its post-processing calls goes where device
memory is short: operators that do not fit beside it are generated all the same.

Device memory is filled with one tensor that nothing reads or writes, up to
less than the operators take; the kept workspace is larger than they are.
"""
import numpy as np
import pytest

from mstm_b200 import configs as C

pytestmark = pytest.mark.gpu


def test_operators_take_the_room():
    import torch
    from mstm_b200 import api

    def cluster(n):
        pos, _ = C.rsa_sphere(n, 1.0, 0.1, seed=n)
        return api.SphereCluster(pos, np.ones(n), np.full(n, 1.5 + 0.02j), mie_epsilon=-9.0)

    rng = np.random.default_rng(1)
    f, g = cluster(120), cluster(120)
    x = rng.normal(size=(g.number_eqns, 2)) + 1j * rng.normal(size=(g.number_eqns, 2))
    want = f.sphereinteraction(x, con_tran=[0, 1])
    ops = f.operator_bytes()[0]
    f.close()
    T = 34
    tm = np.asfortranarray(rng.normal(size=(2 * T * (T + 2),) * 2) + 0.5j)
    before = torch.cuda.mem_get_info()[0]
    sm = g.ranorientscatmatrix(tm, T)["smat"]
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept > 1.5 * ops > 150e6
    leave = int(0.6 * ops)
    fill = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        y = g.sphereinteraction(x, con_tran=[0, 1])
    finally:
        del fill
        torch.cuda.empty_cache()
    # the same kernels on the same inputs, the order of FP64 sums apart
    assert np.abs(y - want).max() <= 1e-12 * np.abs(want).max()
    again = g.ranorientscatmatrix(tm, T)["smat"]   # the workspace comes back
    assert np.abs(again - sm).max() <= 1e-12 * np.abs(sm).max()
    g.close()


def test_scattering_matrix_needs_little():
    """400 spheres of order 3: coefficients, tables and the merge's work take below 64 MB."""
    import torch
    from mstm_b200 import api
    n = 400
    pos, _ = C.rsa_sphere(n, 1.0, 0.1, seed=n)
    g = api.SphereCluster(pos * 0.2, np.full(n, 0.2), np.full(n, 1.5 + 0.02j), mie_epsilon=-3.0)
    h = api.SphereCluster(pos[:4], np.ones(4), np.full(4, 1.5 + 0.02j), mie_epsilon=-3.0)
    h.scattering(np.ones((h.number_eqns, 2), complex), nangles=5)   # the kernels are loaded
    before = torch.cuda.mem_get_info()[0]
    g.scattering(np.ones((g.number_eqns, 2), complex), nangles=5)
    assert before - torch.cuda.mem_get_info()[0] <= 70e6   # two blocks of 32 MB and some tables
    g.close()
    h.close()
