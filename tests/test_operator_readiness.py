"""Spheres whose pairs are partly dense records (an order below
translation_switch_order) and partly rotation records: whichever precision is
asked for first, every later call finds the records of its own precision at the
present positions.

Bounds: the records are FP64 sums of the oracle's terms, 1e-12 of the largest
value as in the other matvec comparisons; FP32 columns and dense records are
rounded once or twice, sums of at most 300 terms: 1e-5.  T matrices of two
contexts differ by their residuals, 1e-10 of the right-hand sides, times the
inverse of I - M H, below 10 for these spheres: 1e-8 of the largest element.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RAD = np.array([1.0] * 6 + [0.05] * 4)
RI = np.array([1.5 + 0.01j] * 6 + [1.6 + 0.1j] * 4)


def _positions(seed):
    rng = np.random.default_rng(seed)
    pos = []
    while len(pos) < len(RAD):
        p = rng.uniform(-5, 5, 3)
        if all(np.linalg.norm(p - q) > 2.2 for q in pos):
            pos.append(p)
    return np.array(pos)


def _first_fp32(g, how, x):
    if how == "pass":
        return g.translation_pass(x, [0, 1], "fp32")
    g.time_translation("mixed", 2, 1)
    return None


@pytest.mark.parametrize("how", ["pass", "time"])
@pytest.mark.parametrize("small", [10, 8])   # dense pairs beside rotated ones, and a cluster of two orders with few of them
def test_fp32_before_fp64(oracle_mod, how, small):
    from mstm_b200 import api
    rad, ri = RAD[:small], RI[:small]
    kw = dict(mie_epsilon=1e-6)
    g = api.SphereCluster(_positions(1)[:small], rad, ri, **kw)
    assert min(g.sphere_order) < 3 <= max(g.sphere_order)
    rng = np.random.default_rng(2)
    x = rng.normal(size=(g.number_eqns, 2)) + 1j * rng.normal(size=(g.number_eqns, 2))
    for seed in (1, 3):   # a new context, then other positions
        pos = _positions(seed)[:small]
        if seed != 1:
            g.set_positions(pos)
        y32 = _first_fp32(g, how, x)
        f = api.SphereCluster(pos, rad, ri, **kw)
        want = f.translation_pass(x, [0, 1], "fp64")
        s = np.abs(want).max()
        if y32 is not None:
            assert np.abs(y32 - want).max() <= 1e-5 * s
        assert np.abs(g.translation_pass(x, [0, 1], "fp64") - want).max() <= 1e-12 * s
        f.close()
        o = oracle_mod.Oracle(pos, rad, ri, mie_eps=1e-6, store_matrix=True, nthreads=4)
        yo = o.sphereinteraction(x, con_tran=[0, 1])
        assert np.abs(g.sphereinteraction(x, con_tran=[0, 1]) - yo).max() <= 1e-12 * np.abs(yo).max()
    g.close()


def test_t_matrix_after_fp32_pass():
    from mstm_b200 import api
    pos = _positions(5)
    g, f = (api.SphereCluster(pos, RAD, RI, mie_epsilon=1e-6) for _ in range(2))
    _first_fp32(g, "pass", np.ones((g.number_eqns, 2), complex))
    kw = dict(t_matrix_order=4, solution_eps=1e-20, convergence_eps=0.0)
    f.t_matrix_order(1e-5, 4)
    g.t_matrix_order(1e-5, 4)
    want, got = f.tmatrix_solution(**kw)["tmat"], g.tmatrix_solution(**kw)["tmat"]
    assert np.abs(got - want).max() <= 1e-8 * np.abs(want).max()
    f.close()
    g.close()
