"""The regular translation of a sphere's expansion to the cluster origin against
exact coupling coefficients: spheres on the z axis, where no rotation enters,
so that an origin coefficient is the sum over the source degrees of axial
elements (axialtrancoefinit, december2023/mstm-modules-33.f90:1680-1722), in
80-bit arithmetic from Clebsch-Gordan coefficients by Racah's formula in
integers and Bessel functions by Miller's recurrence.

Bound, of the largest origin coefficient: an element has errors of 4.4e-15
(couplings) and 2.5e-15 (Bessel functions) of its largest term, 5e-15 together,
and those of up to 14 source degrees add as their root: 2e-14.
"""
import math
from functools import lru_cache

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


@lru_cache(None)
def _row(m, n, l):
    """C_w of (m, n) and (-m, l), w = |n - l| .. n + l: Clebsch-Gordan <n m; l -m | w 0>."""
    f, out = math.factorial, {}
    for w in range(abs(n - l), n + l + 1):
        lo, hi = max(0, l - w - m, n - w - m), min(n + l - w, n - m, l - m)
        den = math.lcm(*(f(t) * f(n + l - w - t) * f(n - m - t) * f(l - m - t) * f(w - l + m + t) * f(w - n + m + t) for t in range(lo, hi + 1)))
        num = sum((-1) ** t * (den // (f(t) * f(n + l - w - t) * f(n - m - t) * f(l - m - t) * f(w - l + m + t) * f(w - n + m + t)))
                  for t in range(lo, hi + 1))
        p = num * num * (2 * w + 1) * f(w + n - l) * f(w - n + l) * f(n + l - w) * f(w) ** 2 * f(n - m) * f(n + m) * f(l + m) * f(l - m)
        q = den * den * f(n + l + w + 1)
        r = math.isqrt((p << 160) // q)     # sqrt(p / q) 2^80
        out[w] = np.copysign(np.ldexp(LD(r >> max(0, r.bit_length() - 64)), max(0, r.bit_length() - 64) - 80), LD(num))
    return out


def _bessel(z, kmax):
    a, b, j = LD(0), LD("1e-2000"), [LD(0)] * (kmax + 1)
    for k in range(kmax + int(z) + 100, 0, -1):
        if k <= kmax:
            j[k] = b
        a, b = b, (2 * k + 1) / z * b - a
    j[0] = b
    s = np.sin(z) / z / b if abs(np.sin(z)) > 0.1 else (np.sin(z) / z - np.cos(z)) / z / a
    return [s * v for v in j]


def _index(m, n, p, L):
    return m + (L + 2) * (n - 1) + (L + 2) * L * p if m >= 0 else n + 1 + (L + 2) * (-m - 1) + (L + 2) * L * p


@pytest.mark.parametrize("L,d", [(14, 35.0), (14, 22.0), (9, 13.8), (4, 1.6)])
def test_origin_coefficients(L, d):
    from mstm_b200 import api
    g = api.SphereCluster(np.array([[0, 0, -d], [0, 0, d]]), np.ones(2), np.full(2, 1.5 + 0.01j), mie_epsilon=-float(L))
    rng = np.random.default_rng(L)
    a = np.zeros((g.number_eqns, 2), complex, order="F")
    nb = 2 * L * (L + 2)
    a[:nb] = rng.normal(size=(nb, 2)) + 1j * rng.normal(size=(nb, 2))
    r = g.scattering(a, max_t_order=100, nangles=3)
    g.close()
    T = r["t_matrix_order"]
    j = _bessel(LD(d), T + L)
    want = np.zeros((2 * T * (T + 2), 2), np.clongdouble)
    for n in range(1, T + 1):
        for l in range(1, L + 1):
            v2 = _row(-1, n, l)
            for ma in range(0, min(n, l) + 1):
                v1, s = _row(-ma, n, l), [LD(0), LD(0)]
                for w in v1:
                    ri = 1 if (n - l + w) % 4 in (0, 1) else -1
                    s[(w - abs(n - l)) % 2] -= (-1) ** ma * np.sqrt(LD(2 * n + 1) * LD(2 * l + 1)) * v1[w] * v2[w] * ri * j[w]
                z = (s[0] + 1j * s[1], s[0] - 1j * s[1])
                for m in {ma, -ma}:
                    for p in range(2):
                        x = z[0 if m == 0 else p if m > 0 else 1 - p] * a[_index(m, l, p, L)]
                        want[_index(m, n, 0, T)] += x
                        want[_index(m, n, 1, T)] += x if p == 0 else -x
    assert np.abs(r["amnp0"] - want).max() <= 2e-14 * np.abs(want).max()
