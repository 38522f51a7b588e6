"""Workloads this library is used for, as timed cases.

Each case is one call a program makes of the library, from the smallest
cluster to the largest aggregate: the matvec that drives a caller's own
iteration (the C ABI, vectors on the GPU), complete fixed-orientation solves
in FP64 and in mixed precision (touching aggregates, dilute clusters, mixed
radii, large orders, inclusions in a host, the FFT path), an ensemble of
configurations, the cluster T matrix with its orientation average, and the
scattering matrix of a solution.

`prepare` draws the spheres from the seed and sets the cluster up (layout, Mie
coefficients, FFT grid); `run` is the call; `exact` restates matvecs and
smaller solves in plain complex128 torch (dense translation matrices from a
quadrature of Wigner d products, a direct solve of the full system).
"""
import ctypes
import math

import numpy as np
import torch

from mstm_b200 import _lib, api, configs

LMAX = 16   # largest sphere order the library takes


# --------------------------------------------------------------------------
# what is measured
# --------------------------------------------------------------------------
def listed():
    return [
        # one interaction product of a caller's own BiCG on the benchmark
        # aggregate: a direct column and a conjugate-transpose column
        dict(name="matvec_aggregate500", kind="matvec", shape="aggregate", n=500, x=2.0, order=9, columns=2, transposed=True),
        # the same product for a lognormal mix of radii (orders 4 to 8)
        dict(name="matvec_mixed_radii300", kind="matvec", shape="radii", n=300, x=1.0, order=0, columns=2, transposed=True),
        # the smallest call: 20 spheres, where latency and launches count
        dict(name="solve_cluster20", kind="solve", shape="cluster", n=20, x=1.0, order=7, precision="mixed"),
        # drop-in FP64 solve of an odd-sized aggregate (the reference's BiCG)
        dict(name="solve_fp64_aggregate203", kind="solve", shape="aggregate", n=203, x=2.0, order=9, precision="fp64"),
        # the benchmark's workload: 500 touching monomers, tuned precision
        dict(name="solve_aggregate500", kind="solve", shape="aggregate", n=500, x=2.0, order=9, precision="mixed"),
        # particles of several sizes, orders by convergence
        dict(name="solve_mixed_radii150", kind="solve", shape="radii", n=150, x=1.0, order=0, precision="mixed"),
        # few large spheres: high orders
        dict(name="solve_fp64_large_spheres40", kind="solve", shape="cluster", n=40, x=5.0, order=14, precision="fp64"),
        # small inclusions in one host sphere
        dict(name="solve_host_inclusions600", kind="solve", shape="host", n=600, x=0.5, order=0, precision="mixed"),
        # many small particles, FFT translation
        dict(name="solve_fft_cylinder2500", kind="solve", shape="cylinder", n=2500, x=1.0, order=7, precision="mixed"),
        # 48 independent clusters of 15 to 40 spheres in one context
        dict(name="ensemble48", kind="ensemble", count=48, n=40, x=1.0, order=7),
        # cluster T matrix and its orientation-averaged scattering matrix
        dict(name="tmatrix_cluster60", kind="tmatrix", n=60, x=1.5, order=8),
        # scattering matrix of a solved aggregate
        dict(name="scattering_aggregate350", kind="scattering", n=350, x=2.0, order=9),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of these ranges."""
    kind = rng.choice(["matvec", "matvec", "solve", "solve", "solve", "solve", "ensemble", "tmatrix", "scattering"])
    if kind in ("matvec", "solve"):
        shape = rng.choice(["aggregate", "aggregate", "cluster", "cluster", "radii"] + (["host", "cylinder"] if kind == "solve" else []))
        x = round(rng.uniform(0.15, 2.2), 2)   # soot monomers upwards
        c = dict(kind=kind, shape=shape, x=x, order=configs.truncation_order(x))
        if shape in ("aggregate", "cluster"):
            c["n"] = _log(rng, 5, 420 if kind == "matvec" else 300)
            if rng.random() < 0.25:   # few large spheres
                c.update(n=_log(rng, 5, 40), x=round(rng.uniform(2.5, 5.0), 2))
                c["order"] = configs.truncation_order(c["x"])
        elif shape == "radii":
            c.update(n=_log(rng, 10, 300 if kind == "matvec" else 200), x=round(rng.uniform(0.7, 1.2), 2), order=0)
        elif shape == "host":
            c.update(n=_log(rng, 50, 700), x=round(rng.uniform(0.35, 0.6), 2), order=0)
        else:
            c.update(n=_log(rng, 700, 2500), x=round(rng.uniform(0.7, 1.0), 2))
            c["order"] = configs.truncation_order(c["x"])
        if kind == "matvec":
            c["columns"] = rng.choice([1, 2, 2, 3, 4])
            c["transposed"] = rng.random() < 0.6
        else:
            c["precision"] = "mixed" if shape == "cylinder" else rng.choice(["mixed", "mixed", "fp64"])
        return c
    x = round(rng.uniform(0.6, 1.5), 2)
    if kind == "ensemble":
        return dict(kind=kind, count=_log(rng, 8, 64), n=rng.randint(10, 48), x=x, order=configs.truncation_order(x))
    if kind == "tmatrix":
        return dict(kind=kind, n=_log(rng, 8, 60), x=x, order=configs.truncation_order(x))
    return dict(kind=kind, n=_log(rng, 30, 350), x=x, order=configs.truncation_order(x))


# --------------------------------------------------------------------------
# the spheres
# --------------------------------------------------------------------------
def _cylinder(n, radius, volume_fraction, seed):
    """Random sequential addition in a cylinder as long as it is wide; the
    candidates come in batches, each kept if no sphere already kept overlaps."""
    rng = np.random.default_rng(seed)
    rc = (n * 4.0 / 3.0 * math.pi * radius ** 3 / volume_fraction / (2.0 * math.pi)) ** (1.0 / 3.0)
    cell, side = 2.0 * radius, int(math.ceil(rc / radius)) + 2
    grid, kept = {}, []
    while len(kept) < n:
        u = rng.random((4 * n, 3))
        r, phi = (rc - radius) * np.sqrt(u[:, 0]), 2.0 * math.pi * u[:, 1]
        p = np.stack([r * np.cos(phi), r * np.sin(phi), (2.0 * u[:, 2] - 1.0) * (rc - radius)], axis=1)
        keys = np.floor(p / cell).astype(int) + side
        for q, k in zip(p.tolist(), keys.tolist()):
            if len(kept) == n:
                break
            ok = True
            for a in (-1, 0, 1):
                for b in (-1, 0, 1):
                    for c in (-1, 0, 1):
                        for o in grid.get((k[0] + a, k[1] + b, k[2] + c), ()):
                            if (q[0] - o[0]) ** 2 + (q[1] - o[1]) ** 2 + (q[2] - o[2]) ** 2 < cell * cell:
                                ok = False
            if ok:
                grid.setdefault(tuple(k), []).append(q)
                kept.append(q)
    return np.array(kept)


def _mixed_radii(n, x, volume_fraction, seed):
    """Spheres of lognormal radii about x (the quantiles of the distribution,
    clipped to 0.4 x .. 2 x), largest first, placed without overlap in a
    bounding sphere."""
    rng = np.random.default_rng(seed)
    z = [math.sqrt(2.0) * torch.erfinv(torch.tensor((2.0 * i + 1.0) / n - 1.0, dtype=torch.float64)).item() for i in range(n)]
    rad = np.clip(x * np.exp(0.4 * np.array(z)), 0.4 * x, 2.0 * x)[::-1].copy()
    bound = (np.sum(rad ** 3) / volume_fraction) ** (1.0 / 3.0)
    pos = np.zeros((0, 3))
    for r in rad:
        while True:
            v = rng.standard_normal((32, 3))
            v *= ((bound - r) * rng.random((32, 1)) ** (1.0 / 3.0)) / np.linalg.norm(v, axis=1, keepdims=True)
            d = np.linalg.norm(v[:, None, :] - pos[None], axis=2) if len(pos) else np.full((32, 1), np.inf)
            free = np.nonzero((d >= r + rad[None, :len(pos)] if len(pos) else d > 0).all(axis=1))[0]
            if len(free):
                pos = np.concatenate([pos, v[free[:1]]])
                break
    return pos, rad


def _index(seed):
    rng = np.random.default_rng([seed, 7])
    return complex(rng.uniform(1.45, 1.65), rng.uniform(0.005, 0.05))


def _spheres(case, seed):
    """positions, radii, refractive indices, mie_epsilon."""
    n, x, shape, m = case["n"], case["x"], case.get("shape", "cluster"), _index(seed)
    if shape == "aggregate":
        pos = configs.pca_aggregate(n, x, 1.8, 1.3, seed=seed)
    elif shape == "radii":
        pos, rad = _mixed_radii(n, x, 0.12, seed)
        return pos, rad, np.full(n, 1.55 + 0.02j), 1.0e-6
    elif shape == "host":
        w = configs.host_inclusions(n, x, 0.12, seed, inclusion_index=m)
        return w["pos"], w["radius"], w["ref_index"], 1.0e-5
    elif shape == "cylinder":
        pos = _cylinder(n, x, 0.2, seed)
    else:
        pos, bound = configs.rsa_sphere(n, x, 0.1, seed=seed)
        pos -= pos.mean(axis=0)   # of one extent whatever the seed
        pos *= (bound + x) / np.linalg.norm(pos, axis=1).max()
    return pos, np.full(n, x), np.full(n, m), -float(case["order"])


def _columns(order, columns, seed, device="cuda"):
    """Coefficient vectors as an iteration meets them: independent complex
    values, falling with the degree as a scattered field's do."""
    g = torch.Generator(device=device).manual_seed(seed)
    out = []
    for L in order:
        fall = torch.tensor([s[0] for s in _slots(L)], device=device, dtype=torch.float64).mul(-0.7).exp()
        fall = torch.cat([fall, fall])[None, :]
        out.append(torch.randn((columns, fall.shape[1]), generator=g, device=device, dtype=torch.complex128) * fall)
    return torch.cat(out, dim=1).contiguous()   # (columns, neqns): column-major neqns x columns


# --------------------------------------------------------------------------
# the calls
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        m = _index(seed)
        members = []
        for c in range(case["count"]):
            n = case["n"] - (7 * c) % (5 * case["n"] // 8)
            members.append((configs.rsa_sphere(n, case["x"], 0.1, seed=seed * 1000 + c)[0], np.full(n, case["x"]), m))
        return dict(case=case, cluster=api.SphereEnsemble(members, mie_epsilon=-float(case["order"])))
    pos, rad, ri, eps = _spheres(case, seed)
    precision = {"matvec": "fp64", "solve": case.get("precision")}.get(kind, "mixed")
    cluster = api.SphereCluster(pos, rad, ri, mie_epsilon=eps, precision=precision)
    state = dict(case=case, cluster=cluster)
    if kind == "matvec":
        k = case["columns"]
        ct = [int(case["transposed"] and r % 2 == 1) for r in range(k)]
        x = _columns(cluster.sphere_order, k, seed)
        state.update(x=x, y=torch.zeros_like(x), ct=(ctypes.c_int * k)(*ct), mm=(ctypes.c_int * k)(*([1] * k)))
        torch.cuda.synchronize()
        _product(state, 1)   # the pair operators, which such a program generates once
    elif case.get("shape") == "cylinder":
        cluster.fft_setup(cell_volume_fraction=0.2)
    elif kind == "tmatrix":
        state["order"] = cluster.t_matrix_order(1.0e-5, 60)
    elif kind == "scattering":
        state["amnp"] = cluster.fixedorsoln(eps=1.0e-8)["amnp"]
    return state


def _product(state, first):
    c = state["cluster"]
    _lib.check(_lib.lib().mstmg_interaction(c.ctx, state["case"]["columns"], state["x"].data_ptr(), state["y"].data_ptr(), state["ct"], state["mm"],
                                            first), "mstmg_interaction")


def run(state):
    kind, c = state["case"]["kind"], state["cluster"]
    if kind == "matvec":
        _product(state, 0)
        return state["y"]
    if kind in ("solve", "ensemble"):
        r = c.fixedorsoln(eps=1.0e-12)
        return dict(amnp=r["amnp"], qeff=r["qeff"], qtot=r["qtot"])
    if kind == "tmatrix":
        t = c.tmatrix_solution(state["order"], solution_eps=1.0e-12, convergence_eps=1.0e-6)
        s = c.ranorientscatmatrix(t["tmat"], t["t_matrix_order"])
        return dict(tmat=t["tmat"], qtot=t["qtot"], sm=s["sm"], smat=s["smat"])
    s = c.scattering(state["amnp"])
    return dict(smat=s["smat"], g=s["g"])


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _radii_order(x):
    """Mean order of spheres of size x at mie_epsilon 1e-6 (about)."""
    return max(3, int(round(x + 4.05 * x ** (1.0 / 3.0))))


def _pair_cost(L):
    """One pair, both directions, one column: operator values (folded
    rotations and the two axial modes) and real multiply-adds per column."""
    rot = sum((n + 1) ** 2 + n * n for n in range(1, L + 1))
    axial = L * L + 2 * sum((L - m + 1) ** 2 for m in range(1, L + 1))
    return rot + 2 * axial, 2 * 2 * (2 * 2 * rot + 4 * axial)


def _products(n, L, pairs, columns, real):
    values, fma = _pair_cost(L)
    vec = 2 * 8 * real // 4 * n * L * (L + 2) * 2
    return dict(bytes=float(pairs * values * real + columns * vec), flops=2.0 * pairs * fma * columns)


def work(case):
    kind, n = case["kind"], case["n"]
    L = case.get("order") or (_radii_order(case["x"]) if case.get("shape") == "radii" else 4)
    if kind == "ensemble":
        n, c = (11 * n) // 16, case["count"]
        one = _products(c * n, L, c * n * (n - 1) // 2, 2, 4)
        return {k: 20 * v for k, v in one.items()}
    pairs = n * (n - 1) // 2
    if kind == "matvec":
        return _products(n, L, pairs, case["columns"], 8)
    if kind == "solve":
        if case["shape"] == "cylinder":
            pairs = n * 30
        products = {"aggregate": 60, "cylinder": 45, "host": 20}.get(case["shape"], 25)
        if case["precision"] == "fp64":
            one, products = _products(n, L, pairs, 2, 8), 2 * products
        else:
            one = _products(n, L, pairs, 2, 4)
        return {k: products * v for k, v in one.items()}
    if kind == "tmatrix":
        T = int(round(case["x"] * (n / 0.1) ** (1.0 / 3.0) + 6))
        one = _products(n, L, pairs, 2 * T * (T + 2), 4)
        return {k: 12 * v for k, v in one.items()}
    T = int(round(2.2 * case["x"] * (n / 0.1) ** (1.0 / 3.0)))
    return dict(bytes=float(2 * n * 2 * L * (L + 2) * 16 + 2 * T * (T + 2) * 32), flops=2.0 * n * 2 * T ** 3 + 16.0 * T ** 4)


# --------------------------------------------------------------------------
# the same in plain complex128
# --------------------------------------------------------------------------
def _slots(L):
    """(n, m) of the entries of one mode of a sphere's block: a(0:L+1, 1:L),
    column-major; a(m, n) for m >= 0, a(n + 1, -m) for m < 0."""
    return [(col, row) if row <= col else (row - 1, -col) for col in range(1, L + 1) for row in range(L + 2)]


def _wigner(n, m, k, t):
    """Wigner d^n_{m k}(theta) at an array of angles (k = -1, 0, 1) by the
    three-term recurrence in the degree from its lowest one."""
    n0 = max(abs(m), abs(k))
    c, s, ct = np.cos(t / 2), np.sin(t / 2), np.cos(t)
    # at the lowest degree d is a single product of half-angle powers
    f = math.sqrt(math.factorial(2 * n0) / (math.factorial(n0 + m) * math.factorial(n0 - m) if abs(k) == n0 else math.factorial(n0 + k) * math.factorial(n0 - k)))
    if abs(m) == n0 and m >= 0:
        d = f * c ** (n0 + k) * (-s) ** (n0 - k)
    elif abs(m) == n0:
        d = f * c ** (n0 - k) * s ** (n0 + k)
    elif k == n0:
        d = f * c ** (n0 + m) * s ** (n0 - m)
    else:
        d = f * c ** (n0 - m) * (-s) ** (n0 + m)
    last, out = np.zeros_like(d), [d]
    for q in range(n0, n):
        a = math.sqrt(((q + 1) ** 2 - m * m) * ((q + 1) ** 2 - k * k))
        b = math.sqrt((q * q - m * m) * (q * q - k * k))
        mk = m * k / (q * (q + 1.0)) if q else 0.0
        new = ((2 * q + 1) * (q + 1) * (ct - mk) * d - ((q + 1) * b / q if q else 0.0) * last) / a
        last, d = d, new
        out.append(d)
    return out


class _Dense:
    """Dense translation matrices H(r) of VSWF coefficients up to order L, in
    the helicity basis (mode p is coupled to itself only)."""

    def __init__(self, L, device):
        self.L, self.dev = L, device
        mn = _slots(L)
        W = 2 * L
        xq, wq = np.polynomial.legendre.leggauss(2 * L + 2)
        t = np.arccos(xq)
        d1 = {}
        for k in (-1, 1):
            for m in range(-L, L + 1):
                for i, v in enumerate(_wigner(L, m, k, t)):
                    d1[max(abs(m), 1) + i, m, k] = v
        d0 = {}
        for v in range(-W, W + 1):
            for i, f in enumerate(_wigner(W, v, 0, t)):
                d0[abs(v) + i, v] = f
        A = np.array([d1[n, -m, -1] for n, m in mn])   # targets
        B = np.array([d1[n, m, 1] for n, m in mn])     # sources
        n_of, m_of = np.array([q[0] for q in mn]), np.array([q[1] for q in mn])
        nt, ns = n_of[:, None], n_of[None, :]
        v = m_of[None, :] - m_of[:, None]
        c = np.sqrt((2 * nt + 1.0) * (2 * ns + 1.0)) * np.where(m_of[None, :] % 2 == 0, 1.0, -1.0)
        par = (nt + ns)
        self.terms = []
        for w in range(W + 1):
            D3 = np.array([d0.get((w, q), np.zeros_like(t)) for q in range(-W, W + 1)])
            # the integral of d^nt_{-mt, -1} d^ns_{ms, 1} d^w_{ms - mt, 0}
            I = np.zeros(v.shape)
            for q in range(-W, W + 1):
                a, b = np.nonzero(v == q)
                if len(a):
                    I[a, b] = np.einsum("zq,zq,q->z", A[a], B[b], wq * D3[-q + W])
            ok = (np.abs(nt - ns) <= w) & (w <= nt + ns) & (np.abs(v) <= w)
            base = np.where(ok, -c * I * (2 * w + 1) / 2.0, 0.0)
            e = (nt - ns + w) % 4                       # i^(nt - ns + w)
            val = np.where(e == 0, 1.0, np.where(e == 1, 1j, np.where(e == 2, -1.0, -1j))) * base
            odd = (par - w) % 2 == 1
            self.terms.append([torch.tensor(z, device=device, dtype=torch.complex128) for z in (val, np.where(odd, -val, val))])
        self.v = torch.tensor(v + W, device=device)
        self.nq = W

    def blocks(self, rv, index):
        """(modes 2, pairs, targets, sources) for pair vectors rv (pairs, 3)."""
        W = self.nq
        r = rv.norm(dim=1)
        ct = rv[:, 2] / r
        z = r * index
        h = [-1j * torch.exp(1j * z) / z, -torch.exp(1j * z) * (1j + z) / z / z]
        for n in range(2, W + 1):
            h.append((2 * n - 1) / z * h[-1] - h[-2])
        phi = torch.atan2(rv[:, 1], rv[:, 0])
        e = torch.exp(1j * phi[:, None] * torch.arange(-W, W + 1, device=self.dev)[None, :])
        st = torch.sqrt(torch.clamp((1 - ct) * (1 + ct), min=0.0))
        p = {}
        for m in range(W + 1):   # normalised Legendre functions sqrt((w-m)!/(w+m)!) P_w^m, Condon-Shortley phase
            p[m, m] = torch.ones_like(ct) if m == 0 else -p[m - 1, m - 1] * st * math.sqrt((2 * m - 1) / (2 * m))
            for w in range(m, W):
                low = math.sqrt((w * w - m * m)) * p[m, w - 1] if w > m else 0.0
                p[m, w + 1] = ((2 * w + 1) * ct * p[m, w] - low) / math.sqrt((w + 1) ** 2 - m * m)
        H = [0.0, 0.0]
        for w in range(W + 1):
            y = torch.zeros((len(r), 2 * W + 1), dtype=torch.complex128, device=self.dev)
            for m in range(w + 1):
                y[:, W + m] = p[m, w]
                y[:, W - m] = (-1) ** m * p[m, w]
            g = (y * e * h[w][:, None])[:, self.v]
            for q in (0, 1):
                H[q] = H[q] + g * self.terms[w][q]
        return torch.stack(H)


def _mie(x, m, L, device):
    """2 x 2 helicity Mie matrices per degree, (L, 2, 2)."""
    mx = m * x
    top = int(max(abs(mx), x) + 4 * max(abs(mx), x) ** (1 / 3.0) + 40)
    D = np.zeros(top + 1, complex)
    for n in range(top, 0, -1):
        D[n - 1] = n / mx - 1.0 / (D[n] + n / mx)
    Dx = np.zeros(top + 1)
    for n in range(top, 0, -1):
        Dx[n - 1] = n / x - 1.0 / (Dx[n] + n / x)
    psi, chi = [math.sin(x)], [math.cos(x)]
    chi.append(math.cos(x) / x + math.sin(x))
    for n in range(1, L + 1):
        psi.append(psi[-1] / (Dx[n] + n / x))
        chi.append((2 * n + 1) / x * chi[n] - chi[n - 1])
    out = np.zeros((L, 2, 2), complex)
    for n in range(1, L + 1):
        xi, xi1 = psi[n] - 1j * chi[n], psi[n - 1] - 1j * chi[n - 1]
        a = ((D[n] / m + n / x) * psi[n] - psi[n - 1]) / ((D[n] / m + n / x) * xi - xi1)
        b = ((m * D[n] + n / x) * psi[n] - psi[n - 1]) / ((m * D[n] + n / x) * xi - xi1)
        out[n - 1] = -0.5 * np.array([[a + b, a - b], [a - b, a + b]])
    return torch.tensor(out, device=device)


def _exact_system(case, seed, device):
    """Spheres, their orders and Mie matrices, and the padded slot of every
    entry of a coefficient vector."""
    pos, rad, ri, eps = _spheres(case, seed)
    order = [int(round(-eps))] * len(rad)
    if eps > 0:   # orders by the convergence test of the Mie efficiency
        order = []
        for x, m in zip(rad, ri):
            stop = int(round(x + 4.0 * x ** (1.0 / 3.0))) + 5
            M = _mie(x, m, stop, "cpu")
            q = np.array([-(2 * n + 1) * 2 * M[n - 1, 0, 0].real.item() for n in range(1, stop + 1)])
            part = np.cumsum(q)
            order.append(int(np.nonzero(np.abs(1 - part / part[-1]) < eps)[0][0]) + 1)
    L = max(order)
    where = {s: i for i, s in enumerate(_slots(L))}
    nb = L * (L + 2)
    slot, mie = [], torch.zeros((len(rad), 2, 2, nb), dtype=torch.complex128, device=device)
    deg = torch.tensor([s[0] - 1 for s in _slots(L)], device=device)
    for i, l in enumerate(order):
        own = [where[s] for s in _slots(l)]
        slot.append(torch.tensor([(i * 2 + p) * nb + q for p in (0, 1) for q in own]))
        M = torch.zeros((L, 2, 2), dtype=torch.complex128, device=device)
        M[:l] = _mie(rad[i], ri[i], l, device)
        mie[i] = M[deg].permute(1, 2, 0)
    return torch.tensor(pos, device=device), order, L, nb, torch.cat(slot).to(device), mie


def exact(case, seed):
    """The product, or the solution of a solve of up to 15,000 unknowns
    (iterated to a residual by `run`), from dense matrices."""
    kind, shape, n = case["kind"], case.get("shape"), case["n"]
    if kind not in ("matvec", "solve") or shape in ("host", "cylinder"):
        return None
    if kind == "solve" and n * 2 * LMAX * (LMAX + 2) > 15000 and n * 2 * (case["order"] or 9) * ((case["order"] or 9) + 2) > 15000:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pos, order, L, nb, slot, mie = _exact_system(case, seed, dev)
    dense = _Dense(L, dev)
    if kind == "solve":
        H = torch.zeros((n, 2, nb, n, 2, nb), dtype=torch.complex128, device=dev)
    else:
        x = _columns(order, case["columns"], seed, dev)
        k = case["columns"]
        ct = [bool(case["transposed"] and r % 2 == 1) for r in range(k)]
        pad = torch.zeros((k, n * 2 * nb), dtype=torch.complex128, device=dev)
        pad[:, slot] = x
        pad = pad.view(k, n, 2, nb)
        # a transposed column starts with the adjoint of the Mie multiply
        u = torch.stack([torch.einsum("ipqs,ips->iqs", mie.conj(), pad[r]) if ct[r] else pad[r] for r in range(k)])
        y = torch.zeros_like(u)
        keep = torch.zeros(n * 2 * nb, dtype=torch.bool, device=dev)
        keep[slot] = True
        keep = keep.view(n, 2, nb)
        plain, trans = [r for r in range(k) if not ct[r]], [r for r in range(k) if ct[r]]
    step = max(1, 2 ** 27 // (nb * nb * 8))
    for i in range(n):
        others = torch.tensor([j for j in range(n) if j != i], device=dev)
        for part in others.split(step):
            B = dense.blocks(pos[i] - pos[part], 1.0)
            if kind == "solve":
                for p in (0, 1):
                    H[i, p][:, part, p, :] = B[p].permute(1, 0, 2)
            else:
                if plain:
                    y[plain, i] += torch.einsum("pjts,rjps->rpt", B, u[plain][:, part])
                if trans:
                    z = torch.einsum("pjts,rpt->rjps", B.conj(), u[trans][:, i])
                    for a, r in enumerate(trans):
                        y[r].index_add_(0, part, z[a])
    if kind == "matvec":
        y = y * keep
        y = torch.stack([y[r] if ct[r] else torch.einsum("ipqs,iqs->ips", mie, y[r]) for r in range(k)])
        return y.reshape(k, -1)[:, slot]
    f = torch.zeros((n, 2, nb, 2), dtype=torch.complex128, device=dev)
    index = {s: i for i, s in enumerate(_slots(L))}
    for d in range(1, L + 1):   # the +z plane wave, both polarisations
        amp = 4.0 * 1j ** (d + 1) * math.sqrt((2 * d + 1) / 2.0) / 4.0
        f[:, 0, index[d, 1], 0], f[:, 1, index[d, -1], 0] = amp, -amp
        f[:, 0, index[d, 1], 1], f[:, 1, index[d, -1], 1] = -1j * amp, -1j * amp
    f = f * torch.exp(1j * pos[:, 2])[:, None, None, None]
    A = -torch.einsum("ipqs,iqszot->ipszot", mie, H.view(n, 2, nb, n, 2, nb)).reshape(n * 2 * nb, n * 2 * nb)
    del H
    b = torch.einsum("ipqs,iqsc->ipsc", mie, f).reshape(n * 2 * nb, 2)
    A = A[slot][:, slot]
    A.diagonal().add_(1.0)
    return dict(amnp=torch.linalg.solve(A, b[slot]), qeff=None, qtot=None)
