"""Performance cases of libstokes_gb300: the calls that programs built on it
spend their time in, over the sizes and options they use.

A libstokes program is linked against the library and calls
``atimes_ewald_3all`` on host vectors, in FP64 unless it asks for mixed
precision; a GPU-resident program calls the ``*_dev`` forms on device buffers.
Suspensions are equal (or unequal) non-overlapping spheres in a cubic periodic
box at volume fractions of 0.05 to 0.35, generalised forces are N(0, 1).

Not among the cases: the iterative solves.  They chain the products below with
a stopping test, so where they stop (and how far from the solution) follows
the last digit of every product.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import libstokes_gb300 as L
from libstokes_gb300 import abi

NC = (3, 6, 11)             # components per particle: F, FT, FTS
FP64_EPS = 1e-12            # libstokes' usual Ewald tolerance
PAIR_FLOPS = (89, 184, 754)  # one real-space pair term: F, FT, FTS
MIXED_EPS = 3e-8            # truncation that single precision can tell from zero


def _product(name, version, n, phi, precision, where, poly=False):
    return dict(name=name, kind="product", version=version, n=n, phi=phi, precision=precision,
                where=where, poly=poly)


def listed():
    return [
        # the smallest call: one drop-in product of a few dozen spheres, as
        # the time loop of a small Stokesian-dynamics program makes it
        _product("f_n64_fp64_host", 0, 64, 0.10, "fp64", "host"),
        # the drop-in product at its usual size, default precision
        _product("fts_n1000_fp64_host", 2, 1000, 0.30, "fp64", "host"),
        # FP64 products of a GPU-resident program (reference runs, the FP64
        # residuals of refined solves)
        _product("ft_n2048_fp64_dev", 1, 2048, 0.25, "fp64", "dev"),
        # the same drop-in call in mixed precision, small and ragged: latency
        _product("ft_n333_mixed_host", 1, 333, 0.15, "mixed", "host"),
        # the library's headline product: FTS, 1000 spheres, mixed precision
        _product("fts_n1000_mixed_dev", 2, 1000, 0.30, "mixed", "dev"),
        # the product of the 4096-sphere Brownian-dynamics workload
        _product("f_n4096_mixed_dev", 0, 4096, 0.20, "mixed", "dev"),
        # the largest: a production-size stresslet product, ragged
        _product("fts_n12001_mixed_dev", 2, 12001, 0.30, "mixed", "dev"),
        # unequal spheres
        _product("fts_n500_poly_mixed_dev", 2, 500, 0.20, "mixed", "dev", poly=True),
        # the dense mobility matrix, for factorisations and eigenvalues
        dict(name="matrix_fts_n256_fp64_dev", kind="matrix", version=2, n=256, phi=0.30),
        # gradients of g . M f with respect to the positions and the box
        dict(name="vjp_ft_n1000_mixed", kind="vjp", version=1, n=1000, phi=0.15),
        # one Brownian-dynamics mid-point step (33 products, device noise)
        dict(name="bd_f_n1000_mixed", kind="bd", version=0, n=1000, phi=0.20),
        # an ensemble: independent systems of mixed sizes in one product
        dict(name="batch_64_mixed", kind="batch", nsys=64, nmin=16, nmax=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    phi = round(rng.uniform(0.05, 0.35), 3)
    if pick < 0.70:
        version = rng.choice((0, 1, 2))
        precision = rng.choice(("fp64", "mixed"))
        poly = rng.random() < 0.15
        top = 2500 if precision == "fp64" else (2000 if poly else 12000)
        return dict(kind="product", version=version, n=_log_int(rng, 64, top), phi=phi,
                    precision=precision, where=rng.choice(("host", "dev")), poly=poly)
    if pick < 0.78:
        return dict(kind="matrix", version=rng.choice((0, 1, 2)), n=_log_int(rng, 24, 256), phi=phi)
    if pick < 0.86:
        # the mixed gradients need a box of about 21 radii
        return dict(kind="vjp", version=rng.choice((0, 1)), n=_log_int(rng, 900, 2000),
                    phi=round(rng.uniform(0.10, 0.30), 3))
    if pick < 0.93:
        return dict(kind="bd", version=rng.choice((0, 1)), n=_log_int(rng, 250, 4096),
                    phi=round(rng.uniform(0.05, 0.25), 3))
    return dict(kind="batch", nsys=rng.randint(8, 64), nmin=16, nmax=rng.randint(64, 512))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _box(n, phi):
    return (n * (4.0 * math.pi / 3.0) / phi) ** (1.0 / 3.0)


def _suspension(n, phi, rng):
    """n non-overlapping unit spheres in a periodic cube: sites of a
    face-centred cubic lattice drawn at random, each sphere moved from its
    site by as much as keeps every distance above 2."""
    box = _box(n, phi)
    m = 1
    while 4 * m ** 3 < n:
        m += 1
    cell = box / m
    base = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    sites = ((g + base) * cell).reshape(-1, 3)
    sites = sites[rng.permutation(len(sites))[:n]]
    room = max(0.0, 0.5 * (cell / math.sqrt(2.0) - 2.001))
    d = rng.standard_normal((n, 3))
    d *= (room * rng.uniform(0, 1, (n, 1)) ** (1 / 3)) / np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(sites + d + rng.uniform(0, box, 3)), box


def _inputs(case, seed):
    """pos, box, radii (or None), x of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 17])
    n, c = case["n"], NC[case["version"]]
    pos, box = _suspension(n, case["phi"], rng)
    rad = rng.uniform(0.7, 1.0, n) if case.get("poly") else None
    return pos, box, rad, rng.standard_normal(c * n)


def _batch_inputs(case, seed):
    rng = np.random.default_rng([seed, 23])
    sizes = np.random.default_rng(case["nsys"]).integers(case["nmin"], case["nmax"] + 1, case["nsys"])
    out = []
    for s, n in enumerate(sizes.tolist()):
        pos, box = _suspension(n, float(rng.uniform(0.05, 0.35)), rng)
        out.append((s % 2, pos, box, rng.standard_normal(NC[s % 2] * n)))
    return out


class _BD:
    def __init__(self, case, seed):
        pos, box, _, _ = _inputs(case, seed)
        self.sys = L.System(case["version"], pos, (box,) * 3)
        self.sys.set_misc(rmin=1.0)
        p = abi.BDParams(peclet=1.0, dt=1e-3, n_cheb=30, n_lanczos=20, cheb_eps=1e-2,
                         check_every=1, lj_e=1.0, lj_r0=2.0, seed=seed % (1 << 31),
                         precision=L.MIXED)
        self.lib, self.h, self.t, self.n = self.sys.lib, C.c_void_p(), 0.0, case["n"]
        L.check(self.lib.stokes_gpu_bd_create(self.sys.sp, C.byref(p), C.byref(self.h)))
        eig = np.zeros(2)
        L.check(self.lib.stokes_gpu_bd_estimate_bounds(self.h, eig.ctypes.data_as(abi._dp)))

    def __del__(self):
        self.lib.stokes_gpu_bd_destroy(self.h)
        self.sys.close()

    def step(self):
        L.check(self.lib.stokes_gpu_bd_run(self.h, self.t, 1))
        self.t += 1e-3
        x = np.empty(3 * self.n)
        L.check(self.lib.stokes_gpu_bd_get_positions(self.h, x.ctypes.data_as(abi._dp)))
        return x


class _Batch:
    def __init__(self, case, seed):
        inp = _batch_inputs(case, seed)
        self.systems = [L.System(v, pos, (box,) * 3) for v, pos, box, _ in inp]
        self.x = np.concatenate([x for *_, x in inp])
        self.lib, self.h = self.systems[0].lib, C.c_void_p()
        arr = (C.POINTER(abi.StokesStruct) * len(inp))(*[s.sp for s in self.systems])
        L.check(self.lib.stokes_gpu_batch_create(arr, len(inp), L.MIXED, C.byref(self.h)))

    def __del__(self):
        self.lib.stokes_gpu_batch_destroy(self.h)
        for s in self.systems:
            s.close()

    def product(self):
        y = np.empty_like(self.x)
        L.check(self.lib.stokes_gpu_batch_atimes(self.h, self.x.ctypes.data_as(abi._dp),
                                                 y.ctypes.data_as(abi._dp)))
        return y


def prepare(case, seed):
    L.load().stokes_gpu_set_error_mode(1)
    kind = case["kind"]
    if kind == "batch":
        return dict(kind=kind, batch=_Batch(case, seed))
    if kind == "bd":
        return dict(kind=kind, bd=_BD(case, seed))
    pos, box, rad, x = _inputs(case, seed)
    s = L.System(case["version"], pos, (box,) * 3)
    if rad is not None:
        s.set_radius(rad)
    st = dict(kind=kind, sys=s, n=s.n)
    if kind == "vjp":
        s.set_precision(L.MIXED)
        st["f"] = x
        st["g"] = np.random.default_rng([seed, 29]).standard_normal(s.n)
    elif kind == "matrix":
        st["pos"] = torch.from_numpy(pos).cuda()
    else:
        mixed = case["precision"] == "mixed"
        s.set_precision(L.MIXED if mixed else L.FP64)
        st["mixed"], st["host"] = mixed, case["where"] == "host"
        if st["host"]:
            st["x"] = x
        else:
            st["pos"], st["x"] = torch.from_numpy(pos).cuda(), torch.from_numpy(x).cuda()
    return st


def run(st):
    """One call.  Results of the mixed paths carry single precision in double
    buffers (their stated error is 1e-6): the program keeps them as float32."""
    kind = st["kind"]
    if kind == "batch":
        return st["batch"].product().astype(np.float32)
    if kind == "bd":
        return st["bd"].step().astype(np.float32)
    s = st["sys"]
    if kind == "vjp":
        dr, db, val = np.empty(3 * s.np), np.empty(3), C.c_double()
        L.check(s.lib.stokes_gpu_vjp(s.sp, *(a.ctypes.data_as(abi._dp)
                                             for a in (st["g"], st["f"], dr, db)), C.byref(val)))
        return dr.astype(np.float32), db.astype(np.float32)
    if kind == "matrix":
        mat = torch.empty(st["n"], st["n"], dtype=torch.float64, device="cuda")
        L.check(s.lib.stokes_gpu_matrix_dev(s.sp, st["pos"].data_ptr(), mat.data_ptr(), None))
        return mat
    if st["host"]:
        y = s.atimes(st["x"])
        return y.astype(np.float32) if st["mixed"] else y
    y = torch.empty(st["n"], dtype=torch.float64, device="cuda")
    L.check(s.lib.stokes_gpu_atimes_dev(s.sp, st["pos"].data_ptr(), st["x"].data_ptr(),
                                        y.data_ptr(), None))
    return y.float() if st["mixed"] else y


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _ewald_flops(n, version, eps):
    """Operations of an Ewald sum of n particles at the split that balances
    the pair terms within the cutoff against the reciprocal sums (half of k
    space, structure factors and back-projection, with and without the sine)."""
    u = math.sqrt(-math.log(eps))
    best = math.inf
    for q in range(4, 80):
        eta = 0.5 * q                        # xi = eta / L
        pairs = n * n * min(1e9, 4.0 / 3.0 * math.pi * (u / eta) ** 3)
        nk = 0.5 * 4.0 / 3.0 * math.pi * (eta * u / math.pi) ** 3
        best = min(best, pairs * PAIR_FLOPS[version] + nk * n * 8 * NC[version])
    return best


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # sizes uniform in [nmin, nmax], half F and half FT
        n = 0.5 * (case["nmin"] + case["nmax"])
        return {"bytes": case["nsys"] * n * 8 * (3 + 2 * 4.5),
                "flops": case["nsys"] * 0.5 * (_ewald_flops(n, 0, MIXED_EPS)
                                               + _ewald_flops(n, 1, MIXED_EPS))}
    n, v = case["n"], case["version"]
    if kind == "bd":
        return {"bytes": 33 * 8 * n * (3 + 2 * NC[v]), "flops": 33 * _ewald_flops(n, v, MIXED_EPS)}
    if kind == "vjp":
        # value and three derivatives of every term
        return {"bytes": 8 * n * (6 + 2 * NC[v]), "flops": 4 * _ewald_flops(n, v, MIXED_EPS)}
    if kind == "matrix":
        nn = (NC[v] * n) ** 2
        # at least some dozen terms per unordered pair of particles
        return {"bytes": 8 * nn + 24 * n, "flops": n * n / 2 * 24 * PAIR_FLOPS[v]}
    eps = MIXED_EPS if case["precision"] == "mixed" else FP64_EPS
    return {"bytes": 8 * n * (3 + 2 * NC[v]), "flops": _ewald_flops(n, v, eps)}


# ---------------------------------------------------------------------------
# the same in plain torch, FP64: Beenakker's Ewald sum of the Rotne-Prager
# mobility with couple and stresslet, at a split of its own.  libstokes' FTS
# result is the split-invariant sum plus twice its reciprocal U-S / E-F
# coupling at its own split, sqrt(pi) / V^(1/3).
# ---------------------------------------------------------------------------
def _sprime(x):
    """F, T, S' (the full stresslet contraction: xx, yy, xy, xz, yz) of x."""
    F = x[..., 0:3]
    T = x[..., 3:6] if x.shape[-1] > 3 else None
    if x.shape[-1] < 11:
        return F, T, None
    sxx, sxy, sxz, syz, syy = x[..., 6:].unbind(-1)
    row = torch.stack
    S = row([row([2 * sxx + syy, sxy, sxz], -1), row([sxy, 2 * syy + sxx, syz], -1),
             row([sxz, syz, torch.zeros_like(sxx)], -1)], -2)
    return F, T, S


def _assemble(U, W, E):
    if W is None:
        return U
    if E is None:
        return torch.cat([U, W], -1)
    e5 = torch.stack([E[..., 0, 0], E[..., 0, 1], E[..., 0, 2], E[..., 1, 2], E[..., 1, 1]], -1)
    return torch.cat([U, W, e5], -1)


def _apply(e, s, x):
    """Pair tensor of direction e and scalars s applied to source vectors x."""
    F, T, S = _sprime(x)
    c = lambda v: v.unsqueeze(-1)  # noqa: E731
    dot = lambda a, b: (a * b).sum(-1, keepdim=True)  # noqa: E731
    cross = torch.linalg.cross
    U = c(s["ya"]) * F + c(s["xa"] - s["ya"]) * dot(e, F) * e
    if T is None:
        return U
    Te, Fe = cross(T, e.expand_as(T)), cross(F, e.expand_as(F))
    U = U + c(s["yb"]) * Te
    W = c(s["yb"]) * Fe + c(s["yc"]) * T + c(s["xc"] - s["yc"]) * dot(e, T) * e
    if S is None:
        return torch.cat([U, W], -1)
    Se = (S @ e.unsqueeze(-1)).squeeze(-1)
    eSe, tr, eF = dot(e, Se), c(S.diagonal(dim1=-2, dim2=-1).sum(-1)), dot(e, F)
    g1, g2, g3 = -s["xg"] / 3, s["yg"], s["xg"] - 2 * s["yg"]
    m1 = 1.5 * s["xm"] - 2 * s["ym"] + 0.5 * s["zm"]
    m2 = 0.5 * (s["zm"] - s["xm"])
    m3 = s["xm"] / 6 - 0.5 * s["zm"]
    U = U - (c(g1) * tr + c(g3) * eSe) * e - 2 * c(g2) * Se
    W = W + 2 * c(s["yh"]) * cross(e.expand_as(Se), Se)
    d = c(g1) * eF + c(m2) * eSe + c(m3) * tr
    ee = c(g3) * eF + c(m1) * eSe + c(m2) * tr
    V = c(g2) * F + c(s["yh"]) * Te + c(s["ym"] - s["zm"]) * Se
    eye = torch.eye(3, dtype=e.dtype, device=e.device)
    outer = e.unsqueeze(-1) * V.unsqueeze(-2)
    E = (d.unsqueeze(-1) * eye + ee.unsqueeze(-1) * e.unsqueeze(-1) * e.unsqueeze(-2)
         + outer + outer.transpose(-1, -2) + c(c(s["zm"])) * S)
    return _assemble(U, W, E)


def _real_scalars(xi, r, a, b, version):
    """Real-space scalars of target radius a and source radius b: derivatives
    of the screened Oseen kernels k (transverse) and h (longitudinal)."""
    u2, ri = (xi * r) ** 2, 1 / r
    ec = torch.erfc(xi * r)
    ex = xi / math.sqrt(math.pi) * torch.exp(-u2)
    s2 = a * a + b * b
    k0 = 2 * (2 * u2 - 3) * ex + ec * ri
    k1 = -2 * ri * (1 + u2 * (4 * u2 - 10)) * ex - ec * ri ** 2
    h0 = 2 * (1 - 2 * u2) * ex + ec * ri
    k2 = 4 * ri ** 2 * (1 + u2 * (14 + u2 * (4 * u2 - 20))) * ex + 2 * ri ** 3 * ec
    h2 = -4 * ri ** 2 * (3 + u2 * (2 + u2 * (4 * u2 - 16))) * ex - 6 * ri ** 3 * ec
    s = {"ya": 0.75 * a * (k0 + k2 * s2 / 6)}
    s["xa"] = 0.75 * a * (h0 + h2 * s2 / 6) + s["ya"]
    if version == 0:
        return s
    kk = 4 * ri ** 2 * (1 + u2 * (6 + u2 * (4 * u2 - 16))) * ex + 2 * ri ** 3 * ec
    h1 = -2 * ri * (1 + u2 * (6 - 4 * u2)) * ex - ec * ri ** 2
    bend = kk + (2 * h0 * ri - k1 - h1) * ri
    s["yb"] = -0.375 * (h0 * ri - k1) * a ** 2
    s["yc"] = 0.1875 * ((h1 - k1) * ri - kk) * a ** 3
    s["xc"] = 0.1875 * bend * a ** 3 + s["yc"]
    if version == 1:
        return s
    k3 = (-4 * ri ** 3 * (3 + u2 * (2 + u2 * (68 + u2 * (8 * u2 - 56)))) * ex - 6 * ri ** 4 * ec)
    k4 = (16 * ri ** 4 * (3 + u2 * (2 + u2 * (-16 + u2 * (76 + u2 * (4 * u2 - 38))))) * ex
          + 24 * ri ** 5 * ec)
    h3 = 4 * ri ** 3 * (9 + u2 * (6 + u2 * (36 + u2 * (8 * u2 - 48)))) * ex + 18 * ri ** 4 * ec
    wg = a * a / 10 + b * b / 6
    s["xg"] = 2.25 * ri * (h0 + h2 * wg) * a ** 2
    s["yg"] = -0.375 * (k1 + h0 * ri + (k3 + h2 * ri) * wg) * a ** 2
    s["yh"] = -0.1875 * bend * a ** 3
    m5 = -0.375 * ri * (k1 + h0 * ri + (k3 + h2 * ri) * s2 / 10)
    m3 = -0.75 * ri ** 2 * (h0 + h2 * s2 / 10)
    m4 = -0.1875 * (kk + (3 * h1 - k1 - 6 * h0 * ri) * ri
                    + (k4 + (3 * h3 - k3 - 6 * h2 * ri) * ri) * s2 / 10)
    s["zm"] = 2 * m5 * a ** 3
    s["xm"] = 6 * m3 * a ** 3 + 3 * s["zm"]
    s["ym"] = 2 * m4 * a ** 3 + s["zm"]
    return s


def _k_half(box, kmax):
    """Half of the reciprocal vectors with |k| <= kmax, as integer triples."""
    m = [int(kmax * float(b) / (2 * math.pi)) + 1 for b in box.detach().cpu()]
    g = torch.stack(torch.meshgrid(*(torch.arange(-v, v + 1, device=box.device) for v in m),
                                   indexing="ij"), -1).reshape(-1, 3)
    half = (g[:, 0] > 0) | ((g[:, 0] == 0) & ((g[:, 1] > 0) | ((g[:, 1] == 0) & (g[:, 2] > 0))))
    g = g[half]
    k = 2 * math.pi * g.to(box.dtype) / box.detach()
    return g[(k * k).sum(-1) <= kmax * kmax]


def _recip(pos, box, rad, x, xi, only_g, version, u):
    """Sum over reciprocal vectors; only_g: the force-stresslet coupling
    alone with libstokes' sign, else all couplings with the invariant sign."""
    n, c = x.shape
    y = torch.zeros_like(x)
    q = rad * rad
    vol = box.prod()
    grid = _k_half(box, 2 * xi * u)
    step = max(1, int(1.2e8 // n))
    for g in grid.split(step):
        k = 2 * math.pi * g.to(pos.dtype) / box
        kk = (k * k).sum(-1)
        kn, z = kk.sqrt(), kk / (4 * xi * xi)
        e = k / kn.unsqueeze(-1)
        w = 2 * math.pi / vol * (1 + z * (1 + 2 * z)) / kk * torch.exp(-z)
        th = pos @ k.T
        co, si = th.cos(), th.sin()
        X = torch.cat([x, q.unsqueeze(-1) * x], -1)
        Cs, Sn = co.T @ X, si.T @ X
        zero = torch.zeros_like(w)

        def op(wt, a, b):
            """weights on the cosine part of a and the sine part of b"""
            s = dict(xa=zero, xc=zero, xg=zero, xm=zero, zm=zero, ya=zero, yb=zero, yc=zero,
                     yg=zero, yh=zero, ym=zero)
            even = {**s, **{t: wt[t] for t in ("ya", "yc", "yh", "ym") if t in wt}}
            odd = {**s, **{t: wt[t] for t in ("yb", "yg") if t in wt}}
            return _apply(e, even, a) + _apply(e, odd, b)

        sg = 1.0 if only_g else -1.0
        # (power of the target radius, power of its square): weights on x, on q x
        table = {
            (1, 0): ({"ya": 6 * w}, {"ya": -kk * w}), (1, 1): ({"ya": -kk * w}, {}),
            (2, 0): ({"yb": 3 * kn * w, "yg": sg * 3 * kn * w}, {"yg": -sg * 0.5 * kk * kn * w}),
            (2, 1): ({"yg": -sg * 0.3 * kk * kn * w}, {}),
            (3, 0): ({"yc": 1.5 * kk * w, "yh": 1.5 * kk * w, "ym": 3 * kk * w},
                     {"ym": -0.3 * kk * kk * w}),
            (3, 1): ({"ym": -0.3 * kk * kk * w}, {}),
        }
        for (p, pq), (w0, wq) in table.items():
            if only_g:
                w0, wq = ({t: v for t, v in d.items() if t == "yg"} for d in (w0, wq))
            if version < 2:
                w0, wq = ({t: v for t, v in d.items() if t not in ("yg", "yh", "ym")}
                          for d in (w0, wq))
            if version < 1:
                w0, wq = ({t: v for t, v in d.items() if t == "ya"} for d in (w0, wq))
            if not w0 and not wq:
                continue
            P = op(w0, Cs[:, :c], -Sn[:, :c]) if w0 else 0
            Q = op(w0, Sn[:, :c], Cs[:, :c]) if w0 else 0
            if wq:
                P = P + op(wq, Cs[:, c:], -Sn[:, c:])
                Q = Q + op(wq, Sn[:, c:], Cs[:, c:])
            y = y + (rad ** p * q ** pq).unsqueeze(-1) * (co @ P + si @ Q)
    return y


def _split(box, widest):
    length = float(box.detach().prod()) ** (1 / 3)
    return min(widest / length, 0.6)


def _images(box, rc):
    n = [max(0, math.ceil(rc / float(b) - 0.5)) for b in box.detach().cpu()]
    return torch.stack(torch.meshgrid(*(torch.arange(-v, v + 1, device=box.device) for v in n),
                                      indexing="ij"), -1).reshape(-1, 3)


U_CUT = 7.0      # erfc(7) = 4e-23


def _exact_product(pos, box, rad, x, version, widest=16.0, chunk=400000):
    """M x, pos [n, 3], box [3], rad [n], x [n, c]."""
    n, c = x.shape
    xi = _split(box, widest)
    rc = U_CUT / xi
    a3, f = rad ** 3, xi / math.sqrt(math.pi)
    a2x = (xi * rad) ** 2
    one = torch.ones_like(rad)
    s = dict(xa=one - rad * f * (6 - 40 / 3 * a2x), xc=0.75 * one - a3 * f * xi * xi * 10,
             xm=0.9 * one - a3 * f * xi * xi * (12 - 30.24 * a2x))
    z = torch.zeros_like(rad)
    s |= dict(ya=s["xa"], yc=s["xc"], ym=s["xm"], zm=s["xm"], yb=z, xg=z, yg=z, yh=z)
    y = _apply(torch.zeros_like(pos), s, x)
    grad = torch.is_grad_enabled() and pos.requires_grad
    for m in _images(box, rc):
        zero_image = not bool(m.any())
        rows = n if grad else max(1, chunk * 8 // n)
        for i0 in range(0, n, rows):
            d = pos.detach().unsqueeze(0) - pos.detach()[i0:i0 + rows].unsqueeze(1)
            w = torch.round(d / box.detach())          # nearest image, then image m of it
            r2 = ((d + (m - w) * box.detach()) ** 2).sum(-1)
            ok = r2 < rc * rc
            if zero_image:
                ok &= r2 > 0
            ii, jj = ok.nonzero(as_tuple=True)
            size = max(1, len(ii)) if grad else chunk
            for i, j in zip(ii.split(size), jj.split(size)):
                v = pos[j] - pos[i0 + i] + (m - w[i, j]) * box
                r = v.norm(dim=-1)
                t = _real_scalars(xi, r, rad[i0 + i], rad[j], version)
                y = y.index_add(0, i0 + i, _apply(v / r.unsqueeze(-1), t, x[j]))
    y = y + _recip(pos, box, rad, x, xi, False, version, U_CUT)
    if version == 2:
        ref = math.sqrt(math.pi) / float(box.detach().prod()) ** (1 / 3)
        y = y + 2 * _recip(pos, box, rad, x, ref, True, version, U_CUT)
    return y


def _exact_matrix(pos, box, version):
    """Dense matrix, FTS in libstokes' extracted form: entry blocks act on
    (2xx+yy, 2xy, 2xz, 2yz, 2yy+xx) of the stresslet."""
    n, c = len(pos), NC[version]
    xi = _split(box, 10.0)
    rc = U_CUT / xi
    unit = torch.eye(c, dtype=pos.dtype, device=pos.device)
    if version == 2:
        unit = unit.clone()
        t = torch.zeros(5, 5, dtype=pos.dtype)
        t[0, 0] = t[4, 4] = t[1, 1] = t[2, 2] = t[3, 3] = 2.0
        t[0, 4] = t[4, 0] = 1.0
        unit[6:, 6:] = torch.linalg.inv(t).to(pos.device)
    one = torch.ones(1, dtype=pos.dtype, device=pos.device)
    f = xi / math.sqrt(math.pi)
    s = dict(xa=one - f * (6 - 40 / 3 * xi ** 2), xc=0.75 * one - f * xi ** 2 * 10,
             xm=0.9 * one - f * xi ** 2 * (12 - 30.24 * xi ** 2))
    z = torch.zeros_like(one)
    s |= dict(ya=s["xa"], yc=s["xc"], ym=s["xm"], zm=s["xm"], yb=z, xg=z, yg=z, yh=z)
    blocks = torch.zeros(n, n, c, c, dtype=pos.dtype, device=pos.device)
    idx = torch.arange(n, device=pos.device)

    def columns(e, sc):
        """blocks of directions e: one application per unit source vector"""
        return torch.stack([_apply(e, sc, unit[:, b].expand(len(e), c)) for b in range(c)], -1)

    blocks[idx, idx] += columns(torch.zeros(1, 3, dtype=pos.dtype, device=pos.device), s)
    d0 = pos.unsqueeze(0) - pos.unsqueeze(1)
    d0 = d0 - box * torch.round(d0 / box)
    for m in _images(box, rc):
        d = d0 + m * box
        r = d.norm(dim=-1)
        ii, jj = ((r < rc) & (r > 0)).nonzero(as_tuple=True)
        v, rr = d[ii, jj], r[ii, jj]
        blocks[ii, jj] += columns(v / rr.unsqueeze(-1), _real_scalars(xi, rr, one, one, version))

    def recip(split, only_g):
        k = 2 * math.pi * _k_half(box, 2 * split * U_CUT).to(pos.dtype) / box
        kk = (k * k).sum(-1)
        kn, q = kk.sqrt(), kk / (4 * split * split)
        w = 2 * math.pi / box.prod() * (1 + q * (1 + 2 * q)) / kk * torch.exp(-q)
        sg = 1.0 if only_g else -1.0
        o = torch.zeros_like(w)
        base = dict(xa=o, xc=o, xg=o, xm=o, zm=o, ya=o, yb=o, yc=o, yg=o, yh=o, ym=o)
        even = dict(base) if only_g else {**base, "ya": 6 * (1 - kk / 3) * w, "yc": 1.5 * kk * w,
                                          "yh": 1.5 * kk * w, "ym": 3 * (1 - kk / 5) * kk * w}
        odd = {**base, "yg": sg * 3 * (1 - 4 / 15 * kk) * kn * w}
        if not only_g:
            odd["yb"] = 3 * kn * w
        e = k / kn.unsqueeze(-1)
        ev, od = columns(e, even), columns(e, odd)
        th = pos @ k.T
        co, si = th.cos(), th.sin()
        for a in range(c):
            for b in range(c):
                if bool(ev[:, a, b].any()):
                    blocks[:, :, a, b] += ((co * ev[:, a, b]) @ co.T + (si * ev[:, a, b]) @ si.T)
                if bool(od[:, a, b].any()):     # carried by sin k.(r_i - r_j)
                    blocks[:, :, a, b] += ((si * od[:, a, b]) @ co.T - (co * od[:, a, b]) @ si.T)

    recip(xi, False)
    if version == 2:
        recip(math.sqrt(math.pi) / float(box.prod()) ** (1 / 3), True)
        recip(math.sqrt(math.pi) / float(box.prod()) ** (1 / 3), True)
    return blocks.permute(0, 2, 1, 3).reshape(n * c, n * c)


def _dev(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64),
                           device="cuda" if torch.cuda.is_available() else "cpu")


def exact(case, seed):
    kind = case["kind"]
    if kind == "bd":
        return None
    if kind == "batch":
        out = []
        for v, pos, box, x in _batch_inputs(case, seed):
            n = len(pos)
            out.append(_exact_product(_dev(pos), _dev([box] * 3), _dev(np.ones(n)),
                                      _dev(x.reshape(n, -1)), v, 10.0).reshape(-1))
        return torch.cat(out).cpu().numpy()
    pos, box, rad, x = _inputs(case, seed)
    n, v = case["n"], case["version"]
    p, b = _dev(pos), _dev([box] * 3)
    if kind == "matrix":
        return _exact_matrix(p, b, v)
    a = _dev(np.ones(n) if rad is None else rad)
    x = _dev(x.reshape(n, -1))
    if kind == "vjp":
        g = _dev(np.random.default_rng([seed, 29]).standard_normal(x.numel()).reshape(n, -1))
        p.requires_grad_(True)
        b.requires_grad_(True)
        (g * _exact_product(p, b, a, x, v, 12.0)).sum().backward()
        return p.grad.reshape(-1).cpu().numpy(), b.grad.cpu().numpy()
    y = _exact_product(p, b, a, x, v).reshape(-1)
    return y.cpu().numpy() if case["where"] == "host" else y
