"""Performance cases of the inverse-acoustics framework.

Each case is one call that a program of this framework makes: assembling
transfer matrices, solving inverse problems, radiation modes, sparse
inversion and the array-design gradient, on device buffers the program keeps.
``prepare`` builds the inputs from the seed alone, ``run`` makes the call
through ``inverseacoustics_gb300.api`` and returns everything it computes, and
``exact`` restates the same quantity in 64 bits with plain torch or numpy.

Sizes: the five workloads of the repository (64 x 162 ESM array; 642-node IBEM
sphere with 120 microphones and 64 bins; order-15 HELS with 256 microphones;
1280-element plate with 192 microphones; 128-microphone array design) and
ranges around them.  Microphone positions carry a small seeded placement
error, as a mounted array does; wavenumbers a small seeded offset.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from inverseacoustics_gb300 import api

C0, RHO0 = 343.0, 1.21
INV4PI = 1.0 / (4.0 * math.pi)

# methods of ia_config.method
GCV, TSVD, FIXED = 0, 1, 2


# --------------------------------------------------------------------- cases
def listed():
    return [
        # One frequency of a small array, as an interactive measurement session
        # solves it: latency and launches decide.
        {"name": "esm_64mic_f1", "kind": "esm", "nx": 8, "ny": 8, "pitch": 0.03, "z": 0.10, "sources": "sphere",
         "m": 162, "bins": 1, "f0": 1000.0, "f1": 1000.0, "rhs": 1, "method": GCV, "k": 0, "grid": True, "prec": 0},
        # Velocity of a vibrating plate from a near-field array, truncated SVD,
        # a block of bins of the 20-2000 Hz sweep.
        {"name": "esm_plate_tsvd", "kind": "esm", "nx": 16, "ny": 12, "pitch": 0.03125, "z": 0.05, "sources": "plate",
         "m": 1280, "bins": 48, "f0": 300.0, "f1": 2000.0, "rhs": 1, "method": TSVD, "k": 36, "grid": False,
         "prec": 0},
        # The headline call: surface velocity of a sphere from 120 microphones,
        # all 64 bins, mixed precision.
        {"name": "ibem_band_mixed", "kind": "ibem", "nu": 8, "mics": 120, "bins": 64, "f0": 100.0, "f1": 2000.0,
         "rhs": 1, "prec": 1},
        # The same inversion at the default precision, an odd number of bins.
        {"name": "ibem_band_fp64", "kind": "ibem", "nu": 8, "mics": 120, "bins": 23, "f0": 100.0, "f1": 2000.0,
         "rhs": 1, "prec": 0},
        # The transfer matrix of one frequency, what a caller of the
        # reference's ibem() asks for: few bins, one large system.
        {"name": "ibem_transfer_f1", "kind": "transfer", "nu": 8, "mics": 120, "bins": 1, "f0": 800.0, "f1": 800.0,
         "prec": 0},
        # Collocation matrices of a finer mesh (1962 nodes) for a caller's own
        # solver: the largest assembly.
        {"name": "ibem_assembly_fine", "kind": "assembly", "nu": 14, "mics": 150, "bins": 5, "f0": 200.0,
         "f1": 2500.0, "prec": 1},
        # Spherical-harmonic expansion, order 15 on a 16 x 16 array, the part
        # of the band that supports this order.
        {"name": "hels_order15", "kind": "hels", "order": 15, "side": 16, "pitch": 0.025, "z": 0.15, "bins": 64,
         "f0": 2250.0, "f1": 3000.0, "rhs": 1},
        # Radiation resistance matrices of the plate, a sweep of bins.
        {"name": "plate_resistance", "kind": "resistance", "nx": 40, "ny": 32, "bins": 64, "f0": 20.0, "f1": 2000.0,
         "spacing": "linear"},
        # Its leading radiation modes.
        {"name": "plate_modes", "kind": "modes", "nx": 40, "ny": 32, "bins": 16, "f0": 900.0, "f1": 1800.0,
         "nmodes": 24, "prec": 0},
        # Radiation modes of a closed body (an ellipsoid) from its IBEM system.
        {"name": "bem_modes_ellipsoid", "kind": "bem_modes", "nu": 8, "mics": 120, "bins": 8, "f0": 400.0,
         "f1": 2000.0, "nmodes": 8, "complex": False, "prec": 0},
        # Sparse source localisation by ADMM, 14 continuation stages.
        {"name": "admm_l1", "kind": "admm", "mics": 120, "m": 642, "bins": 32, "rhs": 1, "norm": 1, "iters": 40,
         "prec": 1},
        # One gradient step of the array design, 16 source fields.
        {"name": "array_design", "kind": "design", "mics": 128, "nu": 8, "bins": 128, "rhs": 16, "grad": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["esm", "ibem", "transfer", "assembly", "hels", "resistance", "modes", "bem_modes", "admm",
                       "design"])
    f0 = round(rng.uniform(150.0, 700.0), 1)
    f1 = round(rng.uniform(1200.0, 2500.0), 1)
    if kind == "esm":
        nx, ny = rng.randint(4, 15), rng.randint(4, 12)
        l = nx * ny
        method = rng.choice([GCV, GCV, TSVD, FIXED])
        m = _logint(rng, max(l, 90), 1280)
        bins = min(_logint(rng, 1, 128), max(1, int(9.0e7 / (l * l * m)) * 10))
        return {"kind": "esm", "nx": nx, "ny": ny, "pitch": round(rng.uniform(0.02, 0.04), 4),
                "z": round(rng.uniform(0.09, 0.15), 3), "sources": "sphere", "m": m, "bins": bins, "f0": f0, "f1": f1,
                "rhs": rng.choice([1, 1, 1, 2, 5]), "method": method, "k": max(2, l // 4) if method == TSVD else 0,
                "grid": False, "prec": rng.choice([0, 0, 1])}
    if kind == "ibem":
        nu, prec = rng.randint(3, 8), rng.choice([0, 1])
        return {"kind": "ibem", "nu": nu, "mics": rng.randint(16, min(130, 10 * nu * nu)),
                "bins": _logint(rng, 1, 64 if prec else 24), "f0": f0, "f1": f1, "rhs": rng.choice([1, 1, 3]),
                "prec": prec}
    if kind == "transfer":
        nu, prec = rng.randint(3, 9), rng.choice([0, 1])
        return {"kind": "transfer", "nu": nu, "mics": rng.randint(1, 160), "bins": _logint(rng, 1, 32), "f0": f0,
                "f1": f1, "prec": prec}
    if kind == "assembly":
        nu = rng.randint(3, 14)
        m = 10 * nu * nu + 2
        return {"kind": "assembly", "nu": nu, "mics": rng.randint(1, 200),
                "bins": min(_logint(rng, 1, 64), max(1, int(2.0e7 / (m * m)))), "f0": f0, "f1": f1,
                "prec": rng.choice([0, 1])}
    if kind == "hels":
        order = rng.randint(4, 15)
        side = int(math.ceil(math.sqrt((order + 1) ** 2 * rng.uniform(0.8, 1.5))))
        side = min(side, 17)
        return {"kind": "hels", "order": order, "side": side, "pitch": 0.025, "z": 0.15,
                "bins": _logint(rng, 1, 64) if side <= 16 else _logint(rng, 1, 24), "f0": 150.0 * order,
                "f1": 150.0 * order + round(rng.uniform(500.0, 1500.0), 1), "rhs": rng.choice([1, 1, 2])}
    if kind == "resistance":
        nx, ny = rng.randint(6, 46), rng.randint(5, 40)
        n = nx * ny
        return {"kind": "resistance", "nx": nx, "ny": ny, "bins": min(_logint(rng, 1, 128), max(1, int(1.05e8 / (n * n)))),
                "f0": f0, "f1": f1, "spacing": rng.choice(["linear", "linear", "octave"])}
    if kind == "modes":
        nx, ny = rng.randint(16, 40), rng.randint(14, 32)
        return {"kind": "modes", "nx": nx, "ny": ny, "bins": _logint(rng, 1, 24),
                "f0": round(rng.uniform(800.0, 1000.0), 1), "f1": round(rng.uniform(1300.0, 1800.0), 1),
                "nmodes": rng.randint(16, 28), "prec": 0}
    if kind == "bem_modes":
        return {"kind": "bem_modes", "nu": rng.randint(4, 8), "mics": rng.randint(8, 120), "bins": _logint(rng, 1, 8),
                "f0": 500.0, "f1": f1, "nmodes": rng.randint(3, 8), "complex": rng.choice([False, False, True]),
                "prec": 0}
    if kind == "admm":
        l = rng.randint(24, 128)
        return {"kind": "admm", "mics": l, "m": rng.randint(l + 8, 700), "bins": _logint(rng, 1, 32),
                "rhs": rng.choice([1, 1, 2]), "norm": rng.choice([1, 1, 2]), "iters": rng.randint(8, 40),
                "prec": rng.choice([0, 1])}
    return {"kind": "design", "mics": rng.randint(16, 128), "nu": rng.randint(4, 8), "bins": _logint(rng, 2, 128),
            "rhs": rng.randint(1, 16), "grad": rng.choice([True, True, False])}


# -------------------------------------------------------- geometry and fields
_CTX = {}


def _context():
    """The program's one library context, on torch's current stream."""
    dev = torch.cuda.current_device()
    if dev not in _CTX:
        _CTX[dev] = api.Context(dev)
    return _CTX[dev]


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _geodesic(nu, axes=(0.1, 0.1, 0.1)):
    """Geodesic sphere of frequency nu (10 nu^2 + 2 nodes, 20 nu^2 triangles)
    scaled to the given half-axes: nodes (3, m), triangles (3, n) int32 with
    (v0 - v2) x (v1 - v2) pointing outward."""
    t = (1.0 + math.sqrt(5.0)) / 2.0
    V = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                  (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)], dtype=np.float64)
    faces = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
             (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11),
             (6, 2, 10), (8, 6, 7), (9, 8, 1)]
    index, pts, tris = {}, [], []
    for a, b, c in faces:
        ids = {}
        for i in range(nu + 1):
            for j in range(nu + 1 - i):
                p = ((nu - i - j) * V[a] + i * V[b] + j * V[c]) / nu
                key = tuple(np.round(p, 9) + 0.0)
                if key not in index:
                    index[key] = len(pts)
                    pts.append(p / np.linalg.norm(p))
                ids[i, j] = index[key]
        for i in range(nu):
            for j in range(nu - i):
                tris.append((ids[i, j], ids[i + 1, j], ids[i, j + 1]))
                if i + j < nu - 1:
                    tris.append((ids[i + 1, j], ids[i + 1, j + 1], ids[i, j + 1]))
    P, E = np.array(pts).T, np.array(tris).T
    p0, p1, p2 = P[:, E[0]], P[:, E[1]], P[:, E[2]]
    out = np.einsum("di,di->i", np.cross((p0 - p2).T, (p1 - p2).T).T, p0 + p1 + p2)
    E[:2, out < 0] = E[1::-1, out < 0]
    return np.ascontiguousarray(P * np.array(axes)[:, None]), np.ascontiguousarray(E.astype(np.int32))


def _fibonacci(m, radius):
    i = np.arange(m) + 0.5
    z = 1.0 - 2.0 * i / m
    a = i * math.pi * (1.0 + math.sqrt(5.0))
    s = np.sqrt(1.0 - z * z)
    return radius * np.stack([s * np.cos(a), s * np.sin(a), z])


def _plate(nx, ny, lx=0.5, ly=0.4):
    x = (np.arange(nx) + 0.5) * lx / nx - lx / 2
    y = (np.arange(ny) + 0.5) * ly / ny - ly / 2
    X, Y = np.meshgrid(x, y, indexing="ij")
    return np.stack([X.ravel(), Y.ravel(), np.zeros(nx * ny)]), lx * ly / (nx * ny)


def _grid_array(rng, nx, ny, pitch, z):
    X, Y = np.meshgrid((np.arange(nx) - (nx - 1) / 2) * pitch, (np.arange(ny) - (ny - 1) / 2) * pitch, indexing="ij")
    p = np.stack([X.ravel(), Y.ravel(), np.full(nx * ny, z)])
    return p + 5e-4 * rng.uniform(-1.0, 1.0, p.shape)


def _hemisphere(rng, count, radius):
    v = rng.normal(size=(3, count))
    v /= np.linalg.norm(v, axis=0)
    v[2] = np.abs(v[2])
    return radius * v


def _wavenumbers(rng, case):
    if case.get("spacing") == "octave":
        f = case["f0"] * (case["f1"] / case["f0"]) ** (np.arange(case["bins"]) / max(1, case["bins"] - 1))
    else:
        f = np.linspace(case["f0"], case["f1"], case["bins"])
    return 2 * math.pi * f * (1.0 + 0.01 * rng.uniform()) / C0


def _cnormal(rng, shape):
    return (rng.normal(size=shape) + 1j * rng.normal(size=shape)) / math.sqrt(2.0)


def _noisy(rng, p, snr_db):
    level = np.sqrt(np.mean(np.abs(p) ** 2, axis=-1, keepdims=True)) * 10.0 ** (-snr_db / 20.0)
    return p + level * _cnormal(rng, p.shape)


def _monopole(P, S, k):
    r = np.sqrt(((P[:, :, None] - S[:, None, :]) ** 2).sum(0))
    return np.exp(1j * k * r) * INV4PI / r


def _spherical(P):
    az = np.arctan2(P[1], P[0])
    return np.stack([np.where(az < 0, az + 2 * math.pi, az), np.arctan2(np.hypot(P[0], P[1]), P[2]),
                     np.sqrt((P ** 2).sum(0))])


def _sphere_field(P, k, a):
    """Fields at P of a sphere of radius a that pulsates and that oscillates
    along z with unit velocity."""
    r = np.sqrt((P ** 2).sum(0))
    pulse = (a / r) * RHO0 * C0 * (1j * k * a / (1j * k * a - 1.0)) * np.exp(1j * k * (r - a))
    h1 = lambda x: -np.exp(1j * x) * (x + 1j) / (x * x)  # noqa: E731
    dh1 = -1j * np.exp(1j * k * a) / (k * a) - 2.0 * h1(k * a) / (k * a)
    return pulse, 1j * RHO0 * C0 * h1(k * r) / dh1 * P[2] / r


def _inputs(case, seed):
    """Host inputs of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    d = {}
    if kind == "admm":
        d["mics"] = _hemisphere(rng, case["mics"], 0.30)
        d["src"] = _fibonacci(case["m"], 0.20)
        k = 2 * math.pi * np.linspace(300.0, 2000.0, case["bins"]) * (1.0 + 0.01 * rng.uniform()) / C0
        H = np.stack([_monopole(d["mics"], d["src"], kk) for kk in k])
        H *= math.sqrt(case["mics"]) / np.sqrt((np.abs(H) ** 2).sum((1, 2), keepdims=True))
        x = np.zeros((case["bins"], case["m"], case["rhs"]), complex)
        for r in range(case["rhs"]):
            x[:, rng.choice(case["m"], 4, replace=False), r] = _cnormal(rng, (1, 4))
        d["H"] = np.ascontiguousarray(H.transpose(0, 2, 1))
        d["p"] = np.ascontiguousarray((H @ x).transpose(0, 2, 1))
        d["lam"] = np.full((case["bins"], case["rhs"]), 0.01) * rng.uniform(0.8, 1.25, (case["bins"], case["rhs"]))
        return d
    if kind == "design":
        rng2 = rng
        d["mics"] = np.stack([rng2.uniform(-0.2, 0.2, case["mics"]), rng2.uniform(-0.2, 0.2, case["mics"]),
                              np.full(case["mics"], 0.12)])
        d["surface"] = _geodesic(case["nu"])[0]
        m = d["surface"].shape[1]
        d["k"] = 2 * math.pi * np.linspace(200.0, 4000.0, case["bins"]) / C0
        d["loglam"] = math.log(0.05) + 0.2 * rng.normal(size=case["bins"])
        d["retreat"] = np.array([0.04])
        g = torch.Generator(device="cuda").manual_seed(seed)
        F, R = case["bins"], case["rhs"]
        d["q"] = torch.randn((F, R, m), dtype=torch.complex128, device="cuda", generator=g)
        d["noise"] = 0.0016 * torch.randn((F, R, case["mics"]), dtype=torch.complex128, device="cuda", generator=g)
        return d
    k = _wavenumbers(rng, case)
    d["k"] = k
    if kind == "esm":
        d["mics"] = _grid_array(rng, case["nx"], case["ny"], case["pitch"], case["z"])
        if case["sources"] == "plate":
            d["src"], area = _plate(40, case["m"] // 40)
            x, y = d["src"][0] / 0.5 + 0.5, d["src"][1] / 0.4 + 0.5
            shapes = np.stack([np.sin(a * math.pi * x) * np.sin(b * math.pi * y) for a in range(1, 6)
                               for b in range(1, 5)])
            q = np.einsum("frs,sm->frm", _cnormal(rng, (len(k), case["rhs"], 20)), shapes) * area
        else:
            d["src"] = _fibonacci(case["m"], 0.05)
            q = _cnormal(rng, (len(k), case["rhs"], case["m"]))
        d["p"] = _noisy(rng, np.stack([q[f] @ _monopole(d["mics"], d["src"], k[f]).T for f in range(len(k))]), 30.0)
    elif kind in ("ibem", "transfer", "assembly", "bem_modes"):
        axes = (0.1, 0.1, 0.1)
        if kind == "bem_modes":
            axes = tuple(np.array([0.13, 0.10, 0.075]) * (1.0 + 0.02 * rng.uniform(size=3)))
        d["nodes"], d["elems"] = _geodesic(case["nu"], axes)
        d["mics"] = _hemisphere(rng, case["mics"], 0.30)
        if kind == "ibem":
            amp = _cnormal(rng, (len(k), case["rhs"], 2))
            f = [_sphere_field(d["mics"], kk, 0.1) for kk in k]
            d["p"] = _noisy(rng, np.stack([amp[i] @ np.stack(f[i]) for i in range(len(k))]), 30.0)
    elif kind == "hels":
        mics = _grid_array(rng, case["side"], case["side"], case["pitch"], case["z"])
        src = rng.normal(size=(3, 40))
        src *= 0.08 * rng.uniform(size=40) ** (1 / 3) / np.linalg.norm(src, axis=0)
        q = _cnormal(rng, (len(k), case["rhs"], 40))
        d["pts"] = _spherical(mics)
        d["p"] = _noisy(rng, np.stack([q[f] @ _monopole(mics, src, k[f]).T for f in range(len(k))]), 25.0)
    elif kind in ("resistance", "modes"):
        d["x"], d["area"] = _plate(case["nx"], case["ny"])
    return d


def _sinc_matrices(x, k, area):
    """R (F, n, n) of the plate by the defining formula, on the GPU."""
    X, kk = _dev(x).T.contiguous(), _dev(k)
    r = ((X[:, None, :] - X[None, :, :]) ** 2).sum(-1).sqrt()
    pref = C0 * RHO0 * area * area * INV4PI
    out = torch.empty((len(k),) + r.shape, dtype=torch.float64, device=r.device)
    for f in range(len(k)):
        kr = kk[f] * r
        out[f] = pref * kk[f] ** 2 * torch.where(kr == 0, torch.ones_like(kr), torch.sin(kr) / kr)
    return out


def prepare(case, seed):
    d = _inputs(case, seed)
    ctx = _context()
    s = {"case": case, "ctx": ctx}
    kind = case["kind"]
    for name in ("mics", "src", "k", "p", "pts", "x", "H", "lam", "surface", "retreat", "loglam", "q", "noise"):
        if name in d:
            s[name] = d[name] if isinstance(d[name], torch.Tensor) else _dev(d[name])
    if "nodes" in d:
        s["mesh"] = api.Mesh(ctx, d["nodes"], d["elems"])
    if kind == "modes":
        s["R"] = _sinc_matrices(d["x"], d["k"], d["area"])
    if kind == "resistance":
        s["area"] = d["area"]
    if kind == "admm":
        s["cfg"] = api.default_admm_config(norm=case["norm"], max_iters=case["iters"], rho=2.0, epsilon=0.0,
                                           precision=case["prec"])
    elif kind == "esm":
        o = {"method": case["method"], "precision": case["prec"]}
        if case["method"] == TSVD:
            o["tsvd_k"] = case["k"]
        if case["method"] == FIXED:
            o["lambda_fixed"] = 0.2
        if case["grid"]:
            o["gcv_lo"], o["gcv_hi"] = 1e-8, 1e2
        s["cfg"] = api.default_config(**o)
    else:
        s["cfg"] = api.default_config(precision=case.get("prec", 0))
    return s


def run(s):
    kind, ctx = s["case"]["kind"], s["ctx"]
    if kind == "esm":
        return api.esm_solve_batch(ctx, s["mics"], s["src"], s["k"], s["p"], s["cfg"])
    if kind == "ibem":
        return api.ibem_solve_batch(ctx, s["mesh"], s["mics"], s["k"], s["p"], s["cfg"])
    if kind == "transfer":
        return api.ibem_transfer_batch(ctx, s["mesh"], s["mics"], s["k"], s["cfg"])
    if kind == "assembly":
        return api.ibem_assemble_batch(ctx, s["mesh"], s["mics"], s["k"], s["cfg"])
    if kind == "hels":
        return api.hels_solve_batch(ctx, s["pts"], s["case"]["order"], s["k"], s["p"], s["cfg"])
    if kind == "resistance":
        return api.sinc_resistance_batch(ctx, s["x"], s["k"], s["area"], s["cfg"])
    if kind == "modes":
        return api.radiation_modes_batch(ctx, s["R"], s["case"]["nmodes"], s["cfg"])
    if kind == "bem_modes":
        return api.bem_modes_batch(ctx, s["mesh"], s["mics"], s["k"], s["case"]["nmodes"], s["cfg"],
                                   complex_modes=s["case"]["complex"])
    if kind == "admm":
        return api.admm_batch(ctx, s["H"], s["p"], s["lam"], s["cfg"])
    out = api.esm_design_batch(ctx, s["mics"], s["surface"], s["retreat"], s["k"], s["loglam"], s["q"], s["noise"],
                               grad=s["case"]["grad"])
    return [t for t in out if t is not None]


# ----------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once, and the operations of the
    contractions and factorisations (a complex multiply-add is 8)."""
    kind, F = case["kind"], case["bins"]

    def solve(l, m, R):   # a decomposition of an l x m operator and the back-projection
        p, q = min(l, m), max(l, m)
        return 8.0 * F * (2.0 * p * p * q + 8.0 / 3.0 * p ** 3 + R * p * q)

    def evals(rows, n):   # exp(ikr)/r and 6 complex sums per quadrature point
        return 60.0 * 7 * rows * n * F

    if kind == "esm":
        l, m, R = case["nx"] * case["ny"], case["m"], case["rhs"]
        return {"bytes": F * (R * (l + m) * 16.0 + l * 8) + 24.0 * (l + m),
                "flops": solve(l, m, R) + 30.0 * F * l * m}
    if kind == "hels":
        l, m, R = case["side"] ** 2, (case["order"] + 1) ** 2, case["rhs"]
        return {"bytes": F * (R * (l + m) * 16.0 + min(l, m) * 8) + 24.0 * l, "flops": solve(l, m, R) + 30.0 * F * l * m}
    if kind in ("ibem", "transfer", "assembly", "bem_modes"):
        m, n, l = 10 * case["nu"] ** 2 + 2, 20 * case["nu"] ** 2, case["mics"]
        geo = 24.0 * (m + l) + 12.0 * n
        if kind == "assembly":
            return {"bytes": geo + 32.0 * F * (m + l) * m, "flops": evals(m + l, n)}
        lu = 8.0 * F * (m ** 3 / 3.0)
        if kind == "bem_modes":
            nm = case["nmodes"]
            return {"bytes": geo + F * nm * (8.0 * m + 16.0 * m + 16.0 * l),
                    "flops": evals(m + l, n) + lu + 8.0 * F * m ** 3 + 8.0 * F * (m * m * l + 2 * nm * m * m)}
        tr = evals(m + l, n) + lu + 8.0 * F * 2 * m * m * l
        if kind == "transfer":
            return {"bytes": geo + 16.0 * F * l * m, "flops": tr}
        return {"bytes": geo + 16.0 * F * case["rhs"] * (l + m), "flops": tr + solve(l, m, case["rhs"])}
    if kind == "resistance":
        n = case["nx"] * case["ny"]
        return {"bytes": 24.0 * n + 8.0 * F * n * n, "flops": 5.0 * F * n * n}
    if kind == "modes":
        n, nm = case["nx"] * case["ny"], case["nmodes"]
        return {"bytes": 8.0 * F * n * n + 8.0 * F * nm * (n + 1), "flops": 2.0 * F * n * n * (nm + 16) * 11}
    if kind == "admm":
        l, m, R = case["mics"], case["m"], case["rhs"]
        n_it = case["iters"] * (14 if case["norm"] == 1 else 1)
        return {"bytes": 16.0 * F * (l * m + R * (l + m)),
                "flops": 8.0 * F * R * n_it * (2.0 * l * m + l * l) + 8.0 * F * (l * l * m + l ** 3)}
    l, m, R = case["mics"], 10 * case["nu"] ** 2 + 2, case["rhs"]
    return {"bytes": 16.0 * F * R * (l + m) + 8.0 * F * R,
            "flops": 8.0 * F * (l * l * m / 2 + l ** 3 / 3 + R * (5.0 if case["grad"] else 3.0) * l * m)}


# ---------------------------------------------------------------------- exact
def _gcv_lambda(s, beta, dof, delta0, grid):
    """GCV lambda of one right-hand side: 200-point grid, then the zero of the
    slope in log lambda on the bracket around the grid minimum."""
    b2 = np.abs(beta) ** 2
    t = np.arange(200) / 199.0
    if grid:
        lam = np.exp(math.log(1e2) + t * (math.log(1e-8) - math.log(1e2)))
    else:
        low = max(s[-1], s[0] * 16 * np.finfo(float).eps)
        lam = low * ((s[0] / low) ** (1.0 / 199)) ** np.arange(199, -1, -1)

    def terms(la):
        f = la * la / (s * s + la * la)
        return (f * f * b2).sum() + delta0, dof + f.sum(), f

    G = [n / (d * d) for n, d, _ in (terms(la) for la in lam)]
    j = int(np.argmin(G))
    lo, hi = lam[min(j + 1, 199)], lam[max(j - 1, 0)]

    def slope(u):
        n, d, f = terms(math.exp(u))
        return 4.0 * (f * f * (1 - f) * b2).sum() * d - 4.0 * n * (f * (1 - f)).sum()

    a, b = math.log(lo), math.log(hi)
    if lo == hi or slope(a) >= 0:
        return lo
    if slope(b) <= 0:
        return hi
    for _ in range(64):
        c = 0.5 * (a + b)
        a, b = (c, b) if slope(c) < 0 else (a, c)
    return math.exp(0.5 * (a + b))


def _solve_exact(H, p, case, method=GCV):
    """x, lambda, s of H[f] x = p[f, r] (H a list of l x m arrays)."""
    xs, lams, ss = [], [], []
    for f, A in enumerate(H):
        U, s, Vh = np.linalg.svd(A, full_matrices=False)
        dof = max(0, A.shape[0] - s.size)
        x, la = [], []
        for b in p[f]:
            beta = U.conj().T @ b
            d0 = max(0.0, np.vdot(b, b).real - np.vdot(beta, beta).real) if dof else 0.0
            if method == TSVD:
                c, lam = np.where(np.arange(s.size) < case["k"], beta / s, 0.0), 0.0
            else:
                lam = 0.2 if method == FIXED else _gcv_lambda(s, beta, dof, d0, case.get("grid", False))
                c = s * beta / (s * s + lam * lam)
            x.append(Vh.conj().T @ c)
            la.append(lam)
        xs.append(x)
        lams.append(la)
        ss.append(s)
    return [np.array(xs), np.array(lams), np.array(ss), None]


def _rules():
    """7-point degree-5 rule, and the 4 x 4 Duffy rule for each vertex."""
    s15 = math.sqrt(15.0)
    a1, b1, w1 = (6 - s15) / 21, (9 + 2 * s15) / 21, (155 - s15) / 2400
    a2, b2, w2 = (6 + s15) / 21, (9 - 2 * s15) / 21, (155 + s15) / 2400
    reg = np.array([(1 / 3, 1 / 3, 9 / 80), (a1, a1, w1), (b1, a1, w1), (a1, b1, w1), (a2, a2, w2), (b2, a2, w2),
                    (a2, b2, w2)])
    g, w = np.polynomial.legendre.leggauss(4)
    g, w = 0.5 * (g + 1.0), 0.5 * w
    sing = []
    for v in range(3):
        rows = []
        for a in range(4):
            for b in range(4):
                n = [0.0, 0.0, 0.0]
                n[v], n[(v + 1) % 3], n[(v + 2) % 3] = 1 - g[a], g[a] * (1 - g[b]), g[a] * g[b]
                rows.append((n[0], n[1], w[a] * w[b] * g[a]))
        sing.append(rows)
    return reg, np.array(sing)


def _collocation(d, k):
    """A, B, A_hs, B_hs of the collocation scheme at one wavenumber."""
    dev = torch.device("cuda")
    P, E = _dev(d["nodes"]), _dev(d["elems"]).long()
    M = _dev(d["mics"])
    m, n = P.shape[1], E.shape[1]
    reg, sing = _rules()
    v = P[:, E]                                                       # (3 coordinates, 3 vertices, n)
    nrm = torch.linalg.cross((v[:, 0] - v[:, 2]).T, (v[:, 1] - v[:, 2]).T).T
    an = nrm.norm(dim=0)

    def terms(x, q, w):
        # x (3, rows or n, 1 or n): contributions of the point q of every element
        N = [q[0], q[1], 1.0 - q[0] - q[1]]
        y = N[0] * v[:, 0] + N[1] * v[:, 1] + N[2] * v[:, 2]
        D = y[:, None, :] - x if x.dim() == 3 else y - x
        r = (D * D).sum(0).sqrt()
        ft = ((nrm[:, None, :] if x.dim() == 3 else nrm) * D).sum(0) / (r * r)
        g = torch.polar(1.0 / r, k * r)
        ga = w * INV4PI * ft * torch.complex(-torch.ones_like(r), k * r) * g
        gb = w * INV4PI * an * g
        return N, ga, gb, -w * INV4PI * ft / r

    def rows(x):
        A = torch.zeros((x.shape[1], m), dtype=torch.complex128, device=dev)
        B = torch.zeros_like(A)
        Cc = torch.zeros((x.shape[1],), dtype=torch.float64, device=dev)
        own = [E[s][None, :] == torch.arange(m, device=dev)[:, None] for s in range(3)] if x is P else None
        mask = (own[0] | own[1] | own[2]) if own else None
        for q in reg:
            N, ga, gb, ct = terms(x[:, :, None], q, q[2])
            if mask is not None:
                ga, gb, ct = (torch.where(mask, torch.zeros_like(t), t) for t in (ga, gb, ct))
            for s in range(3):
                A.index_add_(1, E[s], N[s] * ga)
                B.index_add_(1, E[s], N[s] * gb)
            Cc += ct.sum(1)
        return A, B, Cc

    A, B, Cc = rows(P)
    for s in range(3):                                                # vertex s of the element is the row
        for q in sing[s]:
            N, ga, gb, ct = terms(P[:, E[s]], q, q[2])
            for u in range(3):
                A.index_put_((E[s], E[u]), N[u] * ga, accumulate=True)
                B.index_put_((E[s], E[u]), N[u] * gb, accumulate=True)
            Cc.index_put_((E[s],), ct, accumulate=True)
    A.diagonal().sub_(1.0 + Cc)
    Ah, Bh, _ = rows(M)
    sc = 1j * RHO0 * C0 * k
    return A, B * sc, Ah, Bh * sc


def _harmonics(order, az, el):
    """Y_n^m columns n^2 + n + m at (az, el)."""
    x, s = np.cos(el), np.abs(np.sin(el))
    P = {}
    for m in range(order + 1):
        P[m, m] = (P[m - 1, m - 1] * -(2 * m - 1) * s) if m else np.ones_like(x)
        if m < order:
            P[m + 1, m] = (2 * m + 1) * x * P[m, m]
        for n in range(m + 2, order + 1):
            P[n, m] = ((2 * n - 1) * x * P[n - 1, m] - (n + m - 1) * P[n - 2, m]) / (n - m)
    cols = []
    for n in range(order + 1):
        for m in range(-n, n + 1):
            a = abs(m)
            c = math.sqrt((2 * n + 1) / (4 * math.pi) * math.factorial(n - a) / math.factorial(n + a))
            y = c * P[n, a] * np.exp(1j * a * az)
            cols.append((-1) ** a * y.conj() if m < 0 else y)
    return np.stack(cols, 1)


def _hankel(order, x):
    """h_n(x) = j_n + i y_n, n = 0..order: j_n by downward recurrence from a
    start far above, y_n upward."""
    top = int(order + 30 + x.max())
    j = np.zeros((top + 2, x.size))
    j[top] = 1e-280
    for n in range(top, 0, -1):
        j[n - 1] = (2 * n + 1) / x * j[n] - j[n + 1]
        big = np.abs(j[n - 1]) > 1e200
        j[:, big] *= 1e-200
    j = j[:order + 1] * np.where(np.abs(np.sin(x)) > 0.3, np.sin(x) / x / j[0],
                                 (np.sin(x) / x ** 2 - np.cos(x) / x) / j[1])
    y = np.zeros((order + 1, x.size))
    y[0] = -np.cos(x) / x
    if order:
        y[1] = -np.cos(x) / x ** 2 - np.sin(x) / x
    for n in range(1, order):
        y[n + 1] = (2 * n + 1) / x * y[n] - y[n - 1]
    return j + 1j * y


def _sign(U):
    """Columns with the first component within 1e-6 of the largest magnitude
    real and positive."""
    a = U.abs()
    i = (a >= a.amax(0, keepdim=True) * (1 - 1e-6)).to(torch.int8).argmax(0)
    ph = U[i, torch.arange(U.shape[1], device=U.device)]
    return U * (ph.conj() / ph.abs())


def exact(case, seed):
    kind, F = case["kind"], case["bins"]
    if kind == "esm":
        if F * (case["nx"] * case["ny"]) ** 2 * case["m"] > 3e9:
            return None
        d = _inputs(case, seed)
        return _solve_exact([_monopole(d["mics"], d["src"], k) for k in d["k"]], d["p"], case, case["method"])
    if kind == "hels":
        d = _inputs(case, seed)
        az, el, r = d["pts"]
        Y = _harmonics(case["order"], az, el)
        n = np.array([int(math.isqrt(i)) for i in range((case["order"] + 1) ** 2)])
        return _solve_exact([_hankel(case["order"], k * r)[n].T * Y for k in d["k"]], d["p"], case)
    if kind in ("ibem", "transfer", "assembly", "bem_modes"):
        d = _inputs(case, seed)
        if kind == "bem_modes":
            reg, _ = _rules()
            P, E = _dev(d["nodes"]), _dev(d["elems"]).long()
            N = _dev(np.stack([reg[:, 0], reg[:, 1], 1 - reg[:, 0] - reg[:, 1]]))
            Me = (N * _dev(reg[:, 2])) @ N.T
            v = P[:, E]
            an = torch.linalg.cross((v[:, 0] - v[:, 2]).T, (v[:, 1] - v[:, 2]).T).norm(dim=1)
            G = torch.zeros((P.shape[1],) * 2, dtype=torch.float64, device=P.device)
            for a in range(3):
                for b in range(3):
                    G.index_put_((E[a], E[b]), an * Me[a, b], accumulate=True)
        outs = []
        for k in d["k"]:
            A, B, Ah, Bh = _collocation(d, float(k))
            if kind == "assembly":
                outs.append((A, B, Ah, Bh))
            elif kind == "bem_modes":
                Z = torch.linalg.solve(A, B)
                GZ = G.to(torch.complex128) @ Z
                U, s, _ = torch.linalg.svd(GZ.cpu() if case["complex"] else GZ.real.cpu())
                U = _sign(U[:, :case["nmodes"]]).to(A.device)
                Uc = U.to(torch.complex128)
                outs.append((s[:case["nmodes"]], U.T, ((Ah @ Z - Bh) @ Uc).T, (Z @ Uc).T))
            else:
                outs.append(torch.linalg.solve(A.T, Ah.T).T @ B - Bh)
        if kind == "ibem":
            return _solve_exact([h.cpu().numpy() for h in outs], d["p"], case)
        if kind == "transfer":
            return [torch.stack([h.T for h in outs]), None]
        if kind == "assembly":
            return [torch.stack(t) for t in zip(*outs)]
        return [torch.stack([t.to("cuda") for t in o]) for o in zip(*outs)] + [None]
    if kind == "resistance":
        d = _inputs(case, seed)
        return _sinc_matrices(d["x"], d["k"], d["area"])
    if kind == "modes":
        d = _inputs(case, seed)
        lam, vec = [], []
        for R in _sinc_matrices(d["x"], d["k"], d["area"]):
            w, V = torch.linalg.eigh(R)
            lam.append(w.flip(0)[:case["nmodes"]])
            vec.append(_sign(V.flip(1)[:, :case["nmodes"]]).T)
        return [torch.stack(lam), torch.stack(vec), None]
    if kind == "admm":
        return _admm_exact(case, _inputs(case, seed))
    return _design_exact(case, _inputs(case, seed))


def _admm_exact(case, d):
    """The scaled iteration with (2 A^H A + rho I) c = 2 A^H b + rho x - u per
    update: L1 with 14 stages of a shrinking threshold, or L2."""
    A = _dev(d["H"]).transpose(1, 2)
    b, lam0 = _dev(d["p"]).transpose(1, 2), _dev(d["lam"])[:, None, :]
    rho, m = 2.0, A.shape[2]
    AH = A.mH
    Q, T = torch.linalg.qr(AH)
    x = Q @ torch.linalg.solve(T.mH, b)
    K = 2.0 * (AH @ A) + rho * torch.eye(m, dtype=A.dtype, device=A.device)
    Ki = torch.linalg.inv(K)
    rhs = 2.0 * (AH @ b)
    u = torch.zeros_like(x)
    c, its = torch.zeros_like(x), 0
    stages = 1 if case["norm"] == 2 else 14
    lam = 5.0 * lam0
    for _ in range(stages):
        for _ in range(case["iters"]):
            c = Ki @ (rhs + rho * x - u)
            its += 1
            if case["norm"] == 2:
                x = (rho * c + u) / (2.0 * lam0 + rho)
            else:
                y = c + u / rho
                a = y.abs()
                x = torch.where(a > 0, y / a.clamp_min(1e-300), torch.zeros_like(y)) * (a - lam / rho).clamp_min(0.0)
            u = u + rho * (c - x)
        lam = torch.maximum(0.75 * lam, lam0 / 10.0)
    return [c.transpose(1, 2).contiguous(), None, None]


def _design_exact(case, d):
    """Loss terms, and gradients of their mean by automatic differentiation."""
    mics, surf = _dev(d["mics"]).requires_grad_(), _dev(d["surface"])
    retreat, ll = _dev(d["retreat"]).requires_grad_(), _dev(d["loglam"]).requires_grad_()
    F, R = case["bins"], case["rhs"]
    errs = []
    gm, gd, gl = 0.0, 0.0, 0.0
    for f in range(F):
        src = surf * (1.0 - retreat / surf.norm(dim=0))
        r = ((mics[:, :, None] - src[:, None, :]) ** 2).sum(0).sqrt()
        G = torch.polar(INV4PI / r, float(d["k"][f]) * r)
        q = d["q"][f].T
        p = G @ q + d["noise"][f].T
        K = G @ G.mH + torch.exp(2.0 * ll[f]) * torch.eye(r.shape[0], dtype=G.dtype, device=G.device)
        e = G.mH @ torch.linalg.solve(K, p) - q
        err = (e.abs() ** 2).sum(0).sqrt() / (q.abs() ** 2).sum(0).sqrt()
        errs.append(err.detach())
        if case["grad"]:
            a, b, c = torch.autograd.grad(err.sum() / (F * R), (mics, retreat, ll))
            gm, gd, gl = gm + a, gd + b, gl + c
    out = [torch.stack(errs)]
    return out + ([gm, gd, gl] if case["grad"] else []) + [None]
