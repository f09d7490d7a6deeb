"""The work a program hands to this library, as cases that can be timed and
compared: frequency solves and sweeps, H-matrix products, preconditioner
applications, field evaluations and a training step of the quadrature-order
selector, each through the public entry points.

A case is a dict; ``listed()`` gives the fixed ones, ``draw(rng)`` more of the
same ranges. ``prepare`` makes what a program holds before the call, ``run`` is
one call, ``work`` the bytes and operations it cannot do without and ``exact``
the same result in 64 bits from plain torch.

Mixed-precision results (complex FP32 operators, FP32 sums) carry single
precision, so the programs here keep them as complex64, as one that stores
pressure fields does; results of the complex-FP64 method stay complex128.
"""
import ctypes
import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("3d_bem_gb300")
meshes = importlib.import_module("3d_bem_gb300.meshes")

C0, RHO = 343.0, 1.2


def listed():
    return [
        # the small pulsating sphere: complex FP64 throughout, H-LU
        # preconditioned; launch- and latency-bound, the interactive size
        {"name": "solve_sphere_1280_fp64_hlu", "kind": "solve", "body": "sphere", "n": 1280,
         "extra": 0, "mixed": False, "hlu": True, "rhs": 1, "freq": 200.0, "aca": 1e-4,
         "gmres": 1e-8},
        # the plain complex-FP64 method at a middle size, no preconditioner
        {"name": "solve_sphere_5120_fp64", "kind": "solve", "body": "sphere", "n": 5120,
         "extra": 0, "mixed": False, "hlu": False, "rhs": 1, "freq": 800.0, "aca": 1e-5,
         "gmres": 1e-10},
        # the large sphere in mixed precision with the learned ACA rule table:
        # assembly (ACA) and unpreconditioned GMRES
        {"name": "solve_sphere_20480_mixed", "kind": "solve", "body": "sphere", "n": 20480,
         "extra": 0, "mixed": True, "hlu": False, "rhs": 1, "freq": 1500.0, "aca": 1e-5,
         "gmres": 1e-10},
        # the batched sweep of the driven box: piston and random patches,
        # concurrent workers, long GMRES runs on a small system of odd size
        {"name": "sweep_box_5123_mixed", "kind": "sweep", "body": "box", "n": 5120, "extra": 3,
         "mixed": True, "rhs": 4, "nf": 8, "freq": 50.0, "freq_to": 2000.0, "workers": 4,
         "aca": 1e-5, "gmres": 1e-10},
        # the largest body: impedance walls, eight right-hand sides, GPU H-LU
        {"name": "solve_pencil_81920_mixed_hlu", "kind": "solve", "body": "pencil", "n": 81920,
         "extra": 0, "mixed": True, "hlu": True, "rhs": 8, "freq": 1500.0, "aca": 1e-5,
         "gmres": 1e-10},
        # the smallest call: one H-matrix product of a program's own iteration
        # (complex FP64, odd size)
        {"name": "product_sphere_1283_fp64", "kind": "product", "body": "sphere", "n": 1280,
         "extra": 3, "mixed": False, "rhs": 1, "which": 1, "freq": 200.0, "aca": 1e-4},
        # the product inside the mixed-precision GMRES at the large sphere
        {"name": "product_sphere_20480_fp32", "kind": "product", "body": "sphere", "n": 20480,
         "extra": 0, "mixed": True, "rhs": 1, "which": 1, "freq": 1500.0, "aca": 1e-5},
        # the same with a block of right-hand sides on the slender body
        {"name": "product_pencil_20480_fp32_rhs8", "kind": "product", "body": "pencil",
         "n": 20480, "extra": 0, "mixed": True, "rhs": 8, "which": 1, "freq": 1500.0,
         "aca": 1e-5},
        # forward and backward block-triangular substitution (host buffers)
        {"name": "hlu_solve_pencil_20480_rhs8", "kind": "hlu_solve", "body": "pencil",
         "n": 20480, "extra": 0, "mixed": True, "rhs": 8, "freq": 1500.0, "aca": 1e-5},
        # field map of a boundary solution: as many points as elements
        {"name": "field_sphere_20480_pts_20480_mixed", "kind": "field", "body": "sphere",
         "n": 20480, "extra": 0, "mixed": True, "rhs": 1, "pts": 20480, "sources": 0,
         "freq": 1500.0},
        # a few hundred observation points in FP64, three columns and two
        # point sources, ragged sizes
        {"name": "field_box_5123_pts_997_fp64", "kind": "field", "body": "box", "n": 5120,
         "extra": 3, "mixed": False, "rhs": 3, "pts": 997, "sources": 2, "freq": 700.0},
        # one training step of the quadrature-order selector: forward,
        # backward and the Adam update of a minibatch
        {"name": "train_selector_4096", "kind": "train", "batch": 4096},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "sweep", "product", "product", "hlu_solve",
                       "field", "train"])
    if kind == "train":
        return {"kind": kind, "batch": int(_log(rng, 512, 16384))}
    mixed = rng.random() < 0.65
    extra = rng.randrange(0, 8)
    body = rng.choice(["sphere", "box", "pencil"])
    big = 20480 if mixed else 5120
    n = 1280 * 4 ** rng.randrange(0, 3 if mixed else 2) if body == "sphere" \
        else 2 * int(_log(rng, 640, big / 2))
    freq = {"sphere": _log(rng, 150, 1500), "box": _log(rng, 50, 2000),
            "pencil": _log(rng, 200, 8000)}[body]
    case = {"kind": kind, "body": body, "n": n, "extra": extra, "mixed": mixed,
            "rhs": rng.choice([1, 1, 2, 3, 4, 5, 8]), "freq": round(freq, 2), "aca": 1e-5}
    if kind == "solve":
        # the slender body needs the preconditioner to converge
        case.update(hlu=body == "pencil" or rng.random() < 0.3, gmres=1e-10)
    elif kind == "sweep":
        n = 2 * int(_log(rng, 640, 2560))
        case.update(body="box", n=n, mixed=True, rhs=rng.choice([1, 2, 4]), nf=rng.choice([4, 6, 8]),
                    freq=50.0, freq_to=2000.0, workers=rng.choice([2, 3, 4]), gmres=1e-10)
    elif kind == "product":
        case.update(which=rng.choice([0, 1]))
    elif kind == "hlu_solve":
        pass
    else:
        case.update(pts=int(_log(rng, 64, 20480 if mixed else 2048)), sources=rng.choice([0, 0, 2]),
                    rhs=rng.choice([1, 2, 3, 4]))
    return case


# ---------------------------------------------------------------- bodies

@functools.lru_cache(maxsize=4)
def _mesh(body, n, extra):
    """Triangles of a body; `extra` of them are split at their longest edge,
    which gives the counts no structured mesh has."""
    if body == "sphere":
        tri = meshes.icosphere(int(round(math.log(n / 20, 4))), 1.0)
    elif body == "box":
        tri = meshes.box(n_target=n, exact=True)
    else:
        tri = meshes.pencil(n_target=n)
    rng = np.random.default_rng(n)
    for i in sorted(rng.choice(len(tri), extra, replace=False).tolist()):
        v = tri[i].reshape(3, 3).copy()
        e = max(range(3), key=lambda q: float(((v[q] - v[(q + 1) % 3]) ** 2).sum()))
        a, b, c = v[e], v[(e + 1) % 3], v[(e + 2) % 3]
        m = 0.5 * (a + b)
        tri[i] = np.concatenate([a, m, c])
        tri = np.vstack([tri, np.concatenate([m, b, c])[None]])
    tri.setflags(write=False)
    return tri


def _beta(case, n):
    """Wall admittance of the body: resistive walls on the pencil, rigid ones else."""
    return meshes.wall_admittance(n) if case["body"] == "pencil" else None


def _solver(case, **more):
    tri = _mesh(case["body"], case["n"], case["extra"])
    cfg = dict(wave_speed=C0, density=RHO, precision=int(case["mixed"]), aca_tol=case.get("aca", 1e-5),
               sweep_workers=1)
    cfg.update(more)
    s = pkg.Solver(**cfg)
    s.set_mesh(tri)
    beta = _beta(case, len(tri))
    if beta is None:
        s.set_bc(np.zeros(len(tri)), np.ones(len(tri)))
    else:
        s.set_bc_impedance(beta)
    return s, tri


_KEPT = {}


def _kept_solver(case):
    """The handle a program keeps for a body while it solves one set of
    boundary data after another; one body at a time."""
    key = tuple(sorted((k, v) for k, v in case.items()
                       if k not in ("name", "freq", "freq_to", "nf", "rhs")))
    if key not in _KEPT:
        for s, _ in _KEPT.values():
            s.close()
        _KEPT.clear()
        hlu = bool(case.get("hlu"))
        _KEPT[key] = _solver(case, gmres_tol=case["gmres"], gmres_maxit=1000,
                             selector=2 if case["mixed"] else 0, use_preconditioner=int(hlu),
                             precond_rank=2, sweep_workers=case.get("workers", 1))
    return _KEPT[key]


def _drive(case, tri, rng):
    """Driving data: on the sphere a breathing mode plus a smooth pattern, else
    a piston or ring and random patches, with amplitudes of the seed."""
    n, R = len(tri), case["rhs"]
    seed = int(rng.integers(1 << 30))
    if case["body"] == "sphere":
        c = (tri[:, 0:3] + tri[:, 3:6] + tri[:, 6:9]) / 3.0
        d = rng.standard_normal((3, R))
        g = 1.0 + 0.5 * (c @ d) + 0.1 * rng.standard_normal((n, R))
        return np.asfortranarray(g.astype(np.complex128))
    make = meshes.box_piston_rhs if case["body"] == "box" else meshes.pencil_rhs
    g = make(tri, patches=R - 1, seed=seed)
    return np.asfortranarray(g * np.exp(2j * np.pi * rng.random(R)) * rng.uniform(0.5, 2.0, R))


def _waves(rng, shape):
    a = rng.standard_normal(shape + (2,))
    return np.ascontiguousarray(a).view(np.complex128)[..., 0]


# ---------------------------------------------------------------- prepare / run

def _ext_stream(s):
    return torch.cuda.ExternalStream(pkg.lib().bem_stream(s._h))


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(st, what):
    if st != pkg.BEM_OK:
        raise RuntimeError("%s: status %d" % (what, st))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "train":
        x = _train_inputs(case, rng)
        st = {"case": case, "step": 0, "work": torch.zeros(case["batch"] * 265, device="cuda"),
              "loss": torch.zeros(1, device="cuda")}
        for k, v in x.items():
            st[k] = torch.from_numpy(v).cuda()
        for k in ("grad", "m", "v"):
            st[k] = torch.zeros_like(st["params"])
        return st
    jitter = 1.0 + 0.02 * rng.random()
    st = {"case": case}
    if kind in ("solve", "sweep"):
        st["solver"], tri = _kept_solver(case)
        st["g"] = _drive(case, tri, rng)
        if kind == "solve":
            st["freq"] = case["freq"] * jitter
        else:
            st["freqs"] = meshes.log_frequencies(case["nf"], case["freq"], case["freq_to"]) * jitter
        return st
    s, tri = st["solver"], _ = _solver(case)
    n, R = len(tri), case["rhs"]
    st["freq"] = case["freq"] * jitter
    if kind == "product":
        s.assemble(st["freq"])
        st["x"] = torch.from_numpy(_waves(rng, (R, n))).cuda()
        st["y"] = torch.zeros_like(st["x"])
        if case["mixed"]:
            st["y32"] = torch.zeros((R, n), dtype=torch.complex64, device="cuda")
        st["stream"] = _ext_stream(s)
    elif kind == "hlu_solve":
        s.assemble(st["freq"])
        s.hlu_build()
        st["b"] = np.asfortranarray(_waves(rng, (n, R)))
    else:
        pts, phi, dphi, src = _field_inputs(case, tri, st["freq"], rng)
        st["sources"] = src
        if case["pts"] < 2000:  # a handful of microphones: host arrays in and out
            st.update(pts=pts, phi=phi, dphi=dphi)
        else:
            for k, v in (("pts", pts), ("phi", phi.T), ("dphi", dphi.T)):
                st[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
            for k in ("pf", "pp"):
                st[k] = torch.zeros((R, case["pts"]), dtype=torch.complex128, device="cuda")
                st[k + "32"] = torch.zeros((R, case["pts"]), dtype=torch.complex64, device="cuda")
            st["stream"] = _ext_stream(s)
    torch.cuda.synchronize()
    return st


def _kept(case, *arrays):
    """Results as the program keeps them (see the module's docstring)."""
    return [a.astype(np.complex64) if case["mixed"] else a for a in arrays]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        return _kept(case, *st["solver"].solve(st["freq"], st["g"])[:3])
    if kind == "sweep":
        return _kept(case, st["solver"].sweep(st["freqs"], st["g"])[0])
    if kind == "product":
        s = st["solver"]
        arith = pkg.BEM_ARITH_FP32 if case["mixed"] else pkg.BEM_ARITH_FP64
        _ok(pkg.lib().bem_hmatvec_device_ex(s._h, case["which"], _ptr(st["x"]), _ptr(st["y"]),
                                            case["rhs"], 0, arith), "bem_hmatvec_device_ex")
        if not case["mixed"]:
            return st["y"]
        with torch.cuda.stream(st["stream"]):
            return st["y32"].copy_(st["y"])
    if kind == "hlu_solve":
        return _kept(case, st["solver"].hlu_solve(st["b"]))
    if kind == "field":
        s = st["solver"]
        if "stream" not in st:
            return _kept(case, *s.field(st["freq"], st["pts"], st["phi"], st["dphi"], st["sources"]))
        s.field_device(st["freq"], st["pts"].data_ptr(), case["pts"], st["phi"].data_ptr(),
                       st["dphi"].data_ptr(), case["rhs"], st["pf"].data_ptr(),
                       st["pp"].data_ptr(), st["sources"])
        if not case["mixed"]:
            return [st["pf"], st["pp"]]
        with torch.cuda.stream(st["stream"]):
            return [st["pf32"].copy_(st["pf"]), st["pp32"].copy_(st["pp"])]
    L, stream = pkg.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    st["step"] += 1
    _ok(L.bem_mlp_grad(_ptr(st["params"]), _ptr(st["X"]), _ptr(st["y"]), case["batch"],
                       _ptr(st["grad"]), _ptr(st["loss"]), _ptr(st["work"]), stream),
        "bem_mlp_grad")
    _ok(L.bem_mlp_adam(_ptr(st["params"]), _ptr(st["grad"]), _ptr(st["m"]), _ptr(st["v"]),
                       st["step"], 3e-3, 0.9, 0.999, 1e-8, stream), "bem_mlp_adam")
    return [st["grad"], st["loss"], st["params"]]


# ---------------------------------------------------------------- inputs

_NF, _H, _NC = 24, 64, 5


def _train_inputs(case, rng):
    """A minibatch of normalised features with their labels (classes as uneven
    as the trained selector's) and He-initialised weights."""
    B = case["batch"]
    y = rng.choice(_NC, B, p=[0.02, 0.05, 0.13, 0.3, 0.5]).astype(np.uint8)
    centres = 0.8 * rng.standard_normal((_NC, _NF))
    X = (rng.standard_normal((B, _NF)) + centres[y]).astype(np.float32)
    layers = []
    for i, o in ((_NF, _H), (_H, _H), (_H, _NC)):
        layers += [rng.standard_normal(i * o) * math.sqrt(2.0 / i), 0.05 * rng.standard_normal(o)]
    return {"X": X, "y": y, "params": np.concatenate(layers).astype(np.float32)}


def _field_inputs(case, tri, freq, rng):
    """Observation points around the body and the boundary data of a few
    monopoles inside it."""
    k = 2 * np.pi * freq / C0
    c = (tri[:, 0:3] + tri[:, 3:6] + tri[:, 6:9]) / 3.0
    nrm = np.cross(tri[:, 3:6] - tri[:, 0:3], tri[:, 6:9] - tri[:, 0:3])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    lo, hi = c.min(0), c.max(0)
    mid, size = 0.5 * (lo + hi), float(np.linalg.norm(hi - lo))
    d = rng.standard_normal((case["pts"], 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    pts = mid + d * size * rng.uniform(0.6, 3.0, (case["pts"], 1))
    phi = np.zeros((len(tri), case["rhs"]), np.complex128, order="F")
    dphi = np.zeros_like(phi)
    for r in range(case["rhs"]):
        for _ in range(3):
            v = c - (mid + 0.2 * (hi - lo) * rng.uniform(-1.0, 1.0, 3))
            dist = np.linalg.norm(v, axis=1)
            w = (rng.standard_normal() + 1j * rng.standard_normal()) \
                * np.exp(1j * k * dist) / (4 * np.pi * dist)
            phi[:, r] += w
            dphi[:, r] += w * (1j * k - 1.0 / dist) * (v * nrm).sum(1) / dist
    src = None
    if case["sources"]:
        q = rng.standard_normal((case["sources"], 3))
        q = mid + 4.0 * size * q / np.linalg.norm(q, axis=1, keepdims=True)
        src = np.column_stack([q.astype(np.complex128), _waves(rng, (case["sources"],))])
    return pts, phi, dphi, src


# ---------------------------------------------------------------- work

# Stored entries per element of the assembled system matrix (near field plus
# (m + n + 1) k of the low-rank blocks) at 5,120 elements and their growth per
# factor 4 in size, measured at ACA 1e-5 on the three bodies.
_STORED = {"sphere": (2330.0, 1500.0), "box": (1900.0, 900.0), "pencil": (1370.0, 950.0)}
_POINT_FLOPS = 70.0  # one quadrature point of one entry, all four operators


def _stored(case):
    n = case["n"] + case["extra"]
    at, more = _STORED[case["body"]]
    return n * min(float(n), at + max(-0.5 * at, more * math.log(n / 5120.0, 4)))


def work(case):
    kind = case["kind"]
    if kind == "train":
        B, p = case["batch"], _NF * _H + _H + _H * _H + _H + _H * _NC + _NC
        return {"bytes": B * (_NF * 4 + 1) + 4 * (4 * p + 3 * p + p + 1),
                "flops": 6.0 * B * p + 12.0 * p}
    n, R = case["n"] + case["extra"], case["rhs"]
    if kind == "field":
        M = case["pts"]
        return {"bytes": 72.0 * n + 32.0 * n * R + 24.0 * M + 32.0 * M * R,
                "flops": float(M) * n * (7 * 30.0 + 16.0 * R)}
    e = _stored(case)
    es = 8 if case["mixed"] else 16
    product = {"bytes": e * es + 32.0 * n * R, "flops": 8.0 * e * R}
    if kind == "product":
        return product
    if kind == "hlu_solve":  # rank-2 factors: about a tenth of the stored entries
        return {"bytes": 0.1 * e * es + 32.0 * n * R, "flops": 0.8 * e * R}
    # a solve: the entries of both matrices, the products of GMRES
    its = 10 if case.get("hlu") else (30 if case["body"] == "sphere" else 100)
    one = {"bytes": 72.0 * n + (32.0 + 3 * 16.0) * n * R + 32.0 * n,
           "flops": 2 * e * 16 * _POINT_FLOPS + (its + 4) * product["flops"]}
    nf = case.get("nf", 1)
    return {k: nf * v for k, v in one.items()}


# ---------------------------------------------------------------- 64-bit values

def _orbits(centre, threes, sixes=()):
    """Symmetric triangle rule from its published orbits: barycentric
    coordinates and weights (they sum to 1)."""
    pts = [(1 / 3, 1 / 3, centre)]
    for a, w in threes:
        pts += [(a, a, w), (a, 1 - 2 * a, w), (1 - 2 * a, a, w)]
    for a, b, w in sixes:
        c = 1 - a - b
        pts += [(x, y, w) for x, y in ((a, b), (b, a), (a, c), (c, a), (b, c), (c, b))]
    return pts


# 16 points, order 8 (Dunavant 1985), and 7 points, order 5 (Radon 1948)
_RULE16 = _orbits(0.144315607677787,
                  [(0.459292588292723, 0.095091634267285), (0.170569307751760, 0.103217370534718),
                   (0.050547228317031, 0.032458497623198)],
                  [(0.008394777409958, 0.263112829634638, 0.027230314174435)])
_S15 = math.sqrt(15.0)
_RULE7 = _orbits(9 / 40, [((6 - _S15) / 21, (155 - _S15) / 1200),
                          ((6 + _S15) / 21, (155 + _S15) / 1200)])


class _Geometry:
    """Centroids, normals, areas and vertices on the GPU, in 64 bits."""

    def __init__(self, tri):
        t = torch.from_numpy(np.array(tri)).cuda().reshape(-1, 3, 3)
        self.v = t
        self.c = t.mean(1)
        nr = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
        ln = torch.linalg.vector_norm(nr, dim=1)
        self.n, self.area = nr / ln[:, None], 0.5 * ln
        self.near = 2.0 * float(self.area.sqrt().mean())  # closer pairs are near-singular


def _point_sum(p, n_p, q, n_q, w, k):
    """Sums over the last axis of G, dG/dn_q, dG/dn_p and d2G/dn_p dn_q times w,
    G = exp(ikr) / (4 pi r); p, n_p, n_q (.., 1, 3), q (.., points, 3)."""
    d = p - q
    r = torch.linalg.vector_norm(d, dim=-1)
    a, b = (d * n_p).sum(-1) / r, -(d * n_q).sum(-1) / r
    up = (n_p * n_q).sum(-1)
    G = torch.polar(w / (4 * math.pi * r), k * r)
    ikr = torch.complex(torch.zeros_like(r), k * r)
    d1 = G / r * (ikr - 1)
    d2 = G / r ** 2 * (2 - 2 * ikr - (k * r) ** 2)
    return G.sum(-1), (b * d1).sum(-1), (a * d1).sum(-1), \
        (-(up + a * b) / r * d1 + a * b * d2).sum(-1)


def _closest(v, p):
    """Barycentric coordinates of the closest points of the triangles v to p."""
    a, b, c = v[:, 0], v[:, 1], v[:, 2]
    e0, e1, d = b - a, c - a, p - a
    m = torch.stack([(e0 * e0).sum(1), (e0 * e1).sum(1), (e1 * e1).sum(1)], 1)
    f0, f1 = (d * e0).sum(1), (d * e1).sum(1)
    det = m[:, 0] * m[:, 2] - m[:, 1] ** 2
    s, t = (m[:, 2] * f0 - m[:, 1] * f1) / det, (m[:, 0] * f1 - m[:, 1] * f0) / det
    bary = torch.stack([1 - s - t, s, t], 1)
    best = torch.full_like(s, math.inf)
    edge = torch.zeros_like(bary)
    for q in range(3):
        u, w = v[:, q], v[:, (q + 1) % 3]
        t = (((p - u) * (w - u)).sum(1) / ((w - u) ** 2).sum(1)).clamp(0, 1)
        far = ((p - u - t[:, None] * (w - u)) ** 2).sum(1)
        at = torch.zeros_like(bary)
        at[:, q], at[:, (q + 1) % 3] = 1 - t, t
        edge = torch.where((far < best)[:, None], at, edge)
        best = torch.minimum(best, far)
    return torch.where((bary > 0).all(1)[:, None], bary, edge)


def _near_ops(g, rows, cols, k):
    """The four operators of close pairs: the source triangle split at its
    point closest to the collocation point (moved to an edge or a corner within
    0.05 of it), 5 x 5 polar Gauss-Legendre points about it on every part."""
    x, w = (torch.from_numpy(t).cuda() for t in np.polynomial.legendre.leggauss(5))
    out = torch.zeros((len(rows), 4), dtype=torch.complex128, device="cuda")
    step = 1 << 16
    for o in range(0, len(rows), step):
        i, j = rows[o:o + step], cols[o:o + step]
        v, p = g.v[j], g.c[i]
        bary = _closest(v, p)
        keep = bary > 0.05
        spare = torch.where(keep, 0.0, bary).sum(1) / keep.sum(1)
        bary = torch.where(keep, bary + spare[:, None], 0.0)
        at = (bary[:, :, None] * v).sum(1)
        for q in range(3):  # the part on the edge opposite corner q
            use = torch.nonzero(keep[:, q])[:, 0]
            if not len(use):
                continue
            a, b, c = at[use], v[use, (q + 1) % 3], v[use, (q + 2) % 3]
            ab, ac = b - a, c - a
            lab = torch.linalg.vector_norm(ab, dim=1)
            e0 = ab / lab[:, None]
            e1 = ac - (ac * e0).sum(1)[:, None] * e0
            h = torch.linalg.vector_norm(e1, dim=1)
            e1 = e1 / h[:, None]
            ang = torch.atan2(h, (ac * e0).sum(1))
            ang_b = torch.atan2(h, lab - (ac * e0).sum(1))
            th = 0.5 * ang[:, None] * (1 + x)
            far = lab[:, None] * torch.sin(ang_b)[:, None] / torch.sin(th + ang_b[:, None])
            r = 0.5 * far[:, :, None] * (1 + x)
            pts = a[:, None, None] + (r * torch.cos(th)[:, :, None])[..., None] * e0[:, None, None] \
                + (r * torch.sin(th)[:, :, None])[..., None] * e1[:, None, None]
            wt = 0.25 * ang[:, None, None] * far[:, :, None] * r * w[:, None] * w
            ops = _point_sum(p[use][:, None], g.n[i[use]][:, None], pts.reshape(len(use), 25, 3),
                             g.n[j[use]][:, None], wt.reshape(len(use), 25), k)
            out[o + use] += torch.stack(ops, 1)
    return out


def _self_ops(g, k):
    """L and N of a flat element at its own centroid (polar form, finite part)."""
    x, w = (torch.from_numpy(t).cuda() for t in np.polynomial.legendre.leggauss(32))
    L = torch.zeros(len(g.c), dtype=torch.complex128, device="cuda")
    N = torch.full_like(L, 0.5j * k)
    for e in range(3):
        a, b = g.v[:, e] - g.c, g.v[:, (e + 1) % 3] - g.c
        la, lb = torch.linalg.vector_norm(a, dim=1), torch.linalg.vector_norm(b, dim=1)
        ang = torch.acos((a * b).sum(1) / (la * lb))
        h = torch.linalg.vector_norm(torch.linalg.cross(a, b), dim=1) \
            / torch.linalg.vector_norm(a - b, dim=1)
        t0 = -torch.acos((h / la).clamp(max=1.0))
        foot = ((b - a) * -a).sum(1) > 0  # the foot of the height lies beyond a
        t0 = torch.where(foot, t0, -t0)
        th = t0[:, None] + 0.5 * ang[:, None] * (x + 1)
        R = h[:, None] / torch.cos(th)
        wt = 0.5 * ang[:, None] * w
        E = torch.polar(torch.ones_like(R), k * R)
        L += ((E - 1) * wt).sum(1) / (4 * math.pi * 1j * k)
        N -= (E / R * wt).sum(1) / (4 * math.pi)
    return L, N


def _robin(case, n, k):
    """a of a phi + dphi = g, per element."""
    beta = _beta(case, n)
    if beta is None:
        return torch.zeros(n, dtype=torch.complex128, device="cuda")
    return 1j * k * torch.from_numpy(beta).cuda()


def _dense(case, tri, freq):
    """Right-hand-side and system matrix of the collocation method, rows in
    chunks: yields (first row, phi rows, dphi rows), in the order of `tri`."""
    k = 2 * math.pi * freq / C0
    g = _Geometry(tri)
    n = len(g.c)
    al = 1j / (k + 1.0)  # Kirkup coupling
    a = _robin(case, n, k)
    swap = a.abs() >= 1.0
    ls, ns = _self_ops(g, k)
    step = max(1, (1 << 21) // n)
    for r0 in range(0, n, step):
        i = torch.arange(r0, min(n, r0 + step), device="cuda")
        p, n_p = g.c[i][:, None], g.n[i][:, None]
        ops = [torch.zeros((len(i), n), dtype=torch.complex128, device="cuda") for _ in range(4)]
        for x1, x2, wt in _RULE16:
            q = x1 * g.v[:, 0] + x2 * g.v[:, 1] + (1 - x1 - x2) * g.v[:, 2]
            one = _point_sum(p[:, :, None], n_p[:, :, None], q[None, :, None], g.n[None, :, None],
                             (wt * g.area)[None, :, None], k)
            for o, v in zip(ops, one):
                o += v
        dist = torch.linalg.vector_norm(p - g.c[None], dim=2)
        own = i[:, None] == torch.arange(n, device="cuda")[None]
        at, to = torch.nonzero((dist < g.near) & ~own, as_tuple=True)
        v = _near_ops(g, i[at], to, k)
        for q in range(4):
            ops[q][at, to] = v[:, q]
        L, M, Mt, N = ops
        L[own], M[own], Mt[own], N[own] = ls[i], 0.0, 0.0, ns[i]
        X, Y = L + al * Mt, M + al * N
        X[own] += 0.5 * al
        Y[own] -= 0.5
        # the unknown of an element is dphi where |a| >= |b| = 1, else phi
        yield (r0, torch.where(swap, Y / torch.where(swap, a, 1.0), -X),
               torch.where(swap, X + Y / torch.where(swap, a, 1.0), -a * X - Y))


def _solved(case, tri, freq, g):
    """phi, dphi and p of the dense system, or None where that takes too long."""
    n = len(tri)
    if n > 21000 or (n > 6000 and case["body"] != "sphere"):
        return None
    A = torch.empty((n, n), dtype=torch.complex128, device="cuda")
    gd = torch.from_numpy(np.ascontiguousarray(g)).cuda()
    rhs = torch.empty_like(gd)
    for r0, phi, dphi in _dense(case, tri, freq):
        A[r0:r0 + len(phi)] = dphi
        rhs[r0:r0 + len(phi)] = phi @ gd
    x = torch.linalg.solve(A, rhs) if n <= 6000 else _krylov(A, rhs)
    a = _robin(case, n, 2 * math.pi * freq / C0)[:, None]
    swap = a.abs() >= 1.0
    phi = torch.where(swap, (gd - x) / torch.where(swap, a, 1.0), x)
    dphi = torch.where(swap, x, gd - a * x)
    return [v.cpu().numpy() for v in (phi, dphi, 1j * RHO * 2 * math.pi * freq * phi)]


def _krylov(A, b, steps=80):
    """GMRES without restart, column by column."""
    out = torch.empty_like(b)
    for c in range(b.shape[1]):
        beta = torch.linalg.vector_norm(b[:, c])
        V, H = [b[:, c] / beta], torch.zeros((steps + 1, steps), dtype=b.dtype, device="cuda")
        for j in range(steps):
            w = A @ V[j]
            B = torch.stack(V, 1)
            for _ in range(2):
                h = B.conj().T @ w
                w = w - B @ h
                H[:j + 1, j] += h
            H[j + 1, j] = torch.linalg.vector_norm(w)
            V.append(w / H[j + 1, j])
        e = torch.zeros((steps + 1, 1), dtype=b.dtype, device="cuda")
        e[0] = beta
        out[:, c] = torch.stack(V[:-1], 1) @ torch.linalg.lstsq(H, e).solution[:, 0]
    return out


def _exact_field(case, tri, freq, rng):
    pts, phi, dphi, src = _field_inputs(case, tri, freq, rng)
    k = 2 * math.pi * freq / C0
    g = _Geometry(tri)
    p = torch.from_numpy(pts).cuda()
    ph, dp = (torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (phi, dphi))
    out = torch.zeros((len(pts), case["rhs"]), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 24) // len(tri))
    for o in range(0, len(pts), step):
        for a, b, wt in _RULE7:
            q = a * g.v[:, 0] + b * g.v[:, 1] + (1 - a - b) * g.v[:, 2]
            d = p[o:o + step, None] - q[None]
            r = torch.linalg.vector_norm(d, dim=2)
            G = torch.polar((wt * g.area)[None] / (4 * math.pi * r), k * r)
            t = -(d * g.n[None]).sum(2) / r ** 2
            M = t * G * (torch.complex(torch.zeros_like(r), k * r) - 1)
            out[o:o + step] += M @ ph - G @ dp
    if src is not None:
        for s in src:
            r = torch.linalg.vector_norm(p - torch.from_numpy(s[:3].real.copy()).cuda(), dim=1)
            out += (complex(s[3]) * torch.polar(1 / (4 * math.pi * r), k * r))[:, None]
    both = [out, 1j * RHO * 2 * math.pi * freq * out]
    return [v.cpu().numpy() for v in both] if case["pts"] < 2000 else [v.T.contiguous() for v in both]


def _exact_train(case, rng):
    x = _train_inputs(case, rng)
    prm = torch.from_numpy(x["params"]).double().cuda().requires_grad_()
    X, y = torch.from_numpy(x["X"]).double().cuda(), torch.from_numpy(x["y"]).long().cuda()
    h, o = X, 0
    for i, n in ((_NF, _H), (_H, _H), (_H, _NC)):
        h = h @ prm[o:o + i * n].reshape(i, n) + prm[o + i * n:o + i * n + n]
        h = torch.relu(h) if n == _H else h
        o += i * n + n
    loss = torch.nn.functional.cross_entropy(h, y)
    loss.backward()
    g = prm.grad
    m, v = 0.1 * g, 0.001 * g * g
    new = prm.detach() - 3e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return [g, loss.detach().reshape(1), new]


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, rng)
    if kind == "hlu_solve":  # a rank-2 approximation of the inverse: no value of its own
        return None
    jitter = 1.0 + 0.02 * rng.random()
    tri = _mesh(case["body"], case["n"], case["extra"])
    freq = case["freq"] * jitter
    if kind == "field":
        return _exact_field(case, tri, freq, rng)
    if kind == "product":
        # vectors are in the order of the cluster tree
        perm, _ = pkg.plan_mesh(tri)
        x = torch.from_numpy(_waves(rng, (case["rhs"], len(tri)))).cuda()
        at = torch.from_numpy(perm).cuda()
        xc = torch.empty_like(x)
        xc[:, at] = x
        y = torch.empty_like(xc)
        for r0, phi, dphi in _dense(case, tri, freq):
            y[:, r0:r0 + len(phi)] = ((dphi if case["which"] else phi) @ xc.T).T
        return y[:, at].contiguous()
    g = _drive(case, tri, rng)
    if kind == "solve":
        return _solved(case, tri, freq, g)
    if len(tri) > 6000:
        return None
    fr = meshes.log_frequencies(case["nf"], case["freq"], case["freq_to"]) * jitter
    return [np.stack([_solved(case, tri, float(f), g)[2] for f in fr], axis=2)]
