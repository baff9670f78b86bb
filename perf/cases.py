"""The work whose speed is measured, through the framework's public entry points.

Kinds of call:
  sphere   ``acoustics3d.sphere``: the Mie-check call on an icosphere, a context of its own per call
           (leaf 128, factor 1.5, ACA and solver tolerances 1e-10)
  pvals    ``DiffBEM.set_points`` + ``DiffBEM.pvals``: new vertex positions, one forward solve at one
           frequency, plane wave, pressures at 181 receivers (leaf 32, factor 2, ACA 1e-4, 1e-6)
  band     ``DiffBEM.band_value`` + ``pvals`` with the reference pipeline's parameters (leaf 128,
           factor 1.5, 3 frequencies per band, tolerances 1e-5, point source, 1297-point hemisphere,
           receiver ACA, BiCGSTAB)
  multi    ``DiffBEM.pvals_multi``: several incident fields as one block of right-hand sides
  step     one optimiser step: float32 heightmap texture -> ``TexMap`` -> ``diffusion_coefficient``
           -> backward to the texture (forward and adjoint solves and the shape derivative)
  grads    ``DiffBEM.gradient_multi``: several frequencies x plane-wave directions with the gradient
  served   ``serve.Server`` with 4 slots: a batch of requests over reliefs of three sizes

Reliefs are boxes with a seeded, smoothed 64 x 64 heightmap on the top face (nx x ny x nz quads,
the top face subdivided ``sub`` times), spheres are icospheres with a seeded radius and rotation.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from acoustic_reliefs_gb300 import meshes
from acoustic_reliefs_gb300.acoustics3d import DiffBEM, sphere
from acoustic_reliefs_gb300.autograd import TexMap, diffusion_coefficient
from acoustic_reliefs_gb300.serve import Server

TEX = 64
RECEIVERS = 181
SERVED_SIZES = ((30, 7, 0), (30, 7, 1), (64, 8, 0))  # (nx = nz, ny, subdivisions): 5280, 10680, 20480 triangles


def listed():
    return [
        # the FP64 path, with set-up and teardown of a context in the call: validation against the Mie series
        {"name": "sphere_fp64_1280", "kind": "sphere", "sub": 3, "freq": 500.0, "n": 181, "precision": "fp64"},
        # the smallest solve with the drop-in's defaults (mixed, BiCGSTAB): launches and host latency count
        {"name": "pvals_sphere_1280", "kind": "pvals", "mesh": "sphere", "sub": 3, "freq": 500.0, "precision": "mixed",
         "krylov": "bicgstab"},
        # the smallest relief of the served sweep at mid frequency
        {"name": "pvals_relief_5280", "kind": "pvals", "mesh": "relief", "nx": 30, "ny": 7, "nz": 30, "sub": 0,
         "freq": 2000.0, "precision": "mixed", "krylov": "gmres"},
        # the same solve on the FP64 path, which users compare the mixed one with
        {"name": "pvals_fp64_5280", "kind": "pvals", "mesh": "relief", "nx": 30, "ny": 7, "nz": 30, "sub": 0,
         "freq": 2000.0, "precision": "fp64", "krylov": "gmres"},
        # the benchmark's solve
        {"name": "pvals_relief_20480", "kind": "pvals", "mesh": "relief", "nx": 64, "ny": 8, "nz": 64, "sub": 0,
         "freq": 2000.0, "precision": "mixed", "krylov": "gmres"},
        # the largest relief of the served sweep: memory-bound matvecs, a long assembly
        {"name": "pvals_relief_118680", "kind": "pvals", "mesh": "relief", "nx": 30, "ny": 7, "nz": 30, "sub": 3,
         "freq": 2000.0, "precision": "mixed", "krylov": "gmres"},
        # the reference pipeline's parameters on a mid-size relief (larger leaves, receiver ACA, BiCGSTAB)
        {"name": "band_relief_10680", "kind": "band", "nx": 30, "ny": 7, "nz": 30, "sub": 1, "freq": 1000.0},
        # 16 incidence directions as one block (tensor-core dot pass)
        {"name": "multi16_relief_20480", "kind": "multi", "nx": 64, "ny": 8, "nz": 64, "sub": 0, "freq": 2000.0,
         "rhs": 16, "krylov": "gmres", "incident": "plane"},
        # a ragged block of point sources on an odd-sized relief with the default solver
        {"name": "multi5_relief_7628", "kind": "multi", "nx": 37, "ny": 5, "nz": 41, "sub": 0, "freq": 1000.0,
         "rhs": 5, "krylov": "bicgstab", "incident": "point"},
        # one optimiser step on the smallest sweep relief
        {"name": "step_relief_5280", "kind": "step", "nx": 30, "ny": 7, "nz": 30, "sub": 0, "freq": 1000.0,
         "krylov": "gmres"},
        # the multi-incidence objective with its gradient
        {"name": "grads6_relief_5280", "kind": "grads", "nx": 30, "ny": 7, "nz": 30, "sub": 0, "freq": 1000.0,
         "dirs": 6, "krylov": "gmres"},
        # a served batch: 12 requests of mixed sizes and frequencies, 4 at a time
        {"name": "served_12", "kind": "served", "requests": 12, "low": 500.0, "high": 2500.0},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["sphere", "pvals", "pvals", "pvals", "band", "multi", "multi", "step", "grads", "served"])
    freq = round(_log(rng, 100.0, 3000.0), 1)
    krylov = rng.choice(["gmres", "gmres", "bicgstab"])

    def grid(lo, hi):
        nx = int(round(_log(rng, lo, hi)))
        nz = max(lo, min(hi, nx + rng.randint(-3, 3)))
        return {"nx": nx, "ny": rng.randint(2, 9), "nz": nz, "sub": 0}

    if kind == "sphere":
        return {"kind": kind, "sub": rng.choice([2, 3]), "freq": round(_log(rng, 100.0, 800.0), 1),
                "n": rng.randint(30, 400), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "pvals":
        g = grid(12, 120)
        prec = "fp64" if g["nx"] <= 30 and rng.random() < 0.3 else "mixed"
        return {"kind": kind, "mesh": "relief", **g, "freq": freq, "precision": prec, "krylov": krylov}
    if kind == "band":
        return {"kind": kind, **grid(16, 48), "freq": round(min(freq, 1250.0), 1)}
    if kind == "multi":
        return {"kind": kind, **grid(14, 56), "freq": freq, "rhs": rng.randint(2, 20), "krylov": krylov,
                "incident": rng.choice(["plane", "point"])}
    if kind == "step":
        return {"kind": kind, **grid(10, 48), "freq": freq, "krylov": krylov}
    if kind == "grads":
        return {"kind": kind, **grid(10, 36), "freq": freq, "dirs": rng.randint(2, 18), "krylov": krylov}
    return {"kind": kind, "requests": rng.randint(4, 16), "low": 250.0, "high": round(_log(rng, 800.0, 3000.0), 1)}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _relief(case, seed):
    """(Ps, Es, top vertex ids, their uvs) of the case's relief with the seed's heightmap."""
    P, E, top, uv = (t.cpu().numpy() for t in meshes.relief_device(0.6, 0.6, 0.05, case["nx"], case["ny"], case["nz"],
                                                                  case["sub"]))
    P[top, 1] += meshes.sample_heightmap(meshes.smooth_heightmap(TEX, seed), uv)
    return P, E, top, uv


def _sphere_mesh(case, seed):
    rng = np.random.default_rng(seed)
    P, E = meshes.icosphere(case["sub"], 0.5 * rng.uniform(0.96, 1.04))
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    return P @ (q * np.sign(np.linalg.det(q))).T, E


def _directions(n, seed):
    d = np.random.default_rng(seed + 1).normal(size=(n, 3))
    d[:, 1] = -np.abs(d[:, 1]) - 0.5
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _vectors(case, seed):
    d = _directions(case["rhs"], seed)
    return d if case["incident"] == "plane" else -d * 10.0  # point sources 10 m above the relief


def _band(case):
    bw = 2.0 ** (1.0 / 6.0)
    return [float(f) for f in np.exp(np.linspace(np.log(case["freq"] / bw), np.log(case["freq"] * bw), 3))]


def _requests(case, seed):
    rng = np.random.default_rng(seed + 2)
    n = case["requests"]
    f = np.exp(rng.uniform(math.log(case["low"]), math.log(case["high"]), size=n))
    return [(i % len(SERVED_SIZES), float(f[i])) for i in range(n)]


def _served_mesh(m, seed):
    nx, ny, sub = SERVED_SIZES[m]
    return _relief({"nx": nx, "ny": ny, "nz": nx, "sub": sub}, seed + m)


def _bem(case, precision="mixed", **kw):
    b = DiffBEM(32, 2.0, [case["freq"]], kw.pop("n_freqs", 1), 1e-4, 1e-4, 1e-6, precision=precision, **kw)
    b.silent = True
    b.set_krylov(case.get("krylov", "bicgstab"))
    return b


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "sphere":
        st["mesh"] = _sphere_mesh(case, seed)
    elif kind == "pvals":
        if case["mesh"] == "sphere":
            P, E = _sphere_mesh(case, seed)
            st["Ls"], d = meshes.circle_xz(5.0, RECEIVERS), (0.0, 0.0, -1.0)
        else:
            P, E, _, _ = _relief(case, seed)
            st["Ls"], d = meshes.semicircle(5.0, RECEIVERS), (0.0, -1.0, 0.0)
        st["bem"] = _bem(case, case["precision"], incident=("plane", d))
        st["bem"].set_mesh(P, E)
        st["Ps"] = P
    elif kind == "band":
        P, E, _, _ = _relief(case, seed)
        b = DiffBEM(128, 1.5, [case["freq"]], 3, 1e-5, 1e-5, 1e-5, (0.0, 100.0, 0.0), 50, 5, listener="aca")
        b.silent = True
        b.set_mesh(P, E)
        st["bem"] = b
    elif kind == "multi":
        P, E, _, _ = _relief(case, seed)
        st["bem"] = _bem(case)
        st["bem"].set_mesh(P, E)
        st["vecs"], st["Ls"] = _vectors(case, seed), meshes.semicircle(5.0, RECEIVERS)
    elif kind == "step":
        P, E, top, uv = _relief(case, seed)
        P[top, 1] = 0.05
        st["bem"] = _bem(case, n_freqs=2)
        st["bem"].set_listeners(meshes.semicircle(10.0, RECEIVERS))
        st["bem"].precompute(P, E, top)
        st["map"] = TexMap(uv, (TEX, TEX))
        st["tex"] = torch.tensor(meshes.smooth_heightmap(TEX, seed), dtype=torch.float32, device="cuda",
                                 requires_grad=True)
    elif kind == "grads":
        P, E, top, _ = _relief(case, seed)
        st["bem"] = _bem(case)
        st["bem"].set_listeners(meshes.semicircle(10.0, RECEIVERS))
        st["bem"].precompute(P, E, top)
        st["x"] = np.random.default_rng(seed + 3).uniform(0.0, 0.01, size=len(top))
        st["freqs"], st["dirs"] = [case["freq"], 1.5 * case["freq"]], _directions(case["dirs"], seed)
    else:
        srv = Server(slots=4, krylov="gmres")
        st["ids"] = []
        for m in range(len(SERVED_SIZES)):
            P, E, _, _ = _served_mesh(m, seed)
            st["ids"].append(srv.add_mesh(P, E)[0])
        st["srv"], st["reqs"], st["Ls"] = srv, _requests(case, seed), meshes.semicircle(5.0, RECEIVERS)
    return st


def run(st):
    case, kind = st["case"], st["kind"]
    if kind == "sphere":
        return sphere(st["mesh"], case["freq"], case["n"], 5.0, precision=case["precision"])
    if kind == "pvals":
        st["bem"].set_points(st["Ps"])
        return st["bem"].pvals(case["freq"], st["Ls"])
    if kind == "band":
        return {"c": st["bem"].band_value(case["freq"]), "p": st["bem"].pvals(case["freq"])}
    if kind == "multi":
        p, x = st["bem"].pvals_multi(case["freq"], st["vecs"], st["Ls"], kind=case["incident"], surface=True)
        return {"p": p, "x": x}
    if kind == "step":
        st["tex"].grad = None
        c = diffusion_coefficient(st["map"](st["tex"]), st["bem"])
        (1.0 - c).backward()
        return {"c": c.detach(), "grad": st["tex"].grad}
    if kind == "grads":
        loss, g, c = st["bem"].gradient_multi(st["x"], st["freqs"], st["dirs"])
        return {"loss": loss, "grad": g, "c": c}
    hs = [st["srv"].submit(st["ids"][m], f, st["Ls"]) for m, f in st["reqs"]]
    return [st["srv"].wait(h)[0] for h in hs]


# ---------------------------------------------------------------------------------------------
# work: an estimate from sizes alone, since ranks and iterations come out of the solve itself.
# Stored entries of an H-matrix 194 Ne log2 Ne (57 M on the 20480-triangle relief); one matvec
# per iteration, each reading every entry once (8 flops) for all right-hand sides; iterations
# 30 (f / kHz)^1.6, at least 12; 6 kernel evaluations of about 60 flops per entry to build it.
# ---------------------------------------------------------------------------------------------
def _triangles(c):
    if "nx" not in c:
        return 20 * 4 ** c["sub"]
    return 4 * c["nx"] * c["ny"] + 4 * c["ny"] * c["nz"] + 2 * c["nx"] * c["nz"] * (1 + 4 ** c["sub"])


def _solve_work(ne, f, rhs=1, size=8, orientations=1):
    entries = min(ne * ne, 194.0 * ne * math.log2(ne))
    its = max(12.0, 30.0 * (f / 1000.0) ** 1.6) * orientations
    return entries * size * (1 + its), entries * (360.0 + 8.0 * its * rhs)


def work(case):
    kind = case["kind"]
    if kind == "served":
        sizes = [_triangles({"nx": a, "ny": b, "nz": a, "sub": s}) for a, b, s in SERVED_SIZES]
        mid = math.sqrt(case["low"] * case["high"])
        parts = [_solve_work(sizes[i % len(sizes)], mid) for i in range(case["requests"])]
    else:
        ne = _triangles(case)
        if kind == "band":
            parts = [_solve_work(ne, f) for f in _band(case) + [case["freq"]]]
        elif kind == "step":
            parts = [_solve_work(ne, case["freq"], 1, 8, 2)] * 2
        elif kind == "grads":
            parts = [_solve_work(ne, case["freq"] * s, case["dirs"], 8, 2) for s in (1.0, 1.5)]
        else:
            parts = [_solve_work(ne, case["freq"], case.get("rhs", 1), 16 if case.get("precision") == "fp64" else 8)]
        if kind in ("step", "grads"):  # all-pairs shape derivatives: touched panels x panels x 6 points, twice
            top = 2 * case["nx"] * case["nz"] * 4 ** case["sub"]
            parts.append((0.0, 2.0 * 2 * top * ne * 360.0))
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---------------------------------------------------------------------------------------------
# the same results from the dense operator in 64 bits
# ---------------------------------------------------------------------------------------------
_A, _B, _C, _D = 0.445948490915965, 0.108103018168070, 0.091576213509771, 0.816847572980459
_RULE = [(0.223381589678011, _A, _B), (0.223381589678011, _A, _A), (0.223381589678011, _B, _A),
         (0.109951743655322, _C, _D), (0.109951743655322, _C, _C), (0.109951743655322, _D, _C)]
EXACT_MAX = 21000  # triangles: the dense operator is Ne^2 complex128


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _rows(k, pts, P, E):
    """Double-layer entries of the points (n, 3) against every panel: 1/2 sum_q w e^{-ikr}(1 + ikr) r.n / (4 pi r^3)."""
    a, b, c = P[E[:, 0]], P[E[:, 1]], P[E[:, 2]]
    nrm = torch.linalg.cross(b - a, c - a)
    acc = 0.0
    for w, m, n in _RULE:
        y = a + m * (b - a) + n * (c - a)
        rx, ry, rz = (pts[:, None, d] - y[None, :, d] for d in range(3))
        r = torch.sqrt(rx * rx + ry * ry + rz * rz)
        f = w * (rx * nrm[:, 0] + ry * nrm[:, 1] + rz * nrm[:, 2]) / (r * r * r)
        acc = acc + f * torch.polar(torch.ones_like(r), -k * r) * torch.complex(torch.ones_like(r), k * r)
    return acc * (0.5 / (4.0 * math.pi))


def _dense(k, pts, P, E, step=1024):
    return torch.cat([_rows(k, pts[i:i + step], P, E) for i in range(0, len(pts), step)])


def _incident(k, pts, kind, v):
    v = _t(v)
    if kind == "plane":
        ph = k * (pts @ (v / v.norm()))
        return torch.polar(torch.ones_like(ph), -ph)
    r = (pts - v).norm(dim=1)
    return torch.polar(1.0 / (4.0 * math.pi * r), -k * r)


def _gmres(A, b, most=900):
    """Full GMRES to 1e-13 with two Gram-Schmidt passes."""
    beta = b.norm()
    V = torch.zeros((most + 1, len(b)), dtype=b.dtype, device=b.device)
    H = np.zeros((most + 1, most), np.complex128)
    V[0] = b / beta
    for j in range(most):
        w = A @ V[j]
        h = V[:j + 1].conj() @ w
        w = w - V[:j + 1].T @ h
        g = V[:j + 1].conj() @ w
        w = w - V[:j + 1].T @ g
        nw = w.norm()
        H[:j + 1, j], H[j + 1, j] = (h + g).cpu().numpy(), float(nw)
        V[j + 1] = w / nw
        if j % 10 == 9 or j == most - 1:
            e = np.zeros(j + 2, np.complex128)
            e[0] = float(beta)
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[0]
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) <= 1e-13 * float(beta):
                break
    return V[:len(y)].T @ torch.as_tensor(y, device=b.device)


def _operator(k, P, E):
    A = _dense(k, P[E].mean(1), P, E)
    A.diagonal().sub_(0.5)
    return A


def _wave(f):
    return 2.0 * math.pi * f / 344.0


def _pressures(f, Ps, Es, Ls, kind, vecs):
    """Receiver pressures (n, L) of the incident fields vecs: y = Q x, (K - I/2) x = -b."""
    k, P, E = _wave(f), _t(Ps), torch.as_tensor(np.asarray(Es), dtype=torch.int64, device="cuda")
    A, Q, cen = _operator(k, P, E), _dense(k, _t(Ls), P, E), P[E].mean(1)
    return np.stack([(Q @ _gmres(A, -_incident(k, cen, kind, v))).cpu().numpy() for v in np.atleast_2d(vecs)])


def _coefficient(y):
    v = np.abs(y) ** 2
    return float((v.sum() ** 2 - (v * v).sum()) / ((len(v) - 1) * (v * v).sum()))


def _objective(freqs, fields, group, Ps, Es, top, x, Ls):
    """Coefficients of the groups (one per group, of sum_f |y_f|) and the gradient of their sum over
    the heights x: adjoint solves, then torch's derivative of the frozen bilinear form."""
    E = torch.as_tensor(np.asarray(Es), dtype=torch.int64, device="cuda")
    tp = torch.as_tensor(np.asarray(top), dtype=torch.int64, device="cuda")
    h = _t(x).requires_grad_(True)
    L = _t(Ls)

    def points():
        P = _t(Ps)
        return torch.index_put(P, (tp, torch.ones_like(tp)), P[tp, 1] + h)

    with torch.no_grad():
        P0 = points()
        cen = P0[E].mean(1)
        sol = {}
        for f in sorted(set(freqs)):
            A, Q = _operator(_wave(f), P0, E), _dense(_wave(f), L, P0, E)
            for i, fi in enumerate(freqs):
                if fi == f:
                    s = _gmres(A, -_incident(_wave(f), cen, *fields[i]))
                    sol[i] = (s, Q @ s)
            del A, Q
        coefs, vf = [], {}
        for g in sorted(set(group)):
            mine = [i for i in range(len(freqs)) if group[i] == g]
            yt = sum(sol[i][1].abs() for i in mine)
            v = yt * yt
            S, T, n = v.sum(), (v * v).sum(), len(v) - 1
            coefs.append(float((S * S - T) / (n * T)))
            u = 4 * (S * T - v * S * S) / (n * T * T) * yt
            for i in mine:
                y = sol[i][1]
                vf[i] = u * y.conj() / y.abs()
        lam = {}
        for f in sorted(set(freqs)):
            A, Q = _operator(_wave(f), P0, E), _dense(_wave(f), L, P0, E)
            for i, fi in enumerate(freqs):
                if fi == f:
                    lam[i] = _gmres(A.T, Q.T @ vf[i])
            del A, Q
    step = 256
    for f in sorted(set(freqs)):
        k, mine = _wave(f), [i for i, fi in enumerate(freqs) if fi == f]
        for c0 in list(range(0, len(E), step)) + [-1]:
            P = points()
            if c0 < 0:
                M, rows = _rows(k, L, P, E), None
            else:
                rows = slice(c0, min(c0 + step, len(E)))
                M = _rows(k, P[E[rows]].mean(1), P, E)
            s = 0.0
            for i in mine:
                if rows is None:
                    s = s + (vf[i] @ (M @ sol[i][0])).real
                else:
                    b = _incident(k, P[E[rows]].mean(1), *fields[i])
                    s = s - (lam[i][rows] @ (M @ sol[i][0] + b)).real
            s.backward()
    return coefs, h.grad.cpu().numpy()


def _bilinear(uv):
    """Texel rows, columns and weights (n, 4) of the bilinear lookup at uv, clamped at the far edges."""
    uf, ui = np.modf(uv[:, 0] * TEX - 0.5)
    vf, vi = np.modf(uv[:, 1] * TEX - 0.5)
    uf, vf = np.where(uf < 0, 1 + uf, uf), np.where(vf < 0, 1 + vf, vf)
    ui, vi = np.maximum(ui.astype(int), 0), np.maximum(vi.astype(int), 0)
    u1, v1 = np.minimum(ui + 1, TEX - 1), np.minimum(vi + 1, TEX - 1)
    return (np.stack([vi, vi, v1, v1], 1), np.stack([ui, u1, ui, u1], 1),
            np.stack([(1 - vf) * (1 - uf), (1 - vf) * uf, vf * (1 - uf), vf * uf], 1))


def exact(case, seed):
    kind = case["kind"]
    if kind != "served" and _triangles(case) > (6000 if kind in ("step", "grads") else EXACT_MAX):
        return None
    if kind == "sphere":
        P, E = _sphere_mesh(case, seed)
        th = np.arange(case["n"]) / case["n"] * 2 * math.pi
        Ls = np.column_stack([5.0 * np.cos(th), np.zeros(case["n"]), -5.0 * np.sin(th)])
        return _pressures(case["freq"], P, E, Ls, "plane", (1.0, 0.0, 0.0))[0]
    if kind == "pvals":
        if case["mesh"] == "sphere":
            (P, E), Ls, d = _sphere_mesh(case, seed), meshes.circle_xz(5.0, RECEIVERS), (0.0, 0.0, -1.0)
        else:
            (P, E, _, _), Ls, d = _relief(case, seed), meshes.semicircle(5.0, RECEIVERS), (0.0, -1.0, 0.0)
        return _pressures(case["freq"], P, E, Ls, "plane", d)[0]
    if kind == "band":
        P, E, _, _ = _relief(case, seed)
        el = np.radians([0.0] + [e for e in range(5, 91, 5) for _ in range(72)])
        az = np.radians([0.0] + [a for _ in range(5, 91, 5) for a in range(0, 360, 5)])
        Ls = 50.0 * np.column_stack([np.sin(el) * np.cos(az), np.cos(el), -np.sin(el) * np.sin(az)])
        src = (0.0, 100.0, 0.0)
        y = sum(np.abs(_pressures(f, P, E, Ls, "point", src)[0]) for f in _band(case))
        return {"c": _coefficient(y), "p": _pressures(case["freq"], P, E, Ls, "point", src)[0]}
    if kind == "multi":
        P, E, _, _ = _relief(case, seed)
        Ls = meshes.semicircle(5.0, RECEIVERS)
        return {"p": _pressures(case["freq"], P, E, Ls, case["incident"], _vectors(case, seed)), "x": None}
    if kind == "step":
        P, E, top, uv = _relief(case, seed)
        P[top, 1] = 0.05
        tex = meshes.smooth_heightmap(TEX, seed).astype(np.float32).astype(np.float64)
        r, c, w = _bilinear(uv)
        heights = (tex[r, c] * w).sum(1).astype(np.float32).astype(np.float64)
        bw = 2.0 ** (1.0 / 6.0)
        src = ("point", (0.0, 100.0, 0.0))
        cs, g = _objective([case["freq"] / bw, case["freq"] * bw], [src, src], [0, 0], P, E, top, heights,
                           meshes.semicircle(10.0, RECEIVERS))
        tg = np.zeros((TEX, TEX))
        np.add.at(tg, (r.reshape(-1), c.reshape(-1)), (w * -g[:, None]).reshape(-1))
        return {"c": np.array(cs[0]), "grad": tg}
    if kind == "grads":
        P, E, top, _ = _relief(case, seed)
        x = np.random.default_rng(seed + 3).uniform(0.0, 0.01, size=len(top))
        dirs = _directions(case["dirs"], seed)
        fs = [s * case["freq"] for s in (1.0, 1.5) for _ in dirs]
        fields = [("plane", d) for _ in range(2) for d in dirs]
        cs, g = _objective(fs, fields, list(range(len(fs))), P, E, top, x, meshes.semicircle(10.0, RECEIVERS))
        return {"loss": 1.0 - float(np.mean(cs)), "grad": -g / len(fs), "c": np.array(cs).reshape(2, len(dirs))}
    Ls = meshes.semicircle(5.0, RECEIVERS)
    mesh = [_served_mesh(m, seed)[:2] for m in range(len(SERVED_SIZES))]
    return [_pressures(f, *mesh[m], Ls, "plane", (0.0, -1.0, 0.0))[0] if m == 0 else None
            for m, f in _requests(case, seed)]
