"""Timing cases of the scattering library, through its public Python entry points.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges,
``prepare`` what a program holds before the call (an uploaded problem on its
own context, sources, wavelengths), ``run`` one pass, ``work`` what a pass
cannot do without and ``exact`` the results in plain 64-bit torch.

Particles are geodesic spheres of frequency f (20 f^2 triangles, 60 f^2
unknowns: f = 8 and 16 have the sizes of the 3,840- and 15,360-unknown spheres
of the benchmark) deformed into smooth seeded ellipsoid-like shapes of
30-70 nm semi-axes, with a Drude metal inside, at optical wavelengths.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "for90-mom2_b200"))
import mom_b200 as mom  # noqa: E402
from mom_b200 import meshgen  # noqa: E402

FP64, MIXED = mom.FP64, mom.MIXED
PREC = {"fp64": FP64, "mixed": MIXED}


def listed():
    return [
        # the smallest particle: a call in an optimiser's inner loop, all launches and latency
        {"name": "solve-240-fp64", "kind": "solve", "freq": 2, "precision": "fp64", "sources": 1},
        # a single particle in the reference's own arithmetic, one polarisation
        {"name": "solve-3840-fp64", "kind": "solve", "freq": 8, "precision": "fp64", "sources": 1},
        # a mid-sized particle of a ragged order, three incidences
        {"name": "solve-7260-mixed", "kind": "solve", "freq": 11, "precision": "mixed", "sources": 3},
        # the largest single solve in FP64 (order not a multiple of the block sizes)
        {"name": "solve-11760-fp64", "kind": "solve", "freq": 14, "precision": "fp64", "sources": 2},
        # the benchmark's size: one wavelength in mixed precision
        {"name": "solve-15360-mixed", "kind": "solve", "freq": 16, "precision": "mixed", "sources": 1},
        # a spectrum of particles of uneven sizes, several contexts at once
        {"name": "sweep-4x16-mixed", "kind": "sweep", "freq": 8, "particles": 4, "contexts": 3, "wavelengths": 16,
         "precision": "mixed"},
        # shape and material gradients of one design step (forward solve and backward)
        {"name": "gradient-3840-fp64", "kind": "gradient", "freq": 8, "precision": "fp64", "nodes": True},
        # orientation average: core-shell particle, many incidences on one factorisation
        {"name": "shell-7680-mixed", "kind": "shell", "freq": 8, "precision": "mixed", "sources": 512},
        # its backward direction: gradient of the mean cross sections (transposed solves)
        {"name": "shell-gradient-4320-fp64", "kind": "shell_gradient", "freq": 6, "precision": "fp64", "sources": 96},
        # post-processing of one solution: far-field map and a plane of near fields
        {"name": "maps-3840", "kind": "maps", "freq": 8, "ntheta": 91, "nphi": 180, "plane": 101},
        # second harmonic after the fundamental solve
        {"name": "harmonic-2940-mixed", "kind": "harmonic", "freq": 7, "precision": "mixed"},
        # an eighth of a particle with three mirror planes: eight representations
        {"name": "mirror-8x1800-fp64", "kind": "mirror", "freq": 24, "precision": "fp64"},
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "sweep", "gradient", "shell", "shell_gradient", "maps", "harmonic",
                       "mirror"])
    prec = rng.choice(["fp64", "mixed"])

    def freq(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "solve":
        return {"kind": kind, "freq": freq(2, 15 if prec == "mixed" else 12), "precision": prec,
                "sources": rng.randint(1, 6)}
    if kind == "sweep":
        return {"kind": kind, "freq": freq(4, 8), "particles": rng.randint(1, 4), "contexts": rng.randint(1, 3),
                "wavelengths": rng.randint(3, 16), "precision": prec}
    if kind == "gradient":
        return {"kind": kind, "freq": freq(2, 7), "precision": prec, "nodes": rng.random() < 0.7}
    if kind == "shell":
        return {"kind": kind, "freq": freq(2, 8), "precision": prec, "sources": freq(3, 500)}
    if kind == "shell_gradient":
        return {"kind": kind, "freq": freq(2, 6), "precision": prec, "sources": freq(3, 95)}
    if kind == "maps":
        return {"kind": kind, "freq": freq(2, 10), "ntheta": rng.randint(19, 121), "nphi": rng.randint(37, 241),
                "plane": rng.randint(11, 111)}
    if kind == "harmonic":
        return {"kind": kind, "freq": freq(2, 8), "precision": prec}
    return {"kind": kind, "freq": freq(3, 24), "precision": prec}


# ---- inputs ------------------------------------------------------------------

# Triangle rule of 13 points; the reference's single-precision literals.
_F = np.float32
QW = np.array([_F(-0.149570044467670)] + [_F(0.175615257433204)] * 3 + [_F(0.053347235608839)] * 3
              + [_F(0.077113760890257)] * 6, dtype=np.float64)
_a, _b, _c, _d = 0.333333333333333, 0.479308067841923, 0.260345966079038, 0.869739794195568
_e, _g, _h, _k = 0.065130102902216, 0.638444188569809, 0.312865496004875, 0.048690315425316
QN = np.array([[_a, _b, _c, _c, _d, _e, _e, _g, _g, _h, _h, _k, _k],
               [_a, _c, _c, _b, _e, _e, _d, _k, _h, _k, _g, _h, _g],
               [_a, _c, _b, _c, _e, _d, _e, _h, _k, _g, _k, _g, _h]], dtype=np.float32).astype(np.float64).T

# Physical constants with the reference's single-precision pi.
PI = float(np.float32(3.141592653589))
C0, EPS0, MU0, ETA0 = 2.997924580003e8, 8.8541878176e-12, 4 * PI * 1e-7, 3.767303134622e2


def split_triangle(corners, f):
    """Points and triangles of one flat triangle divided f times along each side."""
    idx, pts = {}, []
    for i in range(f + 1):
        for j in range(f + 1 - i):
            idx[i, j] = len(pts)
            pts.append(((f - i - j) * corners[0] + i * corners[1] + j * corners[2]) / f)
    tri = []
    for i in range(f):
        for j in range(f - i):
            tri.append((idx[i, j], idx[i + 1, j], idx[i, j + 1]))
            if i + j < f - 1:
                tri.append((idx[i + 1, j], idx[i + 1, j + 1], idx[i, j + 1]))
    return np.array(pts), np.array(tri)


def outward(nodes, faces):
    p = nodes[faces]
    flip = np.einsum("ij,ij->i", np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), p.sum(1)) < 0
    faces = faces.copy()
    faces[flip] = faces[flip][:, ::-1]
    return faces


def geodesic(f):
    """Unit sphere of 20 f^2 triangles: (nodes, faces), faces outward."""
    base, tri = meshgen.icosphere(0)
    pts, faces = [], []
    for t in tri:
        p, q = split_triangle(base[t], f)
        faces.append(q + sum(len(x) for x in pts))
        pts.append(p / np.linalg.norm(p, axis=1)[:, None])
    pts, faces = np.vstack(pts), np.vstack(faces)
    _, first, inv = np.unique(np.round(pts, 9) + 0.0, axis=0, return_index=True, return_inverse=True)
    nodes, faces = pts[first], inv.reshape(-1)[faces]
    return nodes, outward(nodes, faces)


def octant(f):
    """One eighth of the unit sphere, f^2 triangles, and the node pairs of its edges on each coordinate plane."""
    pts, faces = split_triangle(np.eye(3), f)
    nodes = pts / np.linalg.norm(pts, axis=1)[:, None]
    faces = outward(nodes, faces)
    pairs = np.unique(np.sort(np.vstack([faces[:, [0, 1]], faces[:, [1, 2]], faces[:, [2, 0]]]), axis=1), axis=0)
    lines = {ax: pairs[(nodes[pairs[:, 0], ax] == 0) & (nodes[pairs[:, 1], ax] == 0)] for ax in range(3)}
    return nodes, faces, lines


def shape(nodes, rng, scale=1.0):
    """A smooth seeded particle (nm): ellipsoid semi-axes and a small quadratic perturbation."""
    axes = rng.uniform(30.0, 70.0, 3) * scale
    q = rng.normal(0.0, 0.02, (3, 3))
    return nodes * axes * (1.0 + np.einsum("ni,ij,nj->n", nodes, q + q.T, nodes))[:, None]


def drude(wl):
    """Permittivity of a Drude metal (plasma 9.0 eV, damping 0.07 eV) at wavelength wl (m)."""
    w = 2 * math.pi * 2.99792458e8 / wl * 6.582119569e-16
    return 1.0 - 81.0 / (w * w + 0.07j * w)


def particle(case, seed, f=None):
    """Mesh (nm), ids, domains, wavelength (m), refractive indices and sources (degrees) of a case."""
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    wl = rng.uniform(480e-9, 800e-9)
    metal = np.sqrt(drude(wl) + 1e-3j)
    if kind in ("shell", "shell_gradient"):
        n1, f1 = geodesic(case["freq"])
        core = shape(n1, rng, 0.7)
        nodes = np.vstack([core, core * rng.uniform(1.4, 1.6)])
        faces = np.vstack([f1, f1 + len(n1)])
        ids = np.r_[np.full(len(f1), 1), np.full(len(f1), 2)]
        doms, ri = [[2], [-2, 1], [-1]], [1.0, metal, math.sqrt(2.13)]
    elif kind == "mirror":
        n1, faces, _ = octant(case["freq"])
        nodes = n1 * rng.uniform(30.0, 70.0, 3)
        ids, doms, ri = np.ones(len(faces), int), [[1], [-1]], [1.0, metal]
    else:
        n1, faces = geodesic(f or case["freq"])
        nodes = shape(n1, rng)
        ids, doms, ri = np.ones(len(faces), int), [[1], [-1]], [1.0, metal]
    srcs = []
    for _ in range(case.get("sources", 1)):
        th, ph, ps = math.degrees(math.acos(rng.uniform(-1, 1))), rng.uniform(0, 360), rng.uniform(0, 360)
        srcs.append((th, ph, ps))
    return {"nodes": nodes, "faces": faces, "ids": ids, "doms": doms, "wl": wl, "ri": ri, "srcs": srcs}


def freqs(case):
    """Frequencies of a sweep's particles: the largest, then smaller ones."""
    return [max(2, int(round(case["freq"] * r))) for r in (1.0, 0.5, 0.625, 0.75)][:case["particles"]]


def source(kind, s):
    if kind.startswith("shell"):  # elliptic polarisation of random phase
        return mom.src_pw_elliptic(s[0], s[1], complex(math.cos(s[2]), math.sin(s[2])))
    return mom.src_pw(*s)


def upload(p, lines=None):
    prob = mom.Problem.from_arrays(p["nodes"], p["faces"], p["ids"], 1e-9, p["doms"])
    solver = mom.Solver(0)
    if lines:
        prob.set_lines(np.vstack([lines[a] for a in range(3)]), np.concatenate([np.full(len(lines[a]), 11 + a)
                                                                               for a in range(3)]))
        for a, b in enumerate(("xplane", "yplane", "zplane")):
            prob.classify_edges(11 + a, b)
    solver.set_problem(prob)
    if lines:
        solver.set_symmetry(["mxp", "myp", "mzp"], prob)
    return solver


def currents(p):
    """Physical-optics currents of a plane wave on the edges: a solution's size and smoothness."""
    t = topology(p)
    cen = (p["nodes"] * 1e-9)[p["faces"]].mean(1)
    rng = np.random.default_rng(int(p["wl"] * 1e15) % (1 << 31))
    a, b = cen[t["plus"]], cen[t["minus"]]
    mid, tan = (a + b) / 2, (b - a) / np.linalg.norm(b - a, axis=1)[:, None]
    nrm = mid / np.linalg.norm(mid, axis=1)[:, None]
    d, e = np.linalg.qr(rng.normal(size=(3, 3)))[0][:2]
    ph = np.exp(2j * np.pi / p["wl"] * (mid @ d))[:, None]
    return np.concatenate([np.einsum("ni,ni->n", np.cross(nrm, ph * np.cross(d, e)) / ETA0, tan) * 2,
                           np.einsum("ni,ni->n", np.cross(ph * e, nrm), tan)])[:, None]


def plane_points(case):
    g = np.linspace(-150e-9, 150e-9, case["plane"])
    x, z = np.meshgrid(g, g, indexing="ij")
    return np.stack([x.ravel(), np.full(x.size, 3e-9), z.ravel()], axis=1)


def prepare(case, seed):
    kind = case["kind"]
    p = particle(case, seed)
    st = {"case": case, "p": p, "omega": mom.omega_of(p["wl"]), "ri": p["ri"],
          "src": [source(kind, s) for s in p["srcs"]]}
    if kind == "sweep":
        rng = np.random.default_rng([seed, 29])
        n, k = case["wavelengths"], case["contexts"]
        st["solvers"], st["om"], st["tab"] = [], [], []
        lam = spectrum(n, rng)
        for i, f in enumerate(freqs(case)):
            q = particle(case, seed + 1000 * i, f)
            for c in range(min(k, n)):
                mine = lam[c::k]
                st["solvers"].append(upload(q))
                st["om"].append([mom.omega_of(w) for w in mine])
                st["tab"].append([[1.0, np.sqrt(drude(w))] for w in mine])
        return st
    st["solver"] = upload(p, octant(case["freq"])[2] if kind == "mirror" else None)
    if kind == "maps":
        st["x"], st["pts"] = currents(p), plane_points(case)
    return st


def spectrum(n, rng):
    return np.linspace(400e-9, 900e-9, n) + rng.uniform(0, 5e-9)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    prec = PREC.get(case.get("precision"))
    om, ri, src = st["omega"], st["ri"], st["src"]
    if kind == "sweep":
        return [list(r) for r in mom.sweep_many(st["solvers"], st["om"], st["tab"], src, prec)]
    s = st["solver"]
    if kind in ("solve", "mirror"):
        x = s.solve_wavelength(om, ri, src, prec)
        return [x] + list(s.cross_sections(om, ri[0], src))
    if kind == "gradient":
        x = s.solve_wavelength(om, ri, src, prec)
        g = s.adjoint(om, ri, src, prec, eps_dom=1, nodes=case["nodes"])
        return [x, g["deps"]] + g.get("dnodes", [])
    if kind == "shell":
        s.solve_wavelength(om, ri, src, prec, want_host=False)
        return list(s.cross_sections(om, ri[0], src))
    if kind == "shell_gradient":
        s.solve_wavelength(om, ri, src, prec, want_host=False)
        return list(s.cross_sections(om, ri[0], src)) + [s.adjoint_mean_eps(om, ri, src, prec, 1)]
    if kind == "maps":
        far = s.rcs(om, ri[0], case["ntheta"], case["nphi"], x=st["x"])
        return [far] + list(s.scat_fields(om, ri[0], st["pts"], x=st["x"], srcs=src))
    s.solve_wavelength(om, ri, src, prec, want_host=False)
    x = s.shg_solve(om, ri, ri, [None, (1.0, 0.1 + 0.02j, -0.3)], prec)
    return [x] + list(s.cross_sections(2 * om, ri[0], [mom.src_none()]))


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    kind, f = case["kind"], case["freq"]

    def assembly(nf, images=1):  # far pairs once per unordered pair, both 3 x 3 blocks of each
        return images * (nf * nf / 2 * 169 * 88 + nf * nf * 3042)

    def solve(n, cols):
        return 8 / 3 * n ** 3 + 8.0 * n * n * cols

    faces, n, ns = 20 * f * f, 60 * f * f, case.get("sources", 1)
    io = 12.0 * faces + 12 * faces + 16 * n * ns
    if kind == "solve":
        fl = 2 * assembly(faces) + solve(n, ns)
    elif kind == "sweep":
        fl = case["wavelengths"] * sum(2 * assembly(20 * g * g) + solve(60 * g * g, 1) for g in freqs(case))
        io = sum(24.0 * 20 * g * g for g in freqs(case)) + 16 * case["wavelengths"] * case["particles"]
    elif kind == "gradient":
        # reverse mode of a face pair costs a few times its evaluation
        fl = 2 * assembly(faces) + solve(n, 3) + (6 if case["nodes"] else 2) * assembly(faces)
        io += 48.0 * faces
    elif kind == "shell":
        fl = 4 * assembly(faces) + 2 * faces * faces * 2 * 14872 / 2 + solve(2 * n, ns)
        io = 48.0 * faces + 56 * ns
    elif kind == "shell_gradient":
        fl = 8 * assembly(faces) + solve(2 * n, 3 * ns) + 8.0 * (2 * n) ** 2 * ns
        io = 48.0 * faces + 56 * ns
    elif kind == "maps":
        pts, dirs = case["plane"] ** 2, case["ntheta"] * case["nphi"]
        fl = pts * faces * 13 * 80.0 + dirs * faces * 13 * 60.0
        io += pts * (24 + 96) + dirs * 8
    elif kind == "harmonic":
        fl = 2 * (2 * assembly(faces) + solve(n, 1))
    else:
        nf = f * f
        n = 3 * f * (f + 1)
        fl = 2 * assembly(nf, 8) + 8 * solve(n, 1)
        io = 24.0 * nf + 8 * 16 * n
    return {"bytes": float(io), "flops": float(fl)}


# ---- the same results in plain 64-bit torch ----------------------------------

def topology(p):
    """Edges of the closed surfaces in order of first appearance; plus = the face that comes first."""
    faces = np.asarray(p["faces"])
    seen, plus, minus, fe = {}, [], [], np.zeros((len(faces), 3), int)
    for n, t in enumerate(faces.tolist()):
        for k in range(3):
            a, b = t[k], t[(k + 1) % 3]
            key = (a, b) if a < b else (b, a)
            if key in seen:
                minus[seen[key]] = n
            else:
                seen[key] = len(plus)
                plus.append(n)
                minus.append(-1)
            fe[n, k] = seen[key]
    return {"plus": np.array(plus), "minus": np.array(minus), "edge": fe, "n": len(plus)}


def dot(a, b):
    return (a * b).sum(-1)


def domains(p, dev):
    """Per domain: faces (inverted ones with their corners exchanged), signs and edges of their RWG halves."""
    t = topology(p)
    out, used = [], set()
    for d in p["doms"]:
        sel = np.nonzero(np.isin(p["ids"], np.abs(d)))[0]
        tri, ed = p["faces"][sel].copy(), t["edge"][sel].copy()
        sg = np.where(t["plus"][ed] == sel[:, None], 1.0, -1.0)
        for i, v in enumerate(p["ids"][sel]):
            if v in used:
                sg[i] = -sg[i]  # the second domain of a surface has the opposite orientation
            if -v in d:
                tri[i] = tri[i][::-1]
                ed[i] = ed[i][[1, 0, 2]]
                sg[i] = sg[i][[1, 0, 2]]
        used |= {abs(v) for v in d}
        out.append((torch.tensor(tri, device=dev), torch.tensor(ed, device=dev), torch.tensor(sg, device=dev)))
    return out, t["n"]


def geometry(x, dom):
    tri, ed, sg = dom
    v = x[tri]
    qn = torch.tensor(QN, device=x.device)
    q = qn[:, 2, None] * v[:, None, 0] + qn[:, 0, None] * v[:, None, 1] + qn[:, 1, None] * v[:, None, 2]
    nxt = v[:, [1, 2, 0]]
    ln = torch.linalg.norm(nxt - v, dim=-1)
    c = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    a2 = torch.linalg.norm(c, dim=-1)
    s = (nxt - v) / ln[..., None]
    m = torch.linalg.cross(s, (c / a2[:, None])[:, None].expand_as(s))
    return {"v": v, "q": q, "cp": v.mean(1), "area": a2 / 2, "n": c / a2[:, None], "s": s, "m": m, "sl": sg * ln,
            "free": v[:, [2, 0, 1]], "ed": ed, "len": ln}


def static_integrals(r, g):
    """Closed-form integrals over triangles g (one per row of r) at points r[..., 3]: of 1/R and R, of both
    times r', and of their gradients."""
    def ex(a):
        return a.unsqueeze(1)

    n, v = ex(g["n"]), g["v"]
    h = dot(n, r - ex(v[:, 0]))
    lm, l1, l3, tt, mm = [], [], [], [], []
    for e in range(3):
        p1, p2, s, m = ex(v[:, e]), ex(v[:, (e + 1) % 3]), ex(g["s"][:, e]), ex(g["m"][:, e])
        a, b = r - p2, r - p1
        rp, rm = torch.sqrt(dot(a, a)), torch.sqrt(dot(b, b))
        sp, sm = -dot(a, s), -dot(b, s)
        c = (rp - sp).abs() > (rm + sm).abs()
        lm.append(torch.log(torch.where(c, rm - sm, rp + sp) / torch.where(c, rp - sp, rm + sm)))
        t = dot(m, b)
        r02 = t * t + h * h
        l1.append(0.5 * r02 * lm[e] + 0.5 * (sp * rp - sm * rm))
        l3.append(0.75 * r02 * l1[e] + 0.25 * (sp * rp ** 3 - sm * rm ** 3))
        tt.append(t)
        mm.append(m)
    u = ex(v) - r.unsqueeze(2)
    u = u / torch.linalg.norm(u, dim=-1, keepdim=True)
    u0, u1, u2 = u[:, :, 0], u[:, :, 1], u[:, :, 2]
    y = dot(u0, torch.linalg.cross(u1, u2)).abs()
    om = 2 * torch.atan2(y, 1 + dot(u0, u1) + dot(u0, u2) + dot(u1, u2))
    om = torch.where(h > 0, om, -om)
    sm1 = -h * om - sum(t * x for t, x in zip(tt, lm))
    s1 = h * h / 3 * sm1 - sum(t * x for t, x in zip(tt, l1)) / 3
    ml1 = sum(m * x[..., None] for m, x in zip(mm, l1))
    ml3 = sum(m * x[..., None] for m, x in zip(mm, l3))
    gm1 = sum(m * x[..., None] for m, x in zip(mm, lm)) + n * om[..., None]
    g1 = ml1 - (h * sm1)[..., None] * n
    rho = r - h[..., None] * n - ex(g["cp"])
    return sm1, s1, ml1 + rho * sm1[..., None], ml3 / 3 + rho * s1[..., None], gm1, g1


def source_integrals(r, g, k, near):
    """Over every face n at points r (M, T, 3): int G, int G (r' - c_n), int grad'G; near (M, F) picks the
    faces whose singular part is taken in closed form."""
    w = torch.tensor(QW, device=r.device)
    d = r[:, :, None, None, :] - g["q"]
    r2 = dot(d, d)
    hit = r2 == 0
    R = torch.sqrt(torch.where(hit, torch.ones_like(r2), r2))
    e = torch.exp(1j * k * R)
    nr = near[:, None, :, None]
    G = torch.where(nr, (e - 1) / R + k * k * R / 2, e / R)
    P = e * (1 / R ** 3 - 1j * k / R ** 2)
    P = torch.where(nr, P - 1 / R ** 3 - k * k / (2 * R), P)
    zero = torch.zeros_like(G)
    G = torch.where(hit, torch.where(nr, 1j * k + zero, zero), G) * w
    P = torch.where(hit, zero, P) * w
    f = g["area"] / (4 * PI)
    i0 = G.sum(-1) * f
    qr = (g["q"] - g["cp"][:, None]).to(G.dtype)
    i1 = torch.einsum("mtfs,fsi->mtfi", G, qr) * f[:, None]
    ig = (P[..., None] * d).sum(-2) * f[:, None]
    mi, ni = torch.nonzero(near, as_tuple=True)
    if len(mi):
        st = static_integrals(r[mi], {a: g[a][ni] for a in ("v", "s", "m", "n", "cp")})
        f4, f8 = 1 / (4 * PI), k * k / (8 * PI)
        at = (mi[:, None], torch.arange(r.shape[1], device=r.device)[None], ni[:, None])
        i0 = i0.index_put(at, f4 * st[0] - f8 * st[1], accumulate=True)
        i1 = i1.index_put(at, f4 * st[2] - f8 * st[3], accumulate=True)
        ig = ig.index_put(at, f4 * st[4] - f8 * st[5], accumulate=True)
    return i0, i1, ig


def source_functions(r, g, ints):
    """int G div f_q, int G f_q, int grad'G x f_q for the three RWG halves of every face."""
    i0, i1, ig = ints
    c = g["sl"] / g["area"][:, None]
    k1 = c * i0[..., None]
    pq = g["free"] - g["cp"][:, None]
    k2 = c[..., None] / 2 * (i1[..., None, :] - pq * i0[..., None, None])
    rp = (r[:, :, None, None, :] - g["free"]).to(i0.dtype)
    k4 = -c[..., None] / 2 * torch.linalg.cross(rp, ig[..., None, :].expand_as(rp))
    return k1, k2, k4


def face_blocks(g, rows, k, c1, c2):
    """S = D + H and K of test faces `rows` against all faces: (M, 3, F, 3) each."""
    w = torch.tensor(QW, device=g["q"].device)
    r, cp = g["q"][rows], g["cp"].detach()
    ave = g["len"].detach().mean()
    dd = cp[rows][:, None] - cp
    near = dot(dd, dd) < (3 * ave) ** 2
    k1, k2, k4 = source_functions(r, g, source_integrals(r, g, k, near))
    sl = g["sl"][rows]
    fp = (sl[:, None, :, None] / 2 * (r[:, :, None] - g["free"][rows][:, None]) * w[:, None, None]).to(k2.dtype)
    dv = (sl[:, None, :] * w[:, None]).to(k2.dtype)
    S = c1 * torch.einsum("mtpi,mtfqi->mpfq", fp, k2) + c2 * torch.einsum("mtp,mtfq->mpfq", dv, k1)
    K = torch.einsum("mtpi,mtfqi->mpfq", fp, k4)
    self_ = torch.arange(len(cp), device=cp.device)[None] == rows[:, None]
    return S, torch.where(self_[:, None, :, None], torch.zeros_like(K), K)


def chunks(F, dev, most=3_000_000):
    per = max(1, most // (169 * F))
    return [torch.arange(i, min(F, i + per), device=dev) for i in range(0, F, per)]


def medium(eps, omega):
    return torch.sqrt(eps) * (omega / C0), -1j * omega * MU0, -1 / (1j * omega * EPS0 * eps), eps / ETA0 ** 2


def matrix(geo, N, omega, eps):
    dev = geo[0]["q"].device
    A = torch.zeros((2, 2, N, N), dtype=torch.complex128, device=dev)
    for g, e in zip(geo, eps):
        k, c1, c2, zs = medium(e, omega)
        ed = g["ed"].reshape(-1)
        for rows in chunks(len(g["cp"]), dev):
            er = g["ed"][rows].reshape(-1)
            for B, put in zip(face_blocks(g, rows, k, c1, c2), (((0, 0, 1.0), (1, 1, zs)), ((1, 0, 1.0), (0, 1, -1.0)))):
                cols = torch.zeros((len(er), N), dtype=B.dtype, device=dev)
                cols.index_add_(1, ed, B.reshape(len(er), len(ed)))
                for i, j, f in put:
                    A[i, j].index_add_(0, er, f * cols)
    return A.permute(0, 2, 1, 3).reshape(2 * N, 2 * N)


def incident(s, kind, k, omega, pts):
    th, ph, ps = s[0] * (PI / 180), s[1] * (PI / 180), s[2] * (PI / 180)
    if kind.startswith("shell"):
        ps = 0.0
    dev = pts.device
    di = torch.tensor([math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)], device=dev,
                      dtype=torch.float64)
    pol = np.array([math.cos(ps) * math.sin(ph) - math.sin(ps) * math.cos(th) * math.cos(ph),
                    -math.cos(ps) * math.cos(ph) - math.sin(ps) * math.cos(th) * math.sin(ph),
                    math.sin(ps) * math.sin(th)], dtype=complex)
    if kind.startswith("shell"):
        pol = pol + complex(math.cos(s[2]), math.sin(s[2])) * np.cross(di.cpu().numpy(), pol)
        pol = pol / np.linalg.norm(pol)
    e0 = torch.tensor(pol, device=dev)
    E = torch.exp(1j * k * (pts @ di))[..., None] * e0
    return E, k / (omega * MU0) * torch.linalg.cross(di.to(E.dtype).expand_as(E), E)


def half_functions(g):
    """f_p at the quadrature points, (F, 13, 3 functions, 3)."""
    return (g["sl"] / (2 * g["area"][:, None]))[:, None, :, None] * (g["q"][:, :, None] - g["free"][:, None])


def rhs(g, N, k, omega, s, kind):
    w = torch.tensor(QW, device=g["q"].device)
    E, H = incident(s, kind, k, omega, g["q"])
    f = (half_functions(g) * w[:, None, None] * g["area"][:, None, None, None]).to(E.dtype)
    out = [torch.zeros(N, dtype=E.dtype, device=E.device).index_add(0, g["ed"].reshape(-1), torch.einsum(
        "ftpi,fti->fp", f, v).reshape(-1)) for v in (E, H)]
    return torch.cat(out)


def sections(g, N, k, omega, s, kind, x, ri):
    """(scattering, absorption) cross sections from the currents x."""
    w = torch.tensor(QW, device=g["q"].device)
    n = g["n"][:, None]
    fn = torch.linalg.cross(n[:, :, None].expand(-1, 13, 3, -1), half_functions(g)).to(x.dtype)
    H = -torch.einsum("fp,ftpi->fti", x[:N][g["ed"]], fn)
    E = torch.einsum("fp,ftpi->fti", x[N:][g["ed"]], fn)
    Ei, Hi = incident(s, kind, k, omega, g["q"])
    nc = n.to(x.dtype)
    Es, Hs = (a - (b - nc * (nc * b).sum(-1, keepdim=True)) for a, b in ((E, Ei), (H, Hi)))
    flux = [(dot(torch.linalg.cross(a, b.conj()).real, n) * w).sum(1) * 0.5 for a, b in ((E, H), (Es, Hs))]
    cc = 2.0 / (EPS0 * C0 * ri)
    tot, sca = ((v * g["area"]).sum() * cc for v in flux)
    return sca, -tot


def far_map(g, N, k, ri, x, ntheta, nphi):
    dev = x.device
    w = torch.tensor(QW, device=dev)
    f = (half_functions(g) * w[:, None, None] * g["area"][:, None, None, None]).to(x.dtype)
    J, M = (torch.einsum("fp,ftpi->fti", v[g["ed"]], f).reshape(-1, 3) for v in (x[:N], x[N:]))
    th = (torch.arange(ntheta, device=dev, dtype=torch.float64) * PI / (ntheta - 1))[:, None]
    ph = (torch.arange(nphi, device=dev, dtype=torch.float64) * 2 * PI / (nphi - 1))[None]
    st, ct, sp, cp = th.sin(), th.cos(), ph.sin(), ph.cos()
    u = torch.stack([st * cp, st * sp, ct.expand(-1, nphi)], -1).reshape(-1, 3)
    ut = torch.stack([ct * cp, ct * sp, (-st).expand(-1, nphi)], -1).reshape(-1, 3).to(x.dtype)
    up = torch.stack([(-sp).expand(ntheta, -1), cp.expand(ntheta, -1), torch.zeros(ntheta, nphi, device=dev,
                     dtype=torch.float64)], -1).reshape(-1, 3).to(x.dtype)
    q = g["q"].reshape(-1, 3)
    out = []
    for a in range(0, len(u), 512):
        phase = torch.exp(-1j * k * (u[a:a + 512] @ q.T))
        nj, nm = phase @ J, phase @ M
        et = dot(nm, up[a:a + 512]) + ETA0 / ri * dot(nj, ut[a:a + 512])
        ep = dot(nm, ut[a:a + 512]) - ETA0 / ri * dot(nj, up[a:a + 512])
        pre = abs(complex(1j * k * torch.exp(1j * k) / (4 * PI)))
        out.append(pre ** 2 * (et.abs() ** 2 + ep.abs() ** 2))
    return torch.cat(out).reshape(ntheta, nphi)


def near_fields(g, N, k, omega, eps, x, pts):
    ave = g["len"].mean()
    c1, c2 = 1j * omega * MU0, 1 / (1j * omega * EPS0 * eps)
    E, H = [], []
    per = max(1, 3_000_000 // (13 * len(g["cp"])))
    for a in range(0, len(pts), per):
        r = pts[a:a + per, None]
        dd = r - g["cp"]
        near = dot(dd, dd) < (3 * ave) ** 2
        ints = source_integrals(r, g, k, near)
        _, k2, k4 = source_functions(r, g, ints)
        k3 = (g["sl"] / g["area"][:, None])[..., None] * ints[2][..., None, :]
        xj, xm = x[:N][g["ed"]], x[N:][g["ed"]]
        E.append(torch.einsum("fq,mtfqi->mi", xj, c1 * k2 + c2 * k3) + torch.einsum("fq,mtfqi->mi", xm, k4))
        H.append(torch.einsum("fq,mtfqi->mi", xm, k2 / c2 + k3 / c1) - torch.einsum("fq,mtfqi->mi", xj, k4))
    return torch.cat(E), torch.cat(H)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("harmonic", "mirror") or case["freq"] > (16 if kind == "solve" else 8):
        return None
    dev = torch.device("cuda")
    if kind == "sweep":
        rng = np.random.default_rng([seed, 29])
        lam, k, out = spectrum(case["wavelengths"], rng), case["contexts"], []
        src = particle(case, seed)["srcs"]
        for i, f in enumerate(freqs(case)):
            q = particle(case, seed + 1000 * i, f)
            for c in range(min(k, len(lam))):
                r = [solved(dict(q, wl=w, ri=[1.0, np.sqrt(drude(w))], srcs=src), kind, dev)[2:] for w in lam[c::k]]
                out.append([np.array([[float(v[j][0])] for v in r]) for j in range(2)])
        return out
    p = particle(case, seed)
    if kind == "maps":
        doms, N = domains(p, dev)
        g = geometry(torch.tensor(p["nodes"] * 1e-9, device=dev), doms[0])
        om, x, pts = mom_omega(p["wl"]), torch.tensor(currents(p)[:, 0], device=dev), torch.tensor(
            plane_points(case), device=dev)
        eps = torch.tensor(1.0 + 0j, dtype=torch.complex128, device=dev)
        k = medium(eps, om)[0]
        E, H = near_fields(g, N, k, om, eps, x, pts)
        Ei, Hi = incident(p["srcs"][0], kind, k, om, pts)
        return [far_map(g, N, k, 1.0, x, case["ntheta"], case["nphi"]).cpu().numpy(),
                (E + Ei)[None].cpu().numpy(), (H + Hi)[None].cpu().numpy()]
    grad = None
    if kind in ("gradient", "shell_gradient"):
        grad = case.get("nodes", False)
    X, cols, sca, ab, *g = solved(p, kind, dev, grad)
    sec = [torch.stack(v).detach().cpu().numpy() for v in (sca, ab)]
    x = X.cpu().numpy()
    if kind == "solve":
        return [x] + sec
    if kind == "gradient":
        return [x, g[0][None]] + [v[None] for v in g[1]]
    return sec if kind == "shell" else sec + [g[0]]


def mom_omega(wl):
    return 2.0 * PI * C0 / wl


def solved(p, kind, dev, grad=None):
    """Solutions and cross sections of a case; with grad, the mean gradients of (extinction, absorption) in the
    metal's permittivity, and (grad true) in every domain's node coordinates."""
    om = mom_omega(p["wl"])
    doms, N = domains(p, dev)
    base = torch.tensor(p["nodes"] * 1e-9, device=dev)
    eps = [torch.tensor(complex(r) ** 2, dtype=torch.complex128, device=dev) for r in p["ri"]]
    geo = [geometry(base, d) for d in doms]
    k0 = medium(eps[0], om)[0]
    A = matrix(geo, N, om, eps)
    Q = torch.stack([rhs(geo[0], N, k0, om, s, kind) for s in p["srcs"]], 1)
    lu, piv = torch.linalg.lu_factor(A)
    X = torch.linalg.lu_solve(lu, piv, Q)
    sec = [sections(geo[0], N, k0, om, s, kind, X[:, i], 1.0) for i, s in enumerate(p["srcs"])]
    out = [X, len(p["srcs"]), [s[0] for s in sec], [s[1] for s in sec]]
    if grad is None:
        return out
    S = len(p["srcs"])
    deps, dn = np.zeros((2, 2)), [[], []]
    W = []
    lam = []
    for o in range(2):
        G = []
        for i, s in enumerate(p["srcs"]):
            xv = X[:, i].clone().requires_grad_(True)
            sc, ab = sections(geo[0], N, k0, om, s, kind, xv, 1.0)
            (sc + ab if o == 0 else ab).backward()
            G.append(xv.grad.conj())
        L = torch.linalg.solve(A.T, torch.stack(G, 1))
        lam.append(L)
        W.append(L @ X.T / S)
    del A, lu
    er, ei = (v.clone().requires_grad_(True) for v in (eps[1].real, eps[1].imag))
    for d, dom in enumerate(doms):
        if d != 1 and not grad:
            continue
        xn = base.clone().requires_grad_(True)
        leaves = [er, ei, xn] if d == 1 else [xn]
        sums = [[0.0 for _ in leaves] for _ in range(2)]

        def add(o, value, more):
            for i, v in enumerate(torch.autograd.grad(value, leaves, retain_graph=more, allow_unused=True)):
                sums[o][i] = sums[o][i] + (0.0 if v is None else v)

        for rows in chunks(len(dom[0]), dev, 6_000_000):
            g = geometry(xn, dom)
            k, c1, c2, zs = medium(torch.complex(er, ei) if d == 1 else eps[d], om)
            Sb, Kb = (v.reshape(len(rows) * 3, -1) for v in face_blocks(g, rows, k, c1, c2))
            a, b = dom[1][rows].reshape(-1)[:, None], dom[1].reshape(-1)[None]
            for o in range(2):
                w = W[o].reshape(2, N, 2, N)
                add(o, -((w[0, a, 0, b] + zs * w[1, a, 1, b]) * Sb + (w[1, a, 0, b] - w[0, a, 1, b]) * Kb).sum().real,
                    o == 0)
        if grad and d == 0:
            for i, s in enumerate(p["srcs"]):
                for o in range(2):
                    g = geometry(xn, dom)
                    sc, ab = sections(g, N, k0, om, s, kind, X[:, i], 1.0)
                    v = (lam[o][:, i] * rhs(g, N, k0, om, s, kind)).sum().real + (sc + ab if o == 0 else ab)
                    add(o, v / S, False)
        for o in range(2):
            if d == 1:
                deps[o] = [float(sums[o][0]), float(sums[o][1])]
            dn[o].append(sums[o][-1])
    out.append(deps)
    if grad:
        out.append([np.stack([dn[o][d].cpu().numpy() for o in range(2)]) for d in range(len(doms))])
    return out
