"""Near fields far away: the K4 integrals (M in E, J in H) from 1 um to 10 cm off a
sphere of 320 faces against sums in extended precision.

At a wavelength of 1 mm the phase is known to the rounding of the distance, so
the distance over the face's size (up to 7e6 here) is the largest ratio in the
problem, and no error may grow with it.  Bound per component, relative to the
sum of the terms' magnitudes, in units of 2^-53: 100 for a term, one per term
for the summation, 8 kL for the phase.
"""
import numpy as np
import pytest

import mom_b200 as M
from mom_b200 import meshgen

pytestmark = pytest.mark.gpu

PI = float(np.float32(3.141592653589))  # the library's
C0 = 2.997924580003e8
L, C = np.longdouble, np.clongdouble


def cross_integral(D, x, k, r):
    """sum_f int grad'G x (current of x) at r, and the sum of its terms' magnitudes."""
    nodes, fn, fe = D["nodes"].astype(L), D["face_node"], D["face_edge"]
    w, q = M.tri_rule()
    p = nodes[fn]
    cen = p.mean(1)
    rho = np.einsum("qk,fki->fqi", q.astype(L)[:, [2, 0, 1]], p) - cen[:, None]
    a, b = np.zeros(len(fn), C), np.zeros((len(fn), 3), C)
    for e in range(3):
        edge = fe[:, e]
        side = np.where(D["edge_face"][edge, 0] == np.arange(len(fn)), 0, 1)
        ends = nodes[D["edge_node"][edge]]
        v = x[D["edge_parent"][edge]] * np.sqrt(((ends[:, 0] - ends[:, 1]) ** 2).sum(1)) * np.where(side, -1, 1) / 2
        a += v
        b -= v[:, None] * (nodes[D["edge_bnode"][edge, side]] - cen)
    d = r.astype(L) - cen[:, None] - rho
    R = np.sqrt((d ** 2).sum(-1))
    phi = w.astype(L) * np.exp(1j * C(k) * R) * (1 / R ** 3 - 1j * C(k) / R ** 2) / (4 * L(PI))
    out = (phi[..., None] * np.cross(d.astype(C), a[:, None, None] * rho + b[:, None])).sum((0, 1))
    size = np.abs(a)[:, None] * np.sqrt((rho ** 2).sum(-1)) + np.sqrt((np.abs(b) ** 2).sum(-1))[:, None]
    return out, (np.abs(phi) * R * size).sum()


@pytest.mark.parametrize("dist", [1e-6, 1e-4, 1e-2, 1e-1])
def test_cross_terms_far_away(built, dist):
    nodes, faces = meshgen.icosphere(2, 50.0)
    p = M.Problem.from_arrays(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]])
    s = M.Solver(0)
    s.set_problem(p)
    om = M.omega_of(1e-3)
    k = om / C0
    rng = np.random.default_rng(0)
    x = rng.standard_normal(s.N) + 1j * rng.standard_normal(s.N)
    pts = rng.standard_normal((3, 3))
    pts *= dist / np.linalg.norm(pts, axis=1)[:, None]
    z = np.zeros(s.N)
    e = s.scat_fields(om, 1.0, pts, x=np.r_[z, x][:, None])[0][0]  # M only: E = K4
    h = s.scat_fields(om, 1.0, pts, x=np.r_[x, z][:, None])[1][0]  # J only: H = -K4
    D = p.domain(0)
    bound = (100 + 13 * len(D["face_node"]) + 8 * k * dist) * 2.0 ** -53
    for i, r in enumerate(pts):
        f, size = cross_integral(D, x, k, r)
        assert np.abs(e[i] - f).max() <= bound * size
        assert np.abs(h[i] + f).max() <= bound * size
    s.close()


@pytest.mark.parametrize("subdiv", [0, 1, 2])
@pytest.mark.parametrize("ns", [1, 3, 9])
def test_splits_of_the_faces(built, subdiv, ns):
    """The faces are split according to the number of points: one, a few and thousands give the same fields."""
    nodes, faces = meshgen.icosphere(subdiv, 50.0)
    s = M.Solver(0)
    s.set_problem(M.Problem.from_arrays(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]]))
    om = M.omega_of(600e-9)
    rng = np.random.default_rng(1)
    x = rng.standard_normal((2 * s.N, ns)) + 1j * rng.standard_normal((2 * s.N, ns))
    pts = rng.uniform(-1.5e-7, 1.5e-7, (20000, 3))
    whole = s.scat_fields(om, 1.0, pts, x=x)
    # sums of 13 points per face in another order; terms up to 100 times the sum
    tol = 100 * 13 * len(faces) * 2.0 ** -53
    for n in (1, 129, 2500):
        for a, b in zip(s.scat_fields(om, 1.0, pts[:n], x=x), whole):
            assert np.abs(a - b[:, :n]).max() <= tol * np.abs(b[:, :n]).max()
    s.close()
