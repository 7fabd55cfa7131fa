"""Gradients for several sources at once: the same values as the all-dual
kernel gives (MOM_ADJ_*_PLAIN=0), for every quadrature rule, and no launch more
than for one source."""
import numpy as np
import pytest

import mom_b200 as M
from mom_b200 import meshgen, workloads as W

pytestmark = pytest.mark.gpu

OM = M.omega_of(600e-9)
RI = [1.0, np.sqrt(W.EPS_AU)]
SRCS = [M.src_pw(0, 90, 0), M.src_pw_elliptic(50, 20, 1j), M.src_pw(75, 300, 20), M.src_pw(120, 250, 60)]


def solved(subdiv, quad, ns):
    nodes, faces = meshgen.icosphere(subdiv, 50.0)
    s = M.Solver(0)
    s.set_problem(M.Problem.from_arrays(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]]), quad)
    s.solve_wavelength(OM, RI, SRCS[:ns], M.FP64, want_host=False)
    return s


def close(a, b):
    # both kernels sum the same FP64 terms, up to 4e6 of them, in other orders
    return np.abs(np.asarray(a) - np.asarray(b)).max() <= 1e-11 * np.abs(b).max()


@pytest.mark.parametrize("subdiv,quad,ns", [(0, "tri_gl1", 1), (0, "tri_gl13", 4), (1, "tri_gl3", 3), (2, "tri_gl4", 2),
                                            (2, "tri_gl7", 4), (2, "tri_gl13", 3)])
def test_eps_gradient_of_several_sources(subdiv, quad, ns, monkeypatch):
    out = []
    for plain in ("1", "0"):
        monkeypatch.setenv("MOM_ADJ_EPS_PLAIN", plain)
        s = solved(subdiv, quad, ns)
        out.append((s.adjoint(OM, RI, SRCS[:ns], M.FP64, eps_dom=1)["deps"],
                    s.adjoint_mean_eps(OM, RI, SRCS[:ns], M.FP64, 1)))
        s.close()
    for a, b in zip(*out):
        assert close(a, b)


def launches(ns, **kw):
    """Launches of the gradients asked for, beyond those of the adjoint solve."""
    s = solved(1, "tri_gl13", ns)
    n = [s.launch_count]
    for args in ({}, kw, {}, kw):  # the second of each: all buffers there
        s.adjoint(OM, RI, SRCS[:ns], M.FP64, **args)
        n.append(s.launch_count)
    s.close()
    return (n[4] - n[3]) - (n[3] - n[2])


def test_eps_gradient_launches():
    assert launches(4, eps_dom=1) == launches(1, eps_dom=1)


@pytest.mark.parametrize("subdiv,quad,ns", [(0, "tri_gl1", 1), (0, "tri_gl13", 4), (1, "tri_gl3", 3), (2, "tri_gl4", 2),
                                            (1, "tri_gl7", 4), (2, "tri_gl13", 3)])
def test_vertex_gradient_of_several_sources(subdiv, quad, ns, monkeypatch):
    out = []
    for plain in ("1", "0"):
        monkeypatch.setenv("MOM_ADJ_VERTEX_PLAIN", plain)
        s = solved(subdiv, quad, ns)
        out.append(s.adjoint(OM, RI, SRCS[:ns], M.FP64, nodes=True)["dnodes"])
        s.close()
    for a, b in zip(*out):
        for k in range(ns):
            assert close(a[k], b[k])


def test_vertex_gradient_launches():
    """Three more sources cost two small launches per source and domain, which prepare their currents."""
    assert launches(4, nodes=True) - launches(1, nodes=True) <= 3 * 2 * 2
