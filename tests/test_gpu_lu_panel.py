"""LU factorisation on orders that reach every form of the cluster panel.

A panel's subpanels run with 1, 2, 4 or 8 rows per thread depending on their
height, so one factorisation passes through every form below its order: 384
(one row, ragged last CTA), 1,536, 6,144 (the forms above 4,096 rows) and, with
the tall forms of the mixed path, 24,576 (more than 16,384 rows).
"""
import numpy as np
import pytest

import mom_b200 as M
from mom_b200 import meshgen, workloads as W

pytestmark = pytest.mark.gpu

OM = M.omega_of(600e-9)
RI = [1.0, np.sqrt(W.EPS_AU)]


def problem(subdiv):
    nodes, faces = meshgen.octasphere(subdiv, 50.0)
    s = M.Solver(0)
    s.set_problem(M.Problem.from_arrays(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]]))
    return s


@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
@pytest.mark.parametrize("subdiv", [2, 3, 4])
@pytest.mark.parametrize("kind", ["gauss", "ties"])
def test_general_matrix(subdiv, prec, kind):
    s = problem(subdiv)
    n = 2 * s.N
    rng = np.random.default_rng(subdiv)
    if kind == "gauss":
        A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    else:  # entries of equal magnitude: every pivot search ties; a heavy permuted diagonal keeps it regular
        A = rng.choice([1.0, -1.0, 1j, -1j], (n, n)).astype(np.complex128)
        A[rng.permutation(n), np.arange(n)] *= 4.0 * n
    q = s.srcvec(OM, RI[0], M.src_pw(0, 90, 0), want_host=True)
    s.set_matrix(A, prec)
    x = s.solve(prec)
    # backward error: n eps in FP64 (a mixed solve is refined to ||r|| <= 1e-12 ||q|| <= 1e-12 ||A|| ||x||)
    eta = np.linalg.norm(A @ x - q) / (np.linalg.norm(A) * np.linalg.norm(x))
    assert eta <= (n * 2.0 ** -53 if prec == M.FP64 else 1e-12)
    s.close()


def test_tallest_cluster_panels():
    s = problem(5)
    assert 2 * s.N == 24576
    s.solve_wavelength(OM, RI, [M.src_pw(0, 90, 0)], M.MIXED, want_host=False)  # raises unless refined to 1e-12
    assert s.iters <= 6
    s.close()
