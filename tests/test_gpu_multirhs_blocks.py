"""Many-right-hand-side solves at orders whose last 256-row block has one, two
or four 64-row steps and at column counts that leave the last CTA partly empty,
against the single-column solve; A x = b, and A^T x = b through the adjoint."""
import numpy as np
import pytest

import mom_b200 as M
from mom_b200 import meshgen, workloads as W

pytestmark = pytest.mark.gpu

OM = M.omega_of(600e-9)
RI = [1.0, np.sqrt(W.EPS_AU)]
MESHES = {64: (meshgen.icosphere, 0), 128: (meshgen.octasphere, 1), 256: (meshgen.icosphere, 1),
          384: (meshgen.octasphere, 2)}


@pytest.mark.parametrize("ns", [17, 66])
@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
@pytest.mark.parametrize("n", sorted(MESHES))
def test_last_block(n, prec, ns):
    make, s = MESHES[n]
    nodes, faces = make(s, 50.0)
    sol = M.Solver(0)
    sol.set_problem(M.Problem.from_arrays(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]]))
    assert -(-2 * sol.N // 64) * 64 == n
    srcs = W.incidences(ns)
    X = sol.solve_wavelength(OM, RI, srcs, prec, 1e-12, 30, want_host=True)
    mean = sol.adjoint_mean_eps(OM, RI, srcs, prec, eps_dom=1)  # 2 ns adjoint columns
    per = []
    for k in range(ns):
        x1 = sol.solve_wavelength(OM, RI, [srcs[k]], prec, 1e-12, 30, want_host=True)[:, 0]
        # condition of the small sphere systems times the rounding (or the refined residual)
        assert np.linalg.norm(X[:, k] - x1) <= (1e-12 if prec == M.FP64 else 1e-10) * np.linalg.norm(x1)
        per.append(sol.adjoint(OM, RI, [srcs[k]], prec, eps_dom=1)["deps"][0])
    assert np.allclose(np.mean(per, axis=0), mean, rtol=1e-8, atol=0)
    sol.close()
