"""Sweeps over eight contexts at once (factorisation on one stream each) against
each context's own sweep, before and after."""
import numpy as np
import pytest

import mom_b200 as M
from mom_b200 import meshgen, workloads as W

pytestmark = pytest.mark.gpu

WLS = np.array([420e-9, 650e-9])
SRC = [M.src_pw(0, 90, 0)]


@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
@pytest.mark.parametrize("sub", [1, 2])
def test_eight_contexts(sub, prec):
    oms = np.array([M.omega_of(w) for w in WLS])
    ri = np.stack([np.ones(len(WLS)), np.sqrt(W.drude_eps(WLS))], axis=1)
    solvers = []
    for k in range(8):
        nodes, faces = meshgen.octasphere(sub, 40.0 + k)
        s = M.Solver(0)
        s.set_problem(M.Problem.from_arrays(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]]))
        solvers.append(s)
    before = [s.sweep(oms, ri, SRC, prec)[:2] for s in solvers]
    many = M.sweep_many(solvers, [oms] * 8, [ri] * 8, SRC, prec)
    after = [s.sweep(oms, ri, SRC, prec)[:2] for s in solvers]
    for b, m, a in zip(before, many, after):
        for i in (0, 1):
            assert np.allclose(m[i], b[i], rtol=1e-9, atol=0)  # another order of the updates
            assert np.array_equal(a[i], b[i])
    for s in solvers:
        s.close()
