"""Several representations of an order at which the mixed path factorises them
one by one: the quarter of a sphere of 24,576 unknowns."""
import numpy as np
import pytest

import mom_b200 as M
from mom_b200 import meshgen

pytestmark = pytest.mark.gpu


def test_large_mixed_representations(built):
    nodes, faces = meshgen.octasphere(5, 50.0)
    fn, ff, lines = meshgen.symmetry_fragment(nodes, faces, [0, 1])
    p = M.Problem.from_arrays(fn, ff, np.ones(len(ff), int), 1e-9, [[1], [-1]])
    p.set_lines(np.concatenate([np.asarray(lines[ax], np.int32).reshape(-1, 2) for ax in (0, 1)]),
                np.concatenate([np.full(len(lines[ax]), 10 + ax, np.int32) for ax in (0, 1)]))
    for ax, name in enumerate(("xplane", "yplane")):
        p.classify_edges(10 + ax, name)
    s = M.Solver(0)
    s.set_problem(p)
    s.set_symmetry(["mxp", "myp"], p)
    n = 2 * s.N
    assert 4608 <= n < 8192
    om, ri = M.omega_of(600e-9), [1.0, np.sqrt(complex(-9, 1.3))]
    srcs = [M.src_pw(20, 40, 10), M.src_pw_elliptic(60, 200, 1j)]
    sig = {}
    for prec in (M.FP64, M.MIXED):
        f0 = s.tensor_flops
        s.solve_wavelength(om, ri, srcs, prec, want_host=False)
        # the updates of four factorisations: 8/3 n^3 real operations each, three tensor-core passes,
        # at least half of them in updates wide enough for the tensor cores
        assert (s.tensor_flops - f0 >= 4 * 4 * n ** 3) == (prec == M.MIXED)
        sig[prec] = np.concatenate(s.cross_sections(om, ri[0], srcs))
    assert np.abs(sig[M.MIXED] - sig[M.FP64]).max() <= 1e-6 * np.abs(sig[M.FP64]).min()
    s.close()


def test_memory_of_a_group(built):
    """Setting a group takes the memory of its matrices and, for the blocks of several actions at once, 1 GiB at most."""
    import torch
    nodes, faces = meshgen.octasphere(5, 50.0)
    fn, ff, lines = meshgen.symmetry_fragment(nodes, faces, [0, 1])
    p = M.Problem.from_arrays(fn, ff, np.ones(len(ff), int), 1e-9, [[1], [-1]])
    p.set_lines(np.concatenate([np.asarray(lines[ax], np.int32).reshape(-1, 2) for ax in (0, 1)]),
                np.concatenate([np.full(len(lines[ax]), 10 + ax, np.int32) for ax in (0, 1)]))
    for ax, name in enumerate(("xplane", "yplane")):
        p.classify_edges(10 + ax, name)
    s = M.Solver(0)
    s.set_problem(p)
    before = torch.cuda.mem_get_info()[0]
    s.set_symmetry(["mxp", "myp"], p)
    taken = before - torch.cuda.mem_get_info()[0]
    n = -(-2 * s.N // 64) * 64
    # three more matrices and diagonal inverses; mapped geometry and near pairs of three actions and two domains
    # (432 bytes of closed forms per pair, at most 100 pairs per face)
    assert taken <= 3 * 16 * n * (n + 128) + 6 * 440 * 100 * len(ff) + (1 << 30)
    s.close()
