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


@pytest.mark.parametrize("k", [-300, 0, 300])
def test_multipliers_of_a_scaled_column(k):
    """One column of multipliers a / z in an identity: x_0 = q_0 / z and x_i = q_i - (a_i / z) q_0."""
    s = problem(2)
    n = 2 * s.N
    rng = np.random.default_rng(7)
    z = np.ldexp(1.0, k) * (1.3 - 1.1j)
    A = np.eye(n, dtype=np.complex128)
    A[:, 0] = z * rng.uniform(-0.6, 0.6, n)
    A[1:, 0] += 1j * z * rng.uniform(-0.2, 0.2, n - 1)
    A[0, 0] = z
    q = s.srcvec(OM, RI[0], M.src_pw(0, 90, 0), want_host=True)[:, 0]
    s.set_matrix(A, M.FP64)
    x = s.solve(M.FP64)[:, 0]
    wide = np.clongdouble
    li, x0 = A[1:, 0].astype(wide) / wide(z), q[0].astype(wide) / wide(z)
    # the quotient (3 u per part), two complex products (sqrt(5) u each) and the sum: below 16 u each
    u = 2.0 ** -53
    assert abs(x[0] - x0) <= 16 * u * abs(x0)
    assert np.all(np.abs(x[1:] - (q[1:] - li * q[0])) <= 16 * u * (np.abs(li * q[0]) + np.abs(q[1:])))
    s.close()


@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
def test_interchanges_within_the_panel(prec):
    """Unitary diagonal blocks in a matrix that is tiny elsewhere: every panel's pivots lie among its own 64 rows,
    so no row leaves it (in a general matrix that is the last panel only), and every column left and right of it
    is interchanged within those rows."""
    s = problem(3)
    n = 2 * s.N
    rng = np.random.default_rng(11)
    A = 1e-6 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    for k in range(0, n, 64):
        g = rng.standard_normal((64, 64)) + 1j * rng.standard_normal((64, 64))
        A[k:k + 64, k:k + 64] = np.linalg.qr(g)[0]
    q = s.srcvec(OM, RI[0], M.src_pw(0, 90, 0), want_host=True)
    s.set_matrix(A, prec)
    x = s.solve(prec)
    eta = np.linalg.norm(A @ x - q) / (np.linalg.norm(A) * np.linalg.norm(x))
    assert eta <= (n * 2.0 ** -53 if prec == M.FP64 else 1e-12)
    s.close()


@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
def test_one_launch_panels_equal_single_subpanels(prec, monkeypatch):
    """A panel beside the update before it runs in one launch, whose subpanels exchange rows between CTAs; alone
    it runs as one launch per subpanel.  Both are backward stable, so the solutions differ by at most twice the
    bound of the backward error times the condition number."""
    rng = np.random.default_rng(5)
    xs = []
    for ahead in ("1", "0"):
        monkeypatch.setenv("MOM_LOOKAHEAD", ahead)
        s = problem(3)
        n = 2 * s.N
        if not xs:
            A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        q = s.srcvec(OM, RI[0], M.src_pw(0, 90, 0), want_host=True)
        s.set_matrix(A, prec)
        xs.append(s.solve(prec))
        bound = n * 2.0 ** -53 if prec == M.FP64 else 1e-12
        assert np.linalg.norm(A @ xs[-1] - q) <= bound * np.linalg.norm(A) * np.linalg.norm(xs[-1])
        s.close()
    cond = np.linalg.norm(A) * np.linalg.norm(np.linalg.inv(A))
    assert np.linalg.norm(xs[0] - xs[1]) <= 2 * bound * cond * np.linalg.norm(xs[1])


@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
def test_bounded_wait_of_the_cluster_panels(prec):
    """A limit of one poll runs out in the first wait for another CTA's message: the factorisation reports it,
    also in FP64, which has no residual check, and the same context solves again with the default limits."""
    s = problem(3)
    n = 2 * s.N
    rng = np.random.default_rng(3)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    q = s.srcvec(OM, RI[0], M.src_pw(0, 90, 0), want_host=True)
    for limit in (0, 1, 0):
        s.set_wait_limits(limit, 0, 0)
        s.set_matrix(A, prec)
        if limit:
            with pytest.raises(M.MomError) as e:
                s.solve(prec)
            assert e.value.status == M.MOM_ERR_TIMEOUT and "panel" in str(e.value)
            continue
        x = s.solve(prec)
        eta = np.linalg.norm(A @ x - q) / (np.linalg.norm(A) * np.linalg.norm(x))
        assert eta <= (n * 2.0 ** -53 if prec == M.FP64 else 1e-12)
    s.close()


@pytest.mark.parametrize("ns", [1, 70])
@pytest.mark.parametrize("exponent", [20, 40])
def test_rows_of_two_sizes(exponent, ns):
    """Half of the rows are 2^-exponent times the others: the mixed factorisation, before any refinement, solves
    a system whose rows differ from these by n 2^-24 of their own size (FP32 arithmetic throughout), and the
    small rows' part of an update is not lost where both kinds are pivots of one block."""
    s = problem(4)
    n = 2 * s.N
    rng = np.random.default_rng(9)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[rng.permutation(n)[:n // 2 + 29]] *= 2.0 ** -exponent
    srcs = W.incidences(ns)
    q = s.srcvec(OM, RI[0], srcs, want_host=True)
    s.set_matrix(A, M.MIXED)
    x = s.solve(M.MIXED, 1e30, 1)
    r = np.abs(A @ x - q)
    assert np.all(r <= n * 2.0 ** -24 * (np.abs(A) @ np.abs(x)))
    s.close()


@pytest.mark.parametrize("prec", [M.FP64, M.MIXED])
def test_panels_of_concurrent_contexts(prec):
    """Twelve contexts of one problem at once share the SMs, so the warps of a panel's CTA run far apart: every
    context gives the same cross sections, to the bit, each time."""
    ctx = [problem(3) for _ in range(12)]
    lam = np.linspace(500e-9, 800e-9, 6)
    om = [[M.omega_of(w) for w in lam]] * len(ctx)
    ri = [[RI] * len(lam)] * len(ctx)
    first = None
    for _ in range(8):
        out = M.sweep_many(ctx, om, ri, [M.src_pw(20, 30, 40)], prec)
        first = first or out[0]
        assert all(np.array_equal(a, b) for o in out for a, b in zip(o, first))
    for s in ctx:
        s.close()


def test_tallest_cluster_panels():
    s = problem(5)
    assert 2 * s.N == 24576
    s.solve_wavelength(OM, RI, [M.src_pw(0, 90, 0)], M.MIXED, want_host=False)  # raises unless refined to 1e-12
    assert s.iters <= 6
    s.close()
