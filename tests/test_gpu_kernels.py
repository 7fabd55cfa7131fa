"""GPU unit tests of individual kernels (through the C ABI)."""
import numpy as np
import pytest

import mom_b200 as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(built):
    s = M.Solver(0)
    yield s
    s.close()


@pytest.mark.parametrize("m,nc,k", [(64, 100, 256), (320, 600, 64), (128, 256, 256), (192, 513, 128), (64, 64, 64),
                                    (1984, 192, 64)])
def test_tensor_core_update_matches_fp64(solver, m, nc, k):
    """The LU trailing update C -= L U on tcgen05 (3xTF32) is FP32-accurate:
    relative Frobenius error <= 1e-5 against the FP64 product of the same FP32
    inputs (a single TF32 pass would give ~1e-3)."""
    rng = np.random.default_rng(m + nc + k)
    cplx = lambda r, c: (rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))).astype(np.complex64)
    L, U, C = cplx(m, k), cplx(k, nc), cplx(m, nc)
    out = solver.selftest_cgemm(L, U, C)
    ref = C.astype(np.complex128) - L.astype(np.complex128) @ U.astype(np.complex128)
    err = np.linalg.norm(out - ref) / np.linalg.norm(ref)
    assert err <= 1e-5, err


def gaussian(rng, r, c):
    return (rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))).astype(np.complex64)


@pytest.mark.parametrize("m,nc,k", [(64, 100, 256), (320, 300, 64), (192, 513, 192), (1984, 192, 16)])
@pytest.mark.parametrize("rows,inner,cols", [(40, 0, 40), (0, 20, 0), (0, 60, 0), (30, 30, 30)])
def test_tensor_core_update_of_graded_operands(solver, m, nc, k, rows, inner, cols):
    """Rows of L, columns of U, and L's columns against U's rows, scaled by powers of two: the result is that of
    the operands without the scalings, so the same bound holds after they are undone."""
    rng = np.random.default_rng(m + nc + k)
    L, U, C = gaussian(rng, m, k), gaussian(rng, k, nc), gaussian(rng, m, nc)
    d1, d2 = (np.exp2(np.round(rng.uniform(-s, s, n))).astype(np.float32) for s, n in ((rows, m), (cols, nc)))
    di = np.exp2(np.round(rng.uniform(-inner / 2, inner / 2, k))).astype(np.float32)
    out = solver.selftest_cgemm(d1[:, None] * L / di, di[:, None] * U * d2, d1[:, None] * C * d2)
    ref = C.astype(np.complex128) - L.astype(np.complex128) @ U.astype(np.complex128)
    err = np.linalg.norm(out.astype(np.complex128) / d1[:, None] / d2 - ref) / np.linalg.norm(ref)
    assert err <= 1e-5, err


@pytest.mark.parametrize("m,nc,k", [(64, 100, 256), (320, 300, 64)])
def test_tensor_core_update_of_uneven_entries(solver, m, nc, k):
    """Entries of any size side by side, and rows and columns of zeros: the error of a column of the update is
    bounded by the largest entry of that column of |L| |U| (the bound of the even operands per term)."""
    rng = np.random.default_rng(k)
    L, U, C = gaussian(rng, m, k), gaussian(rng, k, nc), gaussian(rng, m, nc)
    L *= np.exp2(np.round(rng.uniform(-30, 0, L.shape))).astype(np.float32)
    U *= np.exp2(np.round(rng.uniform(-30, 0, U.shape))).astype(np.float32)
    L[5], L[:, 7], U[9], U[:, 11], C[:, 11] = 0, 0, 0, 0, 0
    out = solver.selftest_cgemm(L, U, C).astype(np.complex128)
    ref = C.astype(np.complex128) - L.astype(np.complex128) @ U.astype(np.complex128)
    size = (np.abs(L).astype(float) @ np.abs(U).astype(float)).max(0) + np.abs(C).max(0)
    assert np.all(np.abs(out - ref).max(0) <= 1e-5 * size)
    assert np.array_equal(out[5], C[5]) and not out[:, 11].any()


def test_tensor_core_update_of_non_finite_operands(solver):
    """Infinities and NaN stay in their rows (of L) and columns (of U)."""
    rng = np.random.default_rng(2)
    L, U, C = gaussian(rng, 128, 64), gaussian(rng, 64, 300), gaussian(rng, 128, 300)
    L[3, 5], L[70, 5], U[9, 7] = np.inf, np.nan, np.nan
    out = solver.selftest_cgemm(L, U, C).astype(np.complex128)
    bad = np.zeros(out.shape, bool)
    bad[[3, 70]], bad[:, 7] = True, True
    assert not np.isfinite(out[bad]).any() and np.isfinite(out[~bad]).all()
    L[[3, 70]], U[:, 7] = 0, 0
    ref = C.astype(np.complex128) - L.astype(np.complex128) @ U.astype(np.complex128)
    assert np.linalg.norm((out - ref)[~bad]) <= 1e-5 * np.linalg.norm(ref[~bad])
