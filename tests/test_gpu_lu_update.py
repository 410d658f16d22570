"""The complex128 LU's trailing update (csrc/lu_oz.cu) where the largest
entries of a row of L and of a column of U meet no entry of their size: the
componentwise bounds of an fp64 factorisation and solve hold there too."""

import numpy as np
import pytest
from test_gpu_lu_panel import factor64

pytestmark = pytest.mark.gpu

U53 = 2.0**-53


def complex_normal(rng, n):
    return rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))


def matrix(kind, n):
    rng = np.random.default_rng(n)
    A = complex_normal(rng, n)
    if kind.startswith("groups"):  # two interleaved groups of unknowns, weakly coupled
        i = np.arange(n)
        A[(i[:, None] + i[None, :]) % 2 == 1] *= float(kind[6:])
    elif kind.startswith("tiny"):  # columns of L of which all but a few rows are small, their neighbours not
        A[:64, :64] += 30 * np.eye(64)
        A[68:, :32] *= float(kind[4:])
    elif kind == "sparse":  # rows and columns without a common inner index, and some with one
        A[64:, 0:64:2] *= rng.uniform(size=(n - 64, 32)) < 0.1
        A[0:64, 64:] *= rng.uniform(size=(64, n - 64)) < 0.1
        A[:64, :64] = 8 * np.diag(rng.uniform(1, 2, 64))
    elif kind == "subnormal":  # the last column below the normal range
        A[:, -1] *= 2.0**-1040
    return A


KINDS = ["groups1e-4", "groups1e-8", "groups1e-12", "tiny1e-12", "tiny1e-16", "tiny1e-30", "sparse"]


@pytest.mark.parametrize("n", [69, 97, 160, 193, 321])  # beside tiles of 128 rows and 32 columns, and whole ones
@pytest.mark.parametrize("kind,transposed", [(k, t) for k in KINDS for t in (False, True)] + [("subnormal", False)])
def test_update_componentwise(gpu, kind, transposed, n):
    from mom25d_gb300 import engine as E

    A = matrix(kind, n)
    if transposed:
        A = np.ascontiguousarray(A.T)
    F, ipiv = factor64(A)
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    P = A.copy()
    for i, p in enumerate(ipiv):
        P[[i, p]] = P[[p, i]]
    # gamma_n |L| |U|, twice for complex arithmetic and twice for this product's own rounding; a product below the
    # normal range is off by half the smallest number in each of its four parts, here and in the factorisation
    assert np.all(np.abs(P - L @ U) <= 4 * n * U53 * (np.abs(L) @ np.abs(U)) + 4 * n * 2.0**-1074)
    G, gpiv = factor64(A, E.M25_LU_NO_TENSOR_CORES)
    assert np.array_equal(F, G) and np.array_equal(ipiv, gpiv)


@pytest.mark.parametrize("eps", [1e-4, 1e-8, 1e-12])
def test_solve_of_weakly_coupled_groups(gpu, eps):
    """The currents that one group induces in the other, eps of its own, to
    the accuracy that a componentwise backward stable LU gives them."""
    import scipy.linalg as sl

    from mom25d_gb300.solver import dense_solve

    n = 256
    A = matrix(f"groups{eps:g}", n)
    B = np.zeros((n, 1), complex)
    B[0::2, 0] = 1.0
    X = dense_solve(A, B, precision="fp64")
    # the exact solution by refinement in extended precision
    lu = sl.lu_factor(A)
    ref = np.zeros((n, 1), np.clongdouble)
    for _ in range(6):
        ref = ref + sl.lu_solve(lu, (B - A.astype(np.clongdouble) @ ref).astype(complex))
    # |A + E| x = b with |E| <= 3 gamma_n |L| |U| (Higham, Accuracy and Stability of Numerical Algorithms, theorem
    # 9.4), twice for complex arithmetic
    p, L, U = sl.lu(A)
    bound = 6 * n * U53 * (np.abs(np.linalg.inv(A)) @ (p @ (np.abs(L) @ np.abs(U))) @ np.abs(ref).astype(float))
    assert np.all(np.abs(X - ref) <= bound)
    assert np.abs(X[1::2]).max() <= 100 * eps * np.abs(X[0::2]).max()
