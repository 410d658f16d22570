"""The complex128 LU part by part: where the real and the imaginary parts of
a matrix differ in size, each keeps the accuracy that fp64 operations give it
(csrc/lu_oz.cu)."""

import numpy as np
import pytest
from test_gpu_lu_panel import factor64

pytestmark = pytest.mark.gpu

U53 = 2.0**-53
TURNS = np.array([1, 1j, -1, -1j])


def matrix(kind, eps, n):
    """X + j eps Y, times j, with rows and columns turned by powers of j, or with Y = 0."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * (eps * rng.standard_normal((n, n)) if kind != "none" else 0.0)
    if kind != "real":
        A = 1j * A
    if kind in ("rows", "both"):
        A = TURNS[rng.integers(0, 4, n)][:, None] * A
    if kind in ("columns", "both"):
        A = A * TURNS[rng.integers(0, 4, n)][None, :]
    return A


@pytest.mark.parametrize("n", [69, 160, 193, 321])
@pytest.mark.parametrize("kind,eps", [(k, e) for k in ("real", "imaginary", "rows", "columns", "both")
                                      for e in (1e-6, 1e-12)] + [("none", 0.0)])
def test_parts_componentwise(gpu, kind, eps, n):
    from mom25d_gb300 import engine as E

    # multiplications by powers of j are exact, so that the small parts stay what they are
    A = matrix(kind, eps, n)
    F, ipiv = factor64(A)
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    P = A.copy()
    for i, p in enumerate(ipiv):
        P[[i, p]] = P[[p, i]]
    # gamma_n of the real products' magnitudes for each part (Higham, Accuracy and Stability of Numerical
    # Algorithms, theorem 9.3), twice for two products per part, twice for the multiplication by a reciprocal
    # pivot and twice for this product's own rounding
    re = P.real - (L.real @ U.real - L.imag @ U.imag)
    im = P.imag - (L.real @ U.imag + L.imag @ U.real)
    a, b, c, d = np.abs(L.real), np.abs(L.imag), np.abs(U.real), np.abs(U.imag)
    assert np.all(np.abs(re) <= 8 * n * U53 * (a @ c + b @ d))
    assert np.all(np.abs(im) <= 8 * n * U53 * (a @ d + b @ c))
    G, gpiv = factor64(A, E.M25_LU_NO_TENSOR_CORES)
    assert np.array_equal(F, G) and np.array_equal(ipiv, gpiv)


@pytest.mark.parametrize("eps", [1e-6, 1e-12])
def test_losses_of_a_solve(gpu, eps):
    """The small part of the solution of (j X + eps R) x = j b, -j eps X^-1 R X^-1 b in the first order, to the
    accuracy of an fp64 solve."""
    from mom25d_gb300.solver import dense_solve

    n = 256
    rng = np.random.default_rng(3)
    X = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    R = rng.standard_normal((n, n))
    b = rng.standard_normal((n, 2))
    x = dense_solve(eps * R + 1j * X, 1j * b, precision="fp64")
    # x = u + j v: X u + eps R v = b, X v = eps R u
    inv = np.linalg.inv(X)
    u = np.linalg.solve(X + eps**2 * R @ inv @ R, b)
    v = eps * np.linalg.solve(X, R @ u)
    # both parts of a backward stable solve: n ulps times the condition of X, below 10 by its diagonal
    assert np.abs(x.real - u).max() <= 100 * n * U53 * np.abs(u).max()
    assert np.abs(x.imag - v).max() <= 100 * n * U53 * np.abs(v).max()


def test_products_that_are_not_there(gpu):
    """The largest entries of a row of L and of a column of U at different inner indices, their product beyond the
    range of doubles: the sum has no term and C stays zero."""
    n = 84
    A = np.eye(n, dtype=complex)
    A[0, 64:83], A[64, 0], A[65:, 0] = 2.0**900, 0.5, 2.0**-600  # row 64 of L has its entry at 0
    A[1, 64:83], A[1, 83], A[65:, 1] = 2.0**-900, 1.0, 0.5       # column 83 of U at 1
    F, ipiv = factor64(A)
    assert np.array_equal(ipiv[:65], np.arange(65)) and F[64, 83] == 0.0
