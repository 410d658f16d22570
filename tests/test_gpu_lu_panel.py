"""The LU's panel (csrc/lu_panel.cu): orders at the edges of its strips,
blocks and clusters against LAPACK's pivots and the backward error bound."""

import ctypes as C

import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 63, 65, 127, 129, 257, 513, 1025, 2049])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_panel_edges(gpu, n, dtype):
    from mom25d_gb300 import engine as E

    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).astype(dtype)
    if n > 40:
        A[11] = A[5]  # equal candidates: the first row wins
        A[:, 30] = 0  # a column without a pivot until the updates fill it
    double = dtype == np.complex128
    ctx = E.Context(0)
    ld = n if double else n + (n & 1)
    F = np.zeros((n, ld), dtype)
    F[:, :n] = A
    ipiv, info = np.zeros(n, np.int32), np.zeros(1, np.int32)
    E.check(ctx.lib.m25_lu_factor(ctx.h, n, E.M25_FP64 if double else E.M25_MIXED, F.ctypes.data, ld,
                                  E.ptr(ipiv, C.c_int32), E.M25_ON_HOST, 0, E.ptr(info, C.c_int32)))
    ctx.close()
    LU = F[:, :n].astype(np.complex128)
    L, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    P = A.astype(np.complex128)
    for i, p in enumerate(ipiv):
        assert i <= p < n
        P[[i, p]] = P[[p, i]]
    # |P A - L U| <= gamma_n |L| |U| (Higham, Accuracy and Stability of Numerical Algorithms, theorem 9.3), the
    # constant doubled twice for complex arithmetic; complex64 in 3xTF32 rounds products at 2^-22
    u = 2.0**-53 if double else 2.0**-22
    assert np.all(np.abs(P - L @ U) <= 4 * n * u * (np.abs(L) @ np.abs(U)) + 1e-300)
    # izamax compares |re| + |im|: multipliers are at most sqrt 2 in modulus
    assert np.abs(L).max() <= np.sqrt(2) * (1 + 8 * u)
    if double and n <= 40:  # no ties, no empty column: LAPACK's own pivots
        assert np.array_equal(ipiv, sl.lu_factor(A)[1])
