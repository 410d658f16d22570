"""The LU's tall panel (panel_kernel in csrc/lu.cu, a cooperative grid),
which factors the columns with more rows than one cluster holds: by itself
at small orders, in a process without cluster panels, and before them at
an order above the limit."""

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def factors(A, flags=0):
    """m25_lu_factor of a host matrix: the factors in place and the interchanges."""
    from mom25d_gb300 import engine as E

    n, double = A.shape[0], A.dtype == np.complex128
    ld = n if double else n + (n & 1)
    F = np.zeros((n, ld), A.dtype)
    F[:, :n] = A
    ipiv, info = np.zeros(n, np.int32), np.zeros(1, np.int32)
    ctx = E.Context(0)
    E.check(ctx.lib.m25_lu_factor(ctx.h, n, E.M25_FP64 if double else E.M25_MIXED, F.ctypes.data, ld,
                                  E.ptr(ipiv, C.c_int32), E.M25_ON_HOST, flags, E.ptr(info, C.c_int32)))
    ctx.close()
    return F[:, :n], ipiv


def check(A, F, ipiv):
    """|P A - L U| <= gamma_n |L| |U| (Higham, Accuracy and Stability of
    Numerical Algorithms, theorem 9.3), the constant doubled twice for complex
    arithmetic; complex64 in 3xTF32 rounds products at 2^-22. Applied to
    vectors of +-1 where the order is too large for the product itself."""
    n = len(A)
    u = 2.0**-53 if A.dtype == np.complex128 else 2.0**-22
    perm = np.arange(n)
    for i, p in enumerate(ipiv):
        assert i <= p < n
        perm[[i, p]] = perm[[p, i]]
    if n <= 1100:
        LU = F.astype(np.complex128)
        L, U, P = np.tril(LU, -1) + np.eye(n), np.triu(LU), A.astype(np.complex128)[perm]
        assert np.all(np.abs(P - L @ U) <= 4 * n * u * (np.abs(L) @ np.abs(U)) + 1e-300)
        assert np.abs(L).max() <= np.sqrt(2) * (1 + 8 * u)
        return
    X = np.random.default_rng(0).choice((-1.0, 1.0), (n, 3)).astype(np.complex128)
    mag = np.ones((n, 1))
    Y, Ym, AX = np.zeros_like(X), np.zeros_like(mag), np.zeros_like(X)
    for r in range(0, n, 512):  # by rows: no second matrix of the same size
        s = slice(r, min(n, r + 512))
        U = np.triu(F[s], r).astype(np.complex128)
        Y[s], Ym[s] = U @ X, np.abs(U) @ mag
        AX[s] = A[perm[s]].astype(np.complex128) @ X
    for r in range(0, n, 512):
        s = slice(r, min(n, r + 512))
        L = np.tril(F[s], r - 1).astype(np.complex128)
        res = np.abs(AX[s] - (L @ Y + Y[s]))
        # the sums above round too: n u |L| (|U| |x|) each, in fp64
        assert np.all(res <= 4 * n * (u + 2.0**-53) * (np.abs(L) @ Ym + Ym[s]))


def matrix(n, dtype):
    rng = np.random.default_rng(n)
    A = np.empty((n, n), dtype)
    for r in range(n):
        A[r] = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    if n > 40:
        A[11] = A[5]  # equal candidates: the first row wins
        A[:, 30] = 0  # a column without a pivot until the updates fill it
    return A


ORDERS = [1, 2, 31, 63, 64, 65, 127, 128, 129, 193, 255, 257, 385, 513]


def test_tall_panels_alone(gpu):
    """The same orders and types as the cluster panel, in a process that has none."""
    code = ("import sys; sys.path[:0] = %r\n"
            "import numpy as np\n"
            "import test_gpu_lu_paths as T\n"
            "for dt in (np.complex128, np.complex64):\n"
            "    for n in T.ORDERS:\n"
            "        A = T.matrix(n, dt)\n"
            "        T.check(A, *T.factors(A))\n"
            "print('all orders')\n" % ([os.path.dirname(__file__), os.path.dirname(os.path.dirname(__file__))],))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, M25_NO_CLUSTER_PANEL="1"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "all orders" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_tall_panels_before_cluster_panels(gpu, dtype):
    """One order above the 8192 rows of a cluster: tall panels first, the cluster's from then on."""
    A = matrix(8192 + 200, dtype)
    check(A, *factors(A))
