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


def factor64(A, flags=0):
    from mom25d_gb300 import engine as E

    n = A.shape[0]
    ctx = E.Context(0)
    F, ipiv, info = np.array(A, np.complex128), np.zeros(n, np.int32), np.zeros(1, np.int32)
    E.check(ctx.lib.m25_lu_factor(ctx.h, n, E.M25_FP64, F.ctypes.data, n, E.ptr(ipiv, C.c_int32), E.M25_ON_HOST, flags,
                                  E.ptr(info, C.c_int32)))
    ctx.close()
    return F, ipiv


@pytest.mark.parametrize("bits", [0x7F7F7F7F7F7F7C, 0x40404040404040, 0x7F80807F80807C])
@pytest.mark.parametrize("scale", [1.0, 2.0**-340, 2.0**300])
def test_update_slices_are_exact(gpu, bits, scale):
    """The complex128 update by integer slices (csrc/lu_oz.cu): one entry
    c - sum l u of 128 products whose digits are all as large as they get
    (0x7F.. every digit 127: the accumulators' largest sums), against exact
    rational arithmetic."""
    from fractions import Fraction

    x = bits / 2.0**55
    A = np.zeros((65, 65), complex)
    A[:64, :64] = 4 * np.eye(64)     # pivots, above |re| + |im| of the row below
    A[64, :64] = x - 1j * x          # a row of A: (re, -im) = (x, x) / 4
    A[:64, 64] = (x + 1j * x) * scale
    F, ipiv = factor64(A)
    assert np.array_equal(ipiv, np.arange(65))
    want = -Fraction(x) * Fraction(x) * 32 * Fraction(scale)
    # one rounding of the sum and of its subtraction; digit products beyond i + j = 9 are below 2^-54
    assert abs(Fraction(F[64, 64].real) - want) <= abs(want) * Fraction(2.0**-51)
    assert F[64, 64].imag == 0.0


@pytest.mark.parametrize("n", [65, 129, 191, 193, 321])
@pytest.mark.parametrize("kind", ["normal", "rows", "cols", "mixed", "wide", "signs"])
def test_update_slices_backward_error(gpu, n, kind):
    """P A - L U of the sliced update against the componentwise bound of an
    fp64 factorisation, also for rows and columns of very different size."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind in ("rows", "mixed"):
        A = A * 10.0 ** rng.uniform(-8, 8, n)[:, None]
    if kind in ("cols", "mixed"):
        A = A * 10.0 ** rng.uniform(-8, 8, n)[None, :]
    if kind == "wide":
        A = A * 10.0 ** rng.uniform(-4, 4, (n, n))
    if kind == "signs":  # +-1 with small noise: the eliminated rows mix entries of 1 and 1e-12
        A = np.where(rng.uniform(size=(n, n)) < 0.5, 1.0, -1.0) * (1 - 1e-12 * rng.uniform(size=(n, n))) + 0j
    F, ipiv = factor64(A)
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    P = A.copy()
    for i, p in enumerate(ipiv):
        P[[i, p]] = P[[p, i]]
    # gamma_n |L| |U|, twice for complex arithmetic and twice for this product's own rounding
    assert np.all(np.abs(P - L @ U) <= 4 * n * 2.0**-53 * (np.abs(L) @ np.abs(U)))
    # the integer sums are exact: the CUDA cores' form gives the same bits
    from mom25d_gb300 import engine as E

    G, gpiv = factor64(A, E.M25_LU_NO_TENSOR_CORES)
    assert np.array_equal(F, G) and np.array_equal(ipiv, gpiv)


def test_update_slices_not_finite(gpu):
    """An infinity or a NaN reaches the factors as it does without the slices."""
    from mom25d_gb300 import engine as E

    rng = np.random.default_rng(5)
    A = rng.standard_normal((200, 200)) + 1j * rng.standard_normal((200, 200))
    for bad in (np.nan, np.inf):
        B = A.copy()
        B[150, 10] = bad
        F, _ = factor64(B)
        G, _ = factor64(B, E.M25_LU_NO_TENSOR_CORES)
        assert not np.isfinite(F).all() and not np.isfinite(G).all()


def via_row_line(nvia):
    """A 50 ohm line beside a pour strip tied to ground by nvia vias."""
    import mom25d_gb300 as G

    mm = 1e-3
    W = 0.5561 * mm
    lay = G.Layout()
    lay.add_rect(-3 * mm, -W / 2, 3 * mm, W / 2)
    lay.add_rect(-3 * mm, W, 3 * mm, W + 0.8 * mm)
    for x in np.linspace(-2.5, 2.5, nvia) * mm:
        lay.add_via(x, W + 0.4 * mm, drill=0.2 * mm, pad=0.4 * mm)
    lay.add_port("P1", (-3 * mm, 0), "-x", W, 4 * mm)
    lay.add_port("P2", (3 * mm, 0), "+x", W, 4 * mm)
    return lay.mesh(max_cell=0.5 * mm, edge_cell=0.1 * mm), G.Substrate(3.66, 0.254 * mm, 0.003, 5.8e7)


@pytest.mark.parametrize("nvia", [1, 3, 8])
@pytest.mark.parametrize("freq", [1.5e9, 9e9])
def test_update_slices_with_vias(gpu, nvia, freq):
    """Via rows are 1e10 times the RWG rows of the impedance matrix: the fp64
    solve of the sliced update is as accurate as LAPACK's (both against a
    solve refined in extended precision; ten times for the two LUs' own
    rounding)."""
    from mom25d_gb300.solver import Solver, dense_solve

    mesh, sub = via_row_line(nvia)
    sol = Solver(mesh, sub, verbose=False)
    Z, B = sol.impedance(freq), sol.port_excitations().astype(complex)
    x = dense_solve(Z, B, precision="fp64", ctx=sol.ctx)
    sol.close()
    d = 1 / np.sqrt(np.abs(np.diag(Z)))
    lu = sl.lu_factor(d[:, None] * Z * d)
    ref = np.zeros_like(B, np.clongdouble)
    for _ in range(4):
        r = B - Z.astype(np.clongdouble) @ ref
        ref = ref + d[:, None] * sl.lu_solve(lu, d[:, None] * r.astype(complex))
    err = [float(np.linalg.norm(v - ref) / np.linalg.norm(ref)) for v in (x, np.linalg.solve(Z, B))]
    assert err[0] <= 10 * err[1] + 1e-15


@pytest.mark.parametrize("offset", [0, 1])
def test_complex64_device_alignment(gpu, offset):
    """Device complex64 arrays at an odd multiple of four bytes give the same
    bits as aligned ones: the LU (rows with a gap), the fill, the solve."""
    import torch

    import mom25d_gb300 as G
    from mom25d_gb300 import engine as E
    from mom25d_gb300 import workloads
    from mom25d_gb300.solver import Solver

    rng = np.random.default_rng(5)

    def dev(n, ld, off):
        buf = torch.zeros(2 * n * ld + 1, dtype=torch.float32, device="cuda")
        return buf, buf[off:off + 2 * n * ld].view(n, ld, 2), C.c_void_p(buf.data_ptr() + 4 * off)

    n, ld = 97, 101
    A = torch.from_numpy(rng.standard_normal((n, ld, 2)).astype(np.float32)).cuda()
    B = torch.from_numpy(rng.standard_normal((n, 2, 2))).cuda()
    _, _, mesh, freqs = workloads.build(G, "tee")
    sol = Solver(mesh, workloads.build(G, "tee")[1], verbose=False, precision="mixed_fill32")
    g, m = sol.greens(float(freqs[0])), mesh.n_unknowns
    out = []
    for off in (0, offset):
        ctx = sol.ctx
        buf, v, p = dev(n, ld, off)
        v.copy_(A)
        ipiv, info = torch.zeros(n, dtype=torch.int32, device="cuda"), np.zeros(3, np.int32)
        torch.cuda.synchronize()
        E.check(ctx.lib.m25_lu_factor(ctx.h, n, E.M25_MIXED, p, ld, C.cast(C.c_void_p(ipiv.data_ptr()),
                                      C.POINTER(C.c_int32)), E.M25_ON_DEVICE, 0, E.ptr(info, C.c_int32)))
        lu = v.cpu().numpy()
        assert np.array_equal(lu[:, n:], A.cpu().numpy()[:, n:])  # the gap keeps its values
        bufz, vz, pz = dev(m, m, off)
        E.check(ctx.lib.m25_assemble(ctx.h, sol.geometry().h, g.h, 0.01, 0.01, 0.01, 0.01, E.M25_MIXED_FILL32, pz, m,
                                     E.M25_ON_DEVICE))
        ctx.synchronize()
        bufs, vs, ps = dev(n, n, off)
        vs.copy_(A[:, :n])
        X = torch.zeros_like(B)
        torch.cuda.synchronize()
        E.check(ctx.lib.m25_dense_solve(ctx.h, n, 2, E.M25_MIXED_FILL32, ps, C.c_void_p(B.data_ptr()),
                                        C.c_void_p(X.data_ptr()), E.M25_ON_DEVICE, 1e-12, 50, E.ptr(info, C.c_int32)))
        ctx.synchronize()
        out.append((lu, ipiv.cpu().numpy(), vz.cpu().numpy(), X.cpu().numpy()))
    sol.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    Z = A.cpu().numpy()[:, :n].astype(float)
    r = (Z[..., 0] + 1j * Z[..., 1]) @ (out[0][3][..., 0] + 1j * out[0][3][..., 1])
    b = B.cpu().numpy()
    # the refinement's own stop: the backward error (1e-12) of one column
    assert np.linalg.norm(r - (b[..., 0] + 1j * b[..., 1])) <= 1e-11 * np.linalg.norm(Z) * np.linalg.norm(out[0][3])


@pytest.mark.parametrize("orders", [(1, 31, 32, 33, 63, 64, 65), (2100, 700, 2100, 97, 1500), (300, 2500, 129, 2500)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solves_of_changing_order(gpu, orders, precision):
    """Solves of one context at the edges of the sweeps' blocks and one order
    after another: what an earlier one left in the flag buffer is no flag."""
    from mom25d_gb300 import engine as E
    from mom25d_gb300.solver import dense_solve

    ctx = E.Context(0)
    for k, n in enumerate(orders):
        rng = np.random.default_rng(n + k)
        A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
        B = rng.standard_normal((n, 3)) + 0j
        for p in (precision, "fp64"):
            X = dense_solve(A, B, precision=p, ctx=ctx)
            # the solves' backward error (Higham, theorem 9.4, with the growth of these diagonally heavy matrices
            # near one), or the refinement's stop at 1e-12
            bound = 1e-12 if p == "mixed" else 8 * n * 2.0**-53
            r = np.abs(A @ X - B).max(0)
            assert np.all(r <= 4 * bound * (np.linalg.norm(A, np.inf) * np.abs(X).max(0) + np.abs(B).max(0)))
    ctx.close()
