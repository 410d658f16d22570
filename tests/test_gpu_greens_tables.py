"""The Sommerfeld integral's J0 tables and the splines (csrc/greens.cu): the
tabulated remainder against the same sum in numpy / scipy over radii at the
edges of its rules, and radius by radius independent of the launch."""

import ctypes as C

import numpy as np
import pytest
from scipy.special import jv

pytestmark = pytest.mark.gpu


def create(ctx, kc, wc, kr, wr, rho, freq=5e9, eps=3.5, t=0.5e-3):
    from mom25d_gb300 import engine as E

    a = dict(t=E.f64([t]), e=E.f64([eps]), ld=E.f64([0.0]), il=E.i32([1]), lz=E.f64([t]),
             kc=E.f64(np.stack([kc.real, kc.imag], 1)), wc=E.f64(np.stack([wc.real, wc.imag], 1)), kr=E.f64(kr),
             wr=E.f64(wr), rho=E.f64(rho))
    d = E.GreensDesc(freq, 1, E.ptr(a["t"]), E.ptr(a["e"]), E.ptr(a["ld"]), 1, E.ptr(a["il"], C.c_int32),
                     E.ptr(a["lz"]), 1, 0.0, 0.0, t, kc.size, kr.size, E.ptr(a["kc"]), E.ptr(a["wc"]), E.ptr(a["kr"]),
                     E.ptr(a["wr"]), rho.size, E.ptr(a["rho"]), 15.0 / t)
    h = C.c_void_p()
    E.check(ctx.lib.m25_greens_create(ctx.h, C.byref(d), C.byref(h)))
    res, info = np.zeros((rho.size, 3), complex), np.zeros(3)
    E.check(ctx.lib.m25_greens_remainder(h, E.ptr(res.view(np.float64)), E.ptr(info)))
    S, lead, coef = np.zeros((3, 1, 1, rho.size), complex), np.zeros((3, 1, 1), complex), np.zeros(
        (1, rho.size - 1, 4, 3), complex)
    E.check(ctx.lib.m25_greens_tables(h, E.ptr(S.view(np.float64)), E.ptr(lead.view(np.float64)),
                                      E.ptr(coef.view(np.float64))))
    ctx.lib.m25_greens_destroy(h)
    return res, S, coef


def slab(k, freq=5e9, eps=3.5, t=0.5e-3):
    """w-free coefficients k (g - leading) / 2 pi of one lossless slab."""
    k0 = 2 * np.pi * freq / 299792458.0
    k1 = k0 * np.sqrt(eps)
    u0, u1 = np.sqrt(k * k - k0 * k0 + 0j), np.sqrt(k * k - k1 * k1 + 0j)
    th = np.tanh(u1 * t)
    dte, dtm = u0 + u1 / th, eps * u0 + u1 * th
    g = [1 / dte, (u0 + u1 * th) / (dte * dtm), u0 * (th / u1) / dtm]
    cv, ka, kv = 2 / (eps + 1), np.sqrt((k0**2 + k1**2) / 2), np.sqrt((eps * k0**2 + k1**2) / (eps + 1))
    lead = [1 / (2 * np.sqrt(k * k - ka * ka + 0j)), cv / (2 * np.sqrt(k * k - kv * kv + 0j))]
    return np.stack([g[0] - lead[0], g[1] - lead[1], g[2] - lead[1]], -1) * (k / (2 * np.pi))[:, None]


# (arc nodes, their largest real and imaginary part, axis nodes, largest, radii): arguments below and beyond the
# tables' first rows, the series, imaginary parts beyond the expansion, axis arguments beyond the table's end
@pytest.mark.parametrize("nkc,kmax,im,nkr,krmax,rmax,n", [
    (1, 100.0, 10.0, 1, 200.0, 0.01, 4),
    (23, 400.0, 20.0, 63, 4e3, 0.05, 33),
    (25, 800.0, 25.0, 129, 4e4, 0.04, 65),
    (49, 600.0, 200.0, 65, 4e4, 0.03, 31),
    (1300, 900.0, 25.0, 7001, 4.2e5, 0.04, 96),
])
def test_sommerfeld_tables(gpu, nkc, kmax, im, nkr, krmax, rmax, n):
    from mom25d_gb300 import engine as E

    rng = np.random.default_rng(n)
    kc = np.sort(rng.uniform(1.0, kmax, nkc)) + 1j * im * rng.uniform(0.1, 1, nkc)
    kr = np.sort(rng.uniform(0.5 * kmax + 400, krmax + kmax + 400, nkr))
    wc, wr = rng.uniform(0.5, 1, nkc) + 0.1j, rng.uniform(0.5, 1, nkr)
    rho = np.concatenate([[0.0], np.sort(rng.uniform(0, rmax, n - 1))])
    ctx = E.Context(0)
    res, S, coef = create(ctx, kc, wc, kr, wr, rho)
    c = np.concatenate([slab(kc) * wc[:, None], slab(kr + 0j) * wr[:, None]])
    k = np.concatenate([kc, kr + 0j])
    J = jv(0, rho[:, None] * k[None, :])
    want, size = J @ c, np.abs(J) @ np.abs(c)
    # the coefficients' own rounding (subtraction of the leading term, some ten operations) and J0's (the
    # argument's rounding in the oracle: eps |r k| J1): per term, relative to the leading terms' magnitude
    mag = np.abs(J) @ (np.abs(c) + np.abs(np.concatenate([wc, wr]))[:, None] / (2 * np.pi))
    arg = (np.abs(rho[:, None] * k[None, :]) * np.abs(jv(1, rho[:, None] * k[None, :]))) @ np.abs(c)
    assert np.all(np.abs(res - want) <= 2.0**-53 * (64 * mag + 4 * arg + 8 * size))
    # a radius's value does not depend on the radii tabulated with it
    part = create(ctx, kc, wc, kr, wr, rho[: max(4, n // 2)])[0]
    assert np.array_equal(part, res[: max(4, n // 2)]) or krmax * rmax > 1e4
    ctx.close()


@pytest.mark.parametrize("n", [4, 5, 6, 33, 129, 600])
@pytest.mark.parametrize("grid", ["even", "growing"])
def test_spline_coefficients(gpu, n, grid):
    from scipy.interpolate import CubicSpline

    from mom25d_gb300 import engine as E

    rho = np.linspace(0, 0.02, n) if grid == "even" else np.concatenate([[0], 1e-5 * 1.012 ** np.arange(n - 1)])
    kc = np.linspace(1, 300, 24) + 5j
    ctx = E.Context(0)
    _, S, coef = create(ctx, kc, 0 * kc + 3.0, np.linspace(400.0, 3e3, 64), np.full(64, 40.0), rho)
    ctx.close()
    h = np.diff(rho)
    for m in range(3):
        want = CubicSpline(rho, S[m, 0, 0]).c  # (4, n - 1), not-a-knot
        # slopes: backward stable solves of a system of condition <= 3 (rows dominated two to one), the data's
        # rounding eps |S| / h in the secants; a coefficient of order p carries it over h^(3 - p)
        noise = 2.0**-53 * 64 * np.abs(S[m]).max() / h.min()
        for p in range(4):
            assert np.all(np.abs(coef[0, :, p, m] - want[p]) <= 8 * noise / h ** (2 - p) + 1e-300)
