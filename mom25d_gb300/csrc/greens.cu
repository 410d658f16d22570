// Tabulated spatial Green's functions at one frequency, computed on the
// device: the remainder of the spectral MPIE kernels after removing the
// leading c e^{-jkR}/(4 pi R) terms, integrated along a lifted Sommerfeld
// path, tabulated on a rho grid and fitted with not-a-knot cubic splines.
// Follows Engine/mom25d/greens.py:111-212 (one grounded slab) and
// Engine/mom25d/layered.py:238-405 (open multilayer stack, Michalski-Zheng
// transmission-line form).
#include <algorithm>
#include <cstring>
#include <vector>

#include "m25_internal.h"
#include "m25_lu.h"

namespace m25 {

constexpr int kMaxLayers = 8;

struct StackDev {
  int nlayer, nlev, single;
  double t[kMaxLayers];
  zd epsc[kMaxLayers], kk[kMaxLayers];
  int il[kMaxLev];
  double zl[kMaxLev];
  double k0, h;
  int top_pec;                     // a PEC cover on the top layer (layered.py:257-275)
  zd lead_c[3][kMaxLev][kMaxLev];  // c_A, c_V, c_W per (observer, source)
  zd kx[2][kMaxLev][kMaxLev];      // k of the A and the V/W leading terms
  double dz[kMaxLev][kMaxLev];
};

// One-slab spectral kernels gA~, gV~, gW~ (greens.py:234-252).
__device__ void slab_spectral(const StackDev& S, zd kr, zd& gA, zd& gV, zd& gW) {
  const double h = S.t[0];
  zd kr2 = kr * kr;
  zd u0 = csqrt(kr2 - zd(S.k0 * S.k0));
  zd u1 = csqrt(kr2 - S.kk[0] * S.kk[0]);
  zd x = u1 * h;
  zd e = cexp(x * -2.0);
  zd u1coth, u1tanh, tanh_over_u1;
  if (cabs(x) < 1e-4) {
    u1coth = zd(1.0 / h) + (u1 * u1) * (h / 3.0);
    u1tanh = (u1 * u1) * h;
    tanh_over_u1 = zd(h);
  } else {
    u1coth = u1 * (zd(1.0) + e) / (zd(1.0) - e);
    u1tanh = u1 * (zd(1.0) - e) / (zd(1.0) + e);
    tanh_over_u1 = u1tanh / (u1 * u1);
  }
  zd dte = u0 + u1coth;
  zd dtm = S.epsc[0] * u0 + u1tanh;
  gA = zd(1.0) / dte;
  gV = (u0 + u1tanh) / (dte * dtm);
  gW = u0 * tanh_over_u1 / dtm;
}

// Multilayer spectral kernels via TE/TM line voltages (layered.py:238-289):
// g[m][i][j], m = A, V, W; i observer level, j source level. Two neighbouring
// lanes work on one node: the layers' constants shared out between them, lane
// `mode` the line voltages of its mode (0: h, 1: e), then the levels j in turn.
// (One thread's chain of ~50 complex divisions, exponentials and roots was the kernel's time.)
__device__ void layered_spectral(const StackDev& S, zd kr, int mode, zd* __restrict__ out) {
  const int N = S.nlayer, L = S.nlev;
  const zd one(1.0);
  auto other = [](zd v) { return zd(__shfl_xor_sync(0xffffffffu, v.re, 1), __shfl_xor_sync(0xffffffffu, v.im, 1)); };
  zd u[kMaxLayers], T[kMaxLayers], Sh[kMaxLayers], iu[kMaxLayers];
  const zd kr2 = kr * kr;
  for (int n0 = 0; n0 < N; n0 += 2) {
    const int n = min(n0 + mode, N - 1);
    const zd un = csqrt(kr2 - S.kk[n] * S.kk[n]);
    const zd x = un * S.t[n], p = cexp(-x), e = cexp(x * -2.0), d = one / (one + e);
    const zd Tn = (one - e) * d, Sn = (p * 2.0) * d, in = one / un;
    const zd uo = other(un), To = other(Tn), So = other(Sn), io = other(in);
    u[n0] = mode ? uo : un;
    T[n0] = mode ? To : Tn;
    Sh[n0] = mode ? So : Sn;
    iu[n0] = mode ? io : in;
    if (n0 + 1 < N) {
      u[n0 + 1] = mode ? un : uo;
      T[n0 + 1] = mode ? Tn : To;
      Sh[n0 + 1] = mode ? Sn : So;
      iu[n0 + 1] = mode ? in : io;
    }
  }
  const zd u0 = csqrt(kr2 - zd(S.k0 * S.k0));
  zd Vm[kMaxLev][kMaxLayers + 1];
  {
    zd y[kMaxLayers];
    for (int n = 0; n < N; ++n) y[n] = mode == 0 ? u[n] : S.epsc[n] * iu[n];
    const zd yair = mode == 0 ? u0 : one / u0;
    zd ydn[kMaxLayers + 1], yup[kMaxLayers + 1];
    ydn[1] = y[0] / T[0];
    for (int k = 2; k <= N; ++k) {
      zd yl = ydn[k - 1], yk = y[k - 1], tk = T[k - 1];
      ydn[k] = yk * (yl + yk * tk) / (yk + yl * tk);
    }
    yup[N] = S.top_pec ? zd(0.0) : yair;  // (unused under a cover: no level on it)
    for (int k = N - 1; k >= 1; --k) {
      zd yk = y[k], tk = T[k];
      if (S.top_pec && k == N - 1) {
        yup[k] = yk / tk;  // layer N shorted by the cover
      } else {
        zd yl = yup[k + 1];
        yup[k] = yk * (yl + yk * tk) / (yk + yl * tk);
      }
    }
    // V_{k-1} / V_k below a source, V_{k+1} / V_k above it: the same for every source level
    zd dn[kMaxLayers + 1], up[kMaxLayers + 1];
    for (int k = 2; k <= N; ++k) dn[k] = Sh[k - 1] * y[k - 1] / (y[k - 1] + ydn[k - 1] * T[k - 1]);
    for (int k = 1; k < N; ++k) {
      if (S.top_pec && k + 1 == N) break;  // V_N = 0 on the cover
      up[k] = Sh[k] * y[k] / (y[k] + yup[k + 1] * T[k]);
    }
    for (int l = 0; l < L; ++l) {
      zd* V = Vm[l];
      for (int k = 0; k <= N; ++k) V[k] = zd(0.0);
      int s = S.il[l];
      V[s] = one / (ydn[s] + yup[s]);
      for (int k = s; k >= 2; --k) V[k - 1] = V[k] * dn[k];
      for (int k = s; k < N; ++k) {
        if (S.top_pec && k + 1 == N) break;
        V[k + 1] = V[k] * up[k];
      }
    }
  }
  const double k02 = S.k0 * S.k0;
  const zd ikr2 = one / kr2;
  for (int j = 0; j < L; ++j) {
    zd cum(0.0);
    int n = 0;
    for (int i = 0; i < L; ++i) {  // levels by rising interface
      const int ii = S.il[i];
      const zd v = Vm[j][ii], vo = other(v);  // both modes at the level
      if (mode == 0) {
        out[(0 * L + i) * L + j] = v;
        out[(1 * L + i) * L + j] = (vo + v * k02) * ikr2;
      } else {
        if (ii < n) {
          cum = zd(0.0);
          n = 0;
        }
        for (; n < ii; ++n) cum += (Vm[j][n + 1] - Vm[j][n]) * (iu[n] * iu[n]);
        out[(2 * L + i) * L + j] = cum;
      }
    }
  }
}

// Leading-term coefficients (greens.py:215-224, layered.py:292-331), one warp
// per level pair (each is a chain of fp64 latencies; one thread for all took L^2 of them); gbig:
// the layered spectral kernels at kbig (spectral_g_kernel's last node).
__global__ void leading_kernel(StackDev* S, double kbig, const zd* __restrict__ gbig) {
  if (threadIdx.x & 31) return;
  StackDev& s = *S;
  const int L = s.nlev, N = s.nlayer;
  if (s.single) {
    if (threadIdx.x) return;
    zd k1 = s.kk[0], e = s.epsc[0];
    zd k02(s.k0 * s.k0);
    zd ka = csqrt((k02 + k1 * k1) * 0.5);
    zd cv = zd(2.0) / (e + zd(1.0));
    zd kv = csqrt((e * k02 + k1 * k1) / (e + zd(1.0)));
    s.lead_c[0][0][0] = zd(1.0);
    s.lead_c[1][0][0] = cv;
    s.lead_c[2][0][0] = cv;
    s.kx[0][0][0] = ka;
    s.kx[1][0][0] = kv;
    s.dz[0][0] = 0.0;
    return;
  }
  const int i = (threadIdx.x >> 5) / L, j = (threadIdx.x >> 5) % L;
  s.dz[i][j] = fabs(s.zl[i] - s.zl[j]);
  if (i == j) {
    int n = s.il[i];
    zd eb = s.epsc[n - 1], kb = s.kk[n - 1], ea, ka;
    if (n == N) {
      ea = zd(1.0);
      ka = zd(s.k0);
    } else {
      ea = s.epsc[n];
      ka = s.kk[n];
    }
    zd cv = zd(2.0) / (ea + eb);
    s.lead_c[0][i][j] = zd(1.0);
    s.lead_c[1][i][j] = cv;
    s.lead_c[2][i][j] = cv;
    s.kx[0][i][j] = csqrt((ka * ka + kb * kb) * 0.5);
    s.kx[1][i][j] = csqrt((eb * (ka * ka) + ea * (kb * kb)) / (ea + eb));
    return;
  }
  zd ux = csqrt(zd(kbig * kbig - s.k0 * s.k0));
  zd f = ux * 2.0 * cexp(ux * s.dz[i][j]);
  zd c[3];
  for (int m = 0; m < 3; ++m) c[m] = f * gbig[(m * L + i) * L + j];
  if (s.zl[j] < s.zl[i]) c[2] = zd(0.0);
  for (int m = 0; m < 3; ++m) {
    // drop the numerical noise of static coefficients' imaginary parts
    if (fabs(c[m].im) < 1e-9 * cabs(c[m])) c[m].im = 0.0;
    s.lead_c[m][i][j] = c[m];
  }
  s.kx[0][i][j] = zd(s.k0);
  s.kx[1][i][j] = zd(s.k0);
}

// coef[q][(m*L + i)*L + j] = w k (g - leading term) / 2pi at every path node
// (in place over the spectral kernels g), one thread per (node, level pair):
// V and W share their leading term's exponential, and A's too where its k is
// the same (i != j). Pairs vary slowest, so that a warp takes one branch.
__global__ void spectral_coef_kernel(const StackDev* __restrict__ Sp, int nkc, const double* __restrict__ kc,
                                     const double* __restrict__ wc, int nkr, const double* __restrict__ kr,
                                     const double* __restrict__ wr, zd* __restrict__ cc, zd* __restrict__ cr) {
  const StackDev& S = *Sp;
  const int L = S.nlev, LL = L * L, nk = nkc + nkr;
  const int q = blockIdx.x * blockDim.x + threadIdx.x, pair = blockIdx.y;
  if (q >= nk) return;
  const int i = pair / L, j = pair % L;
  const bool cpath = q < nkc;
  const int qq = cpath ? q : q - nkc;
  const zd k = cpath ? zd(kc[2 * qq], kc[2 * qq + 1]) : zd(kr[qq], 0.0);
  const zd w = cpath ? zd(wc[2 * qq], wc[2 * qq + 1]) : zd(wr[qq], 0.0);
  zd* c = (cpath ? cc : cr) + (int64_t)qq * 3 * LL + pair;
  const zd scale = (w * k) * (1.0 / (2.0 * kPi));
  const double dz = S.dz[i][j];
  // e^{-ux dz} / (2 ux)
  auto leading = [&](zd kx) {
    const zd ux = csqrt(k * k - kx * kx);
    return (dz == 0.0 ? zd(1.0) : cexp(ux * (-dz))) / (ux * 2.0);
  };
  const zd ka = S.kx[0][i][j], kv = S.kx[1][i][j];
  zd e = leading(ka);
  c[0] = scale * (c[0] - S.lead_c[0][i][j] * e);
  if (kv.re != ka.re || kv.im != ka.im) e = leading(kv);
  c[LL] = scale * (c[LL] - S.lead_c[1][i][j] * e);
  c[2 * LL] = scale * (c[2 * LL] - S.lead_c[2][i][j] * e);
}

// J0 of a complex argument: the trapezoidal rule on Bessel's integral
// J0(z) = (1/2pi) Int_0^{2pi} cos(z sin t) dt, which converges geometrically
// for this periodic integrand (error ~ 2 J_M(z)); M is a multiple of 4 with
// M >= 1.5 |z| + 24, using the symmetry of sin t over the quarter periods.
__device__ inline zd bessel_j0_complex(zd z) {
  double az = hypot(z.re, z.im);
  int M = 4 * (int)ceil((1.5 * az + 24.0) * 0.25);
  int Q = M / 4;
  double sr = 0.0, si = 0.0;
  for (int m = 1; m < Q; ++m) {
    double s = sinpi(2.0 * m / M);
    double a = z.re * s, b = z.im * s;
    double sa, ca;
    sincos(a, &sa, &ca);
    double eb = exp(b), ebi = 1.0 / eb;
    sr += ca * 0.5 * (eb + ebi);
    si -= sa * 0.5 * (eb - ebi);
  }
  // cos z at the quarter points
  double sa, ca;
  sincos(z.re, &sa, &ca);
  double eb = exp(z.im), ebi = 1.0 / eb;
  double cr = ca * 0.5 * (eb + ebi), ci = -sa * 0.5 * (eb - ebi);
  return {(2.0 + 2.0 * cr + 4.0 * sr) / M, (2.0 * ci + 4.0 * si) / M};
}

// J0 at the points of the path. The integral needs it at every pair of a
// radius and a path node, so the cost of one J0 is the cost of the tables
// (fp64 runs at two operations per clock on an SM; CUDA's j0 with its argument
// reduction and the trapezoidal rule above took 85 % of the tabulation). Its Taylor
// coefficients about equidistant points are tabulated once per call instead,
// from J0 and J1 there and the recurrence that Bessel's equation
// x y'' + y' + x y = 0 gives them:
//   (n+2)(n+1) x c_{n+2} = -((n+1)^2 c_{n+1} + c_{n-1} + x c_n).
// Row i holds c_n h^n about i h, for the argument in units of h.
//  - real axis: h = 1/8, degree 8: |J0^(9)| (h/2)^9 / 9! < 5e-17.
//  - lifted arc: h = 1/4 and degree 19, for imaginary parts up to 1.0625 (the
//    path's a rho <= 1): 0.4 x 1.07^20 / 20! < 1e-18. Rows below x = 2, where the
//    expansion would reach the other solutions' singularity at 0, stay
//    empty: the power series serves there.
// The distance to the grid point is fma(r / h, k, -i): the product is not
// rounded by itself, which for r k ~ 1e3 leaves J0 more accurate than j0(r * k).
constexpr int kHankelMin = 25;  // j01_hankel from here on
constexpr int kJ0Step = 8, kJ0Deg = 8, kJ0Row = 10;        // rows of 10 doubles: double2 loads
constexpr int kJ0ArcStep = 4, kJ0ArcDeg = 19, kJ0ArcRow = 20;
constexpr int kJ0ArcMin = 2 * kJ0ArcStep;                   // first row used
constexpr double kJ0ArcIm = 1.0625 * kJ0ArcStep;            // largest |Im z| / h
// Rows at most: arguments up to 16384 and 256, beyond which the functions themselves are called.
constexpr int kJ0Rows = 1 << 17, kJ0ArcRows = 1 << 10;  // (j01_warp: 256)
inline int j0_rows(double xmax, int step, int cap) {
  return !(xmax >= 0) ? 1 : (int)std::min((double)cap, std::floor(xmax * step) + 2.0);
}

// CTAs of 64 threads for the arc's rows
__host__ __device__ inline int j0_arc_ctas(int rows) { return rows > kJ0ArcMin ? (rows - kJ0ArcMin + 1) / 2 : 0; }
// and for the axis's rows below x = 25 (by a warp each, as the arc's) and beyond
__host__ __device__ inline int j0_near_ctas(int rows) { return (min(rows, kJ0Step * kHankelMin) + 1) / 2; }
__host__ __device__ inline int j0_ctas(int rows_r, int rows_a) {
  const int near = j0_near_ctas(rows_r);
  return j0_arc_ctas(rows_a) + near + (max(rows_r - 2 * near, 0) + 63) / 64;
}

// Row i of a table (see above): `step` points per unit, coefficients to
// degree DEG, from c0 = J0 and c1 = -J1 there.
template <int DEG>
__device__ __forceinline__ void j0_row(int i, int step, double c0, double c1, double* __restrict__ out) {
  const double h = 1.0 / step, x = i * h;
  if (i == 0) {  // c_2k = (-1/4)^k / k!^2
    double c = 1.0;
#pragma unroll
    for (int n = 0; n <= DEG; ++n) {
      out[n] = (n & 1) ? 0.0 : c;
      if (n & 1) c *= -0.25 * h * h / (((n + 1) / 2) * ((n + 1) / 2));
    }
    return;
  }
  const double inv = 1.0 / x;
  double cm = 0.0, hn = 1.0;
#pragma unroll
  for (int n = 0; n <= DEG; ++n) {
    out[n] = c0 * hn;
    const double c2 = -fma(fma((double)((n + 1) * (n + 1)), c1, cm), inv, c0) * (1.0 / ((n + 1) * (n + 2)));
    cm = c0;
    c0 = c1;
    c1 = c2;
    hn *= h;
  }
}

// J0 and J1 at one point x <= 256 by a warp: the trapezoidal rule on Bessel's
// integral with 512 points (a quarter period of them, four per lane). Nodes
// share rows, so that an error of a row does not average out over them as their own
// roundings do: many more points than the rule needs average the rounding of
// its terms here (about 2e-17; CUDA's j0 and j1 are off by 1e-15 beyond 8 and by 1e-13 beyond 20).
__device__ void j01_warp(double x, double& y0, double& y1) {
  double s0 = 0.0, s1 = 0.0;
  for (int q = 0; q < 4; ++q) {
    int m = (threadIdx.x & 31) + 32 * q;
    if (m == 0) m = 128;  // the quarter point in the place of the first, a constant
    const double s = sinpi(m / 256.0), a = x * s, r = fma(x, s, -a);
    double sa, ca;
    sincos(a, &sa, &ca);
    const double g = m == 128 ? 2.0 : 4.0;
    s0 = fma(g, fma(-r, sa, ca), s0);
    s1 = fma(g * s, fma(r, ca, sa), s1);
  }
  for (int o = 16; o; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  y0 = (2.0 + s0) * (1.0 / 512.0);
  y1 = s1 * (1.0 / 512.0);
}

// J0 and J1 at x >= 25: Hankel's expansions (Abramowitz & Stegun 9.2.5 - 9.2.10),
// J_v = (2 / pi x)^1/2 (P_v cos chi - Q_v sin chi), chi = x - (v/2 + 1/4) pi, to the
// term of x^-17 (the next one is below 4e-17 at x = 25).
__device__ void j01_hankel(double x, double& y0, double& y1) {
  const double ix = 1.0 / x, amp = rsqrt(kPi * x);
  double s, c, P[2], Q[2];
  sincos(x, &s, &c);
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    double t = 1.0, p = 1.0, q = 0.0;
#pragma unroll
    for (int k = 1; k <= 17; ++k) {
      t *= ix * ((4 * v - (2 * k - 1) * (2 * k - 1)) / (8.0 * k));
      double& sum = (k & 1) ? q : p;
      sum += (k & 2) ? -t : t;
    }
    P[v] = p;
    Q[v] = q;
  }
  y0 = amp * (P[0] * (c + s) - Q[0] * (s - c));
  y1 = amp * (P[1] * (s - c) + Q[1] * (s + c));
}

// The grid point next to r k / h for rs = r / h: its index (false: outside
// 0 .. rows - 1, not a number) and the distance to it in units of h.
__device__ __forceinline__ bool j0_locate(double rs, double k, int rows, int& i, double& d) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5 x 2^52: the sum's low word is the integer next to rs k
  const double t = fma(rs, k, kMagic);
  i = __double2loint(t);
  d = fma(rs, k, kMagic - t);
  return (unsigned)i < (unsigned)rows && __double2hiint(t) == 0x43380000;
}

// J0(r k) on the real axis; rs = r kJ0Step.
__device__ __forceinline__ double j0_real(double r, double rs, double k, const double* __restrict__ tab, int rows) {
  int i;
  double d;
  if (!j0_locate(rs, k, rows, i, d)) return j0(r * k);
  const double2* c = reinterpret_cast<const double2*>(tab + (size_t)i * kJ0Row);
  const double2 c01 = c[0], c23 = c[1], c45 = c[2], c67 = c[3];
  double v = tab[(size_t)i * kJ0Row + 8];
  v = fma(v, d, c67.y);
  v = fma(v, d, c67.x);
  v = fma(v, d, c45.y);
  v = fma(v, d, c45.x);
  v = fma(v, d, c23.y);
  v = fma(v, d, c23.x);
  v = fma(v, d, c01.y);
  return fma(v, d, c01.x);
}

__device__ __noinline__ zd j0_far(zd z) { return bessel_j0_complex(z); }

// J0(z) for |Re z| < 2, |Im z| < 1.1: the power series in -z^2 / 4 (|.| <= 1.27: 1.27^13 / 13!^2 < 1e-18).
__device__ __noinline__ zd j0_series(zd z) {
  const zd w = z * z * -0.25;
  zd v(1.0, 0.0);
#pragma unroll
  for (int k = 12; k >= 1; --k) {
    const zd t = v * w;
    v = zd(fma(t.re, 1.0 / (k * k), 1.0), t.im * (1.0 / (k * k)));
  }
  return v;
}

// J0(r k) on the lifted arc; rs = r kJ0ArcStep. The polynomial with real
// coefficients at the complex distance d by division by t^2 - 2 Re d t +
// |d|^2: two operations per coefficient.
__device__ __forceinline__ zd j0_arc(double r, double rs, zd k, const double* __restrict__ tab, int rows) {
  int i;
  double dr;
  const double di = rs * k.im;
  const bool in = j0_locate(rs, k.re, rows, i, dr) && fabs(di) <= kJ0ArcIm;
  if (!in) return j0_far(k * r);
  if (i < kJ0ArcMin) return j0_series(k * r);
  const double2* c = reinterpret_cast<const double2*>(tab + (size_t)i * kJ0ArcRow);
  const double s = dr + dr, t = fma(dr, dr, di * di);
  double2 a = c[kJ0ArcDeg / 2];
  double b2 = a.y, b1 = fma(s, a.y, a.x);  // b_{n}, b_{n-1} of the quotient
#pragma unroll
  for (int p = kJ0ArcDeg / 2 - 1; p >= 1; --p) {
    a = c[p];
    b2 = fma(s, b1, fma(-t, b2, a.y));
    b1 = fma(s, b2, fma(-t, b1, a.x));
  }
  a = c[0];
  const double q1 = fma(s, b1, fma(-t, b2, a.y));
  return {fma(q1, dr, fma(-t, b1, a.x)), q1 * di};
}

// The learned remainder's network inputs of n radii at frequency f.
struct SurFeatures {
  int n;  // 0: none
  const double* rho;
  double a, rho_ref, f, fmin, fmax;
  float* X;  // (n, 2)
};
__device__ void sur_features(const SurFeatures& s, int i) {
  if (i >= s.n) return;
  s.X[2 * i] = (float)(2.0 * log1p(s.rho[i] / s.a) / log1p(s.rho_ref / s.a) - 1.0);
  s.X[2 * i + 1] = (float)(2.0 * (s.f - s.fmin) / (s.fmax - s.fmin) - 1.0);
}

// The spectral kernels g[(m*L + i)*L + j] at every path node, in one launch:
// nodes q < nkc of the lifted arc into gc, the next nkr of the real axis into
// gr, and (layered stacks) one more node at kbig into gbig for the leading
// terms. A node is a fp64 chain of square roots, exponentials and divisions
// through the layers, on one lane (one slab) or two (layered_spectral); small
// CTAs spread the nodes over the SMs. 7176 nodes of two layers: 48 us (one lane a
// node and a division for every use of 1 / u^2 and 1 / k^2: 82 us).
// The CTAs from nb on fill the J0 tables of the integral and, last, the
// network's inputs.
__global__ void __launch_bounds__(64) spectral_g_kernel(const StackDev* __restrict__ Sp, int nkc,
                                                        const double* __restrict__ kc, int nkr,
                                                        const double* __restrict__ kr, double kbig,
                                                        zd* __restrict__ gc, zd* __restrict__ gr,
                                                        zd* __restrict__ gbig, int nb, double* __restrict__ j0r,
                                                        int rows_r, double* __restrict__ j0a, int rows_a,
                                                        SurFeatures sf) {
  if ((int)blockIdx.x >= nb) {  // the rows of the J0 tables
    const int nj = j0_ctas(rows_r, rows_a);
    if ((int)blockIdx.x >= nb + nj) {
      sur_features(sf, ((int)blockIdx.x - nb - nj) * blockDim.x + threadIdx.x);
      return;
    }
    const int b = (int)blockIdx.x - nb, nba = j0_arc_ctas(rows_a), nbr = j0_near_ctas(rows_r);
    const int w = threadIdx.x >> 5;
    if (b < nba + nbr) {
      const bool arc = b < nba;
      const int i = arc ? kJ0ArcMin + 2 * b + w : 2 * (b - nba) + w;
      double y0, y1;
      j01_warp(arc ? (double)i / kJ0ArcStep : (double)i / kJ0Step, y0, y1);
      if ((threadIdx.x & 31) == 0) {
        if (arc && i < rows_a) j0_row<kJ0ArcDeg>(i, kJ0ArcStep, y0, -y1, j0a + (size_t)i * kJ0ArcRow);
        if (!arc && i < rows_r) j0_row<kJ0Deg>(i, kJ0Step, y0, -y1, j0r + (size_t)i * kJ0Row);
      }
    } else {
      const int i = 2 * nbr + (b - nba - nbr) * blockDim.x + threadIdx.x;
      double y0, y1;
      j01_hankel((double)i / kJ0Step, y0, y1);
      if (i < rows_r) j0_row<kJ0Deg>(i, kJ0Step, y0, -y1, j0r + (size_t)i * kJ0Row);
    }
    return;
  }
  const StackDev& S = *Sp;
  const int NC = 3 * S.nlev * S.nlev;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (S.single) {
    if (t >= nkc + nkr) return;
    const zd k = t < nkc ? zd(kc[2 * t], kc[2 * t + 1]) : zd(kr[t - nkc], 0.0);
    zd* out = t < nkc ? gc + 3 * (int64_t)t : gr + 3 * (int64_t)(t - nkc);
    slab_spectral(S, k, out[0], out[1], out[2]);
    return;
  }
  const int q = min(t >> 1, nkc + nkr);  // the lanes beyond repeat the last node (all lanes take the exchanges)
  const zd k = q < nkc ? zd(kc[2 * q], kc[2 * q + 1]) : zd(q < nkc + nkr ? kr[q - nkc] : kbig, 0.0);
  zd* out = q < nkc ? gc + (int64_t)q * NC : q < nkc + nkr ? gr + (int64_t)(q - nkc) * NC : gbig;
  layered_spectral(S, k, t & 1, out);
}

// Splits of the node sum: at most kSomArcSplit ranges of the arc's nodes and
// kSomRealSplit of the axis's, about 24 and 64 nodes in each, whatever the
// radii launched with it, so that a radius's value does not depend on which
// radii share its launch.
constexpr int kSomArcSplit = 48, kSomRealSplit = 96;
inline int som_split_arc(int nkc) { return std::min(kSomArcSplit, std::max(1, (nkc + 23) / 24)); }
inline int som_split_real(int nkr) { return std::min(kSomRealSplit, std::max(1, (nkr + 63) / 64)); }

struct SomArgs {
  int ne;
  const int* idx;  // radii rho[idx[e]] (NULL: rho[e])
  const double* rho;
  int nsa, nsr;  // ranges of arc and real nodes
  int nkc;
  const double* kc;
  const zd* coef_c;
  int nkr;
  const double* kr;
  const zd* coef_r;
  const double *j0r, *j0a;  // J0 tables
  int rows_r, rows_a;
  double* part;
  const int* skip;
};

// part[s][c][re / im][e] = sum over the nodes of range s of J0(rho k)
// coef[k][c] at radius rho[idx[e]]; ranges 0 .. nsa - 1 on the lifted arc
// (complex J0; the dearer ones, so they start first), then nsr on the real
// axis. A CTA takes 32 radii, one per lane, and its four warps every fourth node of the
// range: the coefficients are the same for all lanes (a thread per node had
// to sum its 2 NC values over the CTA for every radius, more work than the
// products), and the warps' sums meet once, in shared memory. Bound by fp64
// operations: 11 for a real J0, about 50 for a complex one, 2 NC and 4 NC for the
// products. 372 radii x 7176 nodes, 12 columns (the via transition's tables):
// 270 us, 1180 us before; 233 radii, 3 columns 74 us, some 430 us before.
// With skip set (the learned remainder was accepted) the CTAs return at once.
// Launched behind the network's kernel, which it does not read, it runs beside it: it waits for that one's end
// only at its own.
template <int NC>
__global__ void __launch_bounds__(128) sommerfeld_kernel(SomArgs a) {
  if (a.skip && *a.skip) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e = blockIdx.y * 32 + lane, s = blockIdx.x;
  const int ee = min(e, a.ne - 1);
  const double r = a.rho[a.idx ? a.idx[ee] : ee];
  double acc_re[NC], acc_im[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc_re[c] = acc_im[c] = 0.0;
  if (s < a.nsa) {
    const int q0 = (int)((int64_t)a.nkc * s / a.nsa), q1 = (int)((int64_t)a.nkc * (s + 1) / a.nsa);
    const double rs = r * kJ0ArcStep;
    for (int q = q0 + w; q < q1; q += 4) {
      const zd J = j0_arc(r, rs, zd(a.kc[2 * q], a.kc[2 * q + 1]), a.j0a, a.rows_a);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const zd v = ldc(a.coef_c + (int64_t)q * NC + c);
        acc_re[c] = fma(J.re, v.re, fma(-J.im, v.im, acc_re[c]));
        acc_im[c] = fma(J.re, v.im, fma(J.im, v.re, acc_im[c]));
      }
    }
  } else {
    const int sr = s - a.nsa;
    const int q0 = (int)((int64_t)a.nkr * sr / a.nsr), q1 = (int)((int64_t)a.nkr * (sr + 1) / a.nsr);
    const double rs = r * kJ0Step;
#pragma unroll 2
    for (int q = q0 + w; q < q1; q += 4) {
      const double J = j0_real(r, rs, a.kr[q], a.j0r, a.rows_r);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const zd v = ldc(a.coef_r + (int64_t)q * NC + c);
        acc_re[c] = fma(J, v.re, acc_re[c]);
        acc_im[c] = fma(J, v.im, acc_im[c]);
      }
    }
  }
  // the warps' sums, four columns at a time: warp w adds up column c0 + w
  __shared__ double red[4][8][32];
#pragma unroll
  for (int c0 = 0; c0 < NC; c0 += 4) {
    if (c0) __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c0 + j < NC) {
        red[w][2 * j][lane] = acc_re[c0 + j];
        red[w][2 * j + 1][lane] = acc_im[c0 + j];
      }
    __syncthreads();
    if (c0 + w < NC && e < a.ne) {
      double* o = a.part + ((int64_t)s * NC + c0 + w) * 2 * a.ne + e;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        o[h * a.ne] = (red[0][2 * w + h][lane] + red[1][2 * w + h][lane]) +
                      (red[2][2 * w + h][lane] + red[3][2 * w + h][lane]);
    }
  }
  grid_wait();
}

// res[idx[e]][c] = sum over the node ranges s of part[s][c][..][e]: eight
// lanes per value, each every eighth range.
__global__ void __launch_bounds__(256) sommerfeld_sum_kernel(int ne, int NC, const int* __restrict__ idx, int nsplit,
                                                             const double* __restrict__ part, zd* __restrict__ res,
                                                             const int* __restrict__ skip) {
  if (skip && *skip) return;
  const int nv = ne * NC * 2, t0 = blockIdx.x * 32, l = threadIdx.x & 31, g = threadIdx.x >> 5;
  __shared__ double red[8][32];
  const int t = t0 + l;
  double v = 0.0;
  if (t < nv)
    for (int s = g; s < nsplit; s += 8) v += part[(int64_t)s * nv + t];
  red[g][l] = v;
  __syncthreads();
  if (g == 0 && t < nv) {
    for (int k = 1; k < 8; ++k) v += red[k][l];
    const int e = t % ne, ch = t / ne;
    double* o = reinterpret_cast<double*>(res + (int64_t)(idx ? idx[e] : e) * NC + (ch >> 1));
    o[ch & 1] = v;
  }
}

// S tables: closed-form expm1 part of the leading term, the Sommerfeld
// remainder and, for gA, the ground-plane loss kernel (greens.py:298-335,
// layered.py:391-405).  S layout (3, L, L, nrho).
__global__ void table_kernel(const StackDev* __restrict__ Sp, int nrho, const double* __restrict__ rho,
                             const zd* __restrict__ res, double omega, zd zs_ground, zd* __restrict__ Stab) {
  const StackDev& S = *Sp;
  const int L = S.nlev, NC = 3 * L * L;
  int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= NC * nrho) return;
  int c = gid / nrho, ir = gid % nrho;
  int m = c / (L * L), i = (c / L) % L, j = c % L;
  double r = rho[ir];
  double dz = S.dz[i][j];
  double R = sqrt(r * r + dz * dz);
  zd k = S.kx[m == 0 ? 0 : 1][i][j];
  zd f;
  if (R > 0) {
    f = cexpm1(zd(0.0, -1.0) * k * R) / (4.0 * kPi * R);
  } else {
    f = (zd(0.0, -1.0) * k) / (4.0 * kPi);
  }
  zd v = S.lead_c[m][i][j] * f + res[(int64_t)ir * NC + c];
  if (m == 0 && (zs_ground.re != 0.0 || zs_ground.im != 0.0)) {
    double d = S.zl[i] + S.zl[j];
    double p = d / (2.0 * kPi * pow(r * r + d * d, 1.5));
    v += zs_ground / zd(0.0, omega * kMu0) * p;
  }
  Stab[(int64_t)c * nrho + ir] = v;
}

// Not-a-knot cubic spline of every column (scipy CubicSpline's system for
// the nodal slopes, solved by forward elimination / back substitution), as
// piecewise coefficients c[interval][p] of (r - x_i)^(3-p).
// coef layout (pair, interval, power, {A, V, W}).
// One CTA per column: radii, values and the sweep's arrays in shared memory
// (the elimination is a chain of dependent steps: it runs on one thread from
// shared memory), the coefficients of the intervals in parallel.
// Tridiagonal system a_i x_{i-1} + b_i x_i + c_i x_{i+1} = d_i, i < m (a_0 =
// c_{m-1} = 0), diagonally dominant, solved by parallel cyclic reduction
// (Hockney) with every thread of the CTA: round r combines each row with the
// rows 2^r above and below, which removes their couplings; after ceil(log2 m)
// rounds every row reads b_i x_i = d_i. A spline's rows are dominated by their
// diagonal two to one, so that the couplings fall below (2 - sqrt 3)^(2^r) of
// it: the rounds end when all are below 2^-60 and adding them would change no
// digit (six rounds instead of eight at 220 rows). Rows are kept scaled by
// their diagonal (b = 1), which leaves one division per row and round
// instead of two. Shared-memory arrays of m entries: a, b, c, d and the copies
// a2, c2, d2 (ping-pong); x receives the solution (it may be d). The
// caller synchronises before the call; the call ends with the CTA synchronised. A serial
// elimination would chain m dependent fp64 divisions; here the chain is the rounds.
template <class T>
__device__ void pcr_solve(int m, double* a, double* b, double* c, T* d, double* a2, double* c2, T* d2, T* x) {
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const double inv = 1.0 / b[i];
    a[i] *= inv;
    c[i] *= inv;
    d[i] = d[i] * inv;
  }
  __syncthreads();
  for (int st = 1; st < m; st <<= 1) {
    bool coupled = false;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      const bool lo = i - st >= 0, hi = i + st < m;
      const double ai = lo ? a[i] : 0.0, ci = hi ? c[i] : 0.0;
      const double al = lo ? a[i - st] : 0.0, cl = lo ? c[i - st] : 0.0;
      const double ah = hi ? a[i + st] : 0.0, ch = hi ? c[i + st] : 0.0;
      const double inv = 1.0 / fma(-ai, cl, fma(-ci, ah, 1.0));
      T nd = d[i];
      if (lo) nd = nd - d[i - st] * ai;
      if (hi) nd = nd - d[i + st] * ci;
      const double na = -ai * al * inv, nc = -ci * ch * inv;
      a2[i] = na;
      c2[i] = nc;
      d2[i] = nd * inv;
      coupled |= fabs(na) + fabs(nc) > 8.673617379884035e-19;  // 2^-60 of the diagonal
    }
    const int more = __syncthreads_or(coupled);
    double* t;
    t = a, a = a2, a2 = t;
    t = c, c = c2, c2 = t;
    T* td = d;
    d = d2, d2 = td;
    if (!more) break;
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) x[i] = d[i];
  __syncthreads();
}

__host__ __device__ inline size_t spline_smem(int n) { return (size_t)n * (2 * sizeof(double) + 4 * sizeof(zd)); }
// with the reduced system solved by pcr_solve (n - 2 rows)
__host__ __device__ inline size_t spline_smem_pcr(int n) {
  return (size_t)n * (2 * sizeof(double) + 3 * sizeof(zd)) + (size_t)(n - 2) * (5 * sizeof(double) + 2 * sizeof(zd));
}

// Not-a-knot cubic spline of one table column (scipy CubicSpline's slope
// form): rows a_i s_{i-1} + b_i s_i + c_i s_{i+1} = d_i for the slopes s,
// the first and last rows the not-a-knot conditions. PCR: rows 0 and n - 1
// are eliminated into rows 1 and n - 2, which leaves a strictly diagonally
// dominant system for s_1 .. s_{n-2} (pcr_solve); else (tables too long for
// its shared memory) one thread eliminates and substitutes serially.
template <bool PCR>
__global__ void __launch_bounds__(128) spline_kernel(int L, int nrho, const double* __restrict__ xg,
                                                     const zd* __restrict__ Stab, zd* __restrict__ coef) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int col = blockIdx.x;
  const int n = nrho;
  zd* y = reinterpret_cast<zd*>(smem_raw);  // (n) values
  zd* s = y + n;                            // (n) slopes
  zd* sl = s + n;                           // (n - 1) secant slopes
  double* x = reinterpret_cast<double*>(sl + n);
  double* dx = x + n;                       // (n - 1) interval widths
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    x[i] = xg[i];
    y[i] = Stab[(int64_t)col * n + i];
  }
  __syncthreads();
  // the widths and secant slopes (independent of the recurrence), in parallel
  for (int i = threadIdx.x; i < n - 1; i += blockDim.x) {
    dx[i] = x[i + 1] - x[i];
    sl[i] = (y[i + 1] - y[i]) / dx[i];
  }
  __syncthreads();
  // row i of the slope system
  auto row = [&](int i, double& a, double& b, double& c, zd& d) {
    if (i == 0) {
      const double dx0 = dx[0], dx1 = dx[1], d0 = x[2] - x[0];
      a = 0;
      b = dx1;
      c = d0;
      d = (sl[0] * ((dx0 + 2 * d0) * dx1) + sl[1] * (dx0 * dx0)) / d0;
    } else if (i == n - 1) {
      const double dxl = dx[n - 2], dxm = dx[n - 3], d1 = x[n - 1] - x[n - 3];
      a = d1;
      b = dxm;
      c = 0;
      d = (sl[n - 3] * (dxl * dxl) + sl[n - 2] * ((2 * d1 + dxl) * dxm)) / d1;
    } else {
      a = dx[i];
      b = 2 * (dx[i - 1] + dx[i]);
      c = dx[i - 1];
      d = (sl[i - 1] * dx[i] + sl[i] * dx[i - 1]) * 3.0;
    }
  };
  if constexpr (PCR) {
    const int m = n - 2;
    double* ra = dx + n;
    double* rb = ra + m;
    double* rc = rb + m;
    double* ra2 = rc + m;
    double* rc2 = ra2 + m;
    zd* rd = reinterpret_cast<zd*>(rc2 + m);
    zd* rd2 = rd + m;
    for (int i = 1 + threadIdx.x; i <= n - 2; i += blockDim.x) {
      double a, b, c;
      zd d;
      row(i, a, b, c, d);
      if (i == 1) {  // s_0 = (d_0 - c_0 s_1) / b_0
        double a0, b0, c0;
        zd d0;
        row(0, a0, b0, c0, d0);
        b -= a * c0 / b0;
        d = d - d0 * (a / b0);
        a = 0.0;
      }
      if (i == n - 2) {  // s_{n-1} = (d_{n-1} - a_{n-1} s_{n-2}) / b_{n-1}
        double al, bl, cl;
        zd dl;
        row(n - 1, al, bl, cl, dl);
        b -= c * al / bl;
        d = d - dl * (c / bl);
        c = 0.0;
      }
      ra[i - 1] = a;
      rb[i - 1] = b;
      rc[i - 1] = c;
      rd[i - 1] = d;
    }
    __syncthreads();
    pcr_solve<zd>(m, ra, rb, rc, rd, ra2, rc2, rd2, s + 1);
    if (threadIdx.x == 0) {
      double a, b, c;
      zd d;
      row(0, a, b, c, d);
      s[0] = (d - s[1] * c) / b;
      row(n - 1, a, b, c, d);
      s[n - 1] = (d - s[n - 2] * a) / b;
    }
  } else {
    zd* cp = reinterpret_cast<zd*>(dx + n);  // (n) modified diagonal (re), upper diagonal (im)
    if (threadIdx.x == 0) {
      // forward sweep
      double bprev = 0, cprev = 0;
      for (int i = 0; i < n; ++i) {
        double a, b, c;
        zd d;
        row(i, a, b, c, d);
        if (i > 0) {
          double mlt = a / bprev;
          b -= mlt * cprev;
          d -= s[i - 1] * mlt;
        }
        s[i] = d;       // holds the modified rhs
        cp[i] = zd(b);  // modified diagonal
        bprev = b;
        cprev = c;
        if (i < n - 1) cp[i].im = c;
      }
      // back substitution
      s[n - 1] = s[n - 1] / cp[n - 1].re;
      for (int i = n - 2; i >= 0; --i) s[i] = (s[i] - s[i + 1] * cp[i].im) / cp[i].re;
    }
  }
  __syncthreads();
  const int pair = col % (L * L), m = col / (L * L);
  for (int i = threadIdx.x; i < n - 1; i += blockDim.x) {
    const double h = dx[i];
    const zd si = sl[i];
    zd t = (s[i] + s[i + 1] - si * 2.0) / h;
    zd* o = coef + (((int64_t)pair * (n - 1) + i) * 4) * 3;
    o[0 * 3 + m] = t / h;
    o[1 * 3 + m] = (si - s[i]) / h - t;
    o[2 * 3 + m] = s[i];
    o[3 * 3 + m] = y[i];
  }
}

// float copies of a (na) and of b (nb)
__global__ void to_f32_kernel(const double* __restrict__ a, float* __restrict__ oa, int64_t na,
                              const double* __restrict__ b, float* __restrict__ ob, int nb) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < na)
    oa[i] = float(a[i]);
  else if (i < na + nb)
    ob[i - na] = float(b[i - na]);
}

// ------------------------------------------------------ learned remainder
// Not-a-knot cubic spline through (x_j, y_j), j < K (K >= 4), with every
// thread of the CTA: the second derivatives M_j. The end conditions (third
// derivative continuous at x_1 and x_{K-2}) give M_0 and M_{K-1} in terms of
// their neighbours; substituted into rows 1 and K - 2 they leave a strictly
// diagonally dominant tridiagonal system for M_1 .. M_{K-2}, solved by
// pcr_solve. scratch: 7 (K - 2) doubles of shared memory. The caller
// synchronises before the call; the call ends synchronised.
template <class XF, class YF>
__device__ void spline_notaknot(int K, XF x, YF y, double* M, double* scratch) {
  const int m = K - 2;  // unknowns M_1 .. M_{K-2}
  double *a = scratch, *b = a + m, *c = b + m, *d = c + m;
  double *a2 = d + m, *c2 = a2 + m, *d2 = c2 + m;
  auto h = [&](int j) { return x(j + 1) - x(j); };
  for (int k = 1 + threadIdx.x; k <= m; k += blockDim.x) {
    double ak = h(k - 1), bk = 2.0 * (h(k - 1) + h(k)), ck = h(k);
    const double dk = 6.0 * ((y(k + 1) - y(k)) / h(k) - (y(k) - y(k - 1)) / h(k - 1));
    if (k == 1) {  // M_0 = ((h_0 + h_1) M_1 - h_0 M_2) / h_1
      bk += h(0) * (h(0) + h(1)) / h(1);
      ck -= h(0) * h(0) / h(1);
      ak = 0.0;
    }
    if (k == m) {  // M_{K-1} = ((h_{K-3} + h_{K-2}) M_{K-2} - h_{K-2} M_{K-3}) / h_{K-3}
      const double p = h(K - 3), q = h(K - 2);
      ak -= q * q / p;
      bk += q * (p + q) / p;
      ck = 0.0;
    }
    a[k - 1] = ak;
    b[k - 1] = bk;
    c[k - 1] = ck;
    d[k - 1] = dk;
  }
  __syncthreads();
  pcr_solve<double>(m, a, b, c, d, a2, c2, d2, M + 1);
  if (threadIdx.x == 0) {
    M[0] = ((h(0) + h(1)) * M[1] - h(0) * M[2]) / h(1);
    M[K - 1] = ((h(K - 3) + h(K - 2)) * M[K - 2] - h(K - 2) * M[K - 3]) / h(K - 3);
  }
  __syncthreads();
}

// The cubic of interval j of a spline with second derivatives M at x.
__device__ inline double spline_eval(double x0, double x1, double y0, double y1, double M0, double M1, double xv) {
  const double h = x1 - x0, t = xv - x0;
  const double b = (y1 - y0) / h - h * (2.0 * M0 + M1) / 6.0;
  return y0 + t * (b + t * (0.5 * M0 + t * (M1 - M0) / (6.0 * h)));
}

// Learned remainder. The Sommerfeld integral has been evaluated at the ne
// radii ie[] (sorted; res holds it there): the knots (every radius below the
// near limit, then every stride-th radius and the last) at positions kpos[]
// of ie, and one validation radius in the middle of each gap between knots at
// positions vpos[]. Y: the network at every table radius (2 NC scaled
// outputs, res = scale x Y).
//
// Judge, one CTA per real column (re / im of each of the NC columns): the
// residual (integral - network) at the knots is interpolated by a not-a-knot
// spline, and the network + spline compared with the integral at the
// validation radii. colerr[2 col] = the largest error there, colerr[2 col +
// 1] = the largest |remainder| of the column's complex column over the ne
// radii. Shared memory: (2 ne + 10 nk) doubles.
__global__ void __launch_bounds__(256) sur_judge_kernel(int NC, const double* __restrict__ rho, int ne,
                                                        const int* __restrict__ ie, int nk,
                                                        const int* __restrict__ kpos, int nv,
                                                        const int* __restrict__ vpos, const float* __restrict__ Y,
                                                        const double* __restrict__ scale, const zd* __restrict__ res,
                                                        double* __restrict__ colerr) {
  extern __shared__ double sm[];
  __shared__ double red_e[8], red_s[8];
  grid_trigger();  // sur_fill_kernel starts beside this one
  const int ncol = 2 * NC, col = blockIdx.x;
  double* xs = sm;       // radius of integrated radius e
  double* ys = xs + ne;  // residual there
  double* xk = ys + ne;
  double* yk = xk + nk;
  double* M = yk + nk;
  double* scratch = M + nk;
  double smax = 0.0;
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    const int i = ie[e];
    const zd v = res[(int64_t)i * NC + (col >> 1)];
    xs[e] = rho[i];
    ys[e] = ((col & 1) ? v.im : v.re) - scale[col] * (double)Y[(int64_t)i * ncol + col];
    smax = fmax(smax, sqrt(v.re * v.re + v.im * v.im));
  }
  __syncthreads();
  for (int j = threadIdx.x; j < nk; j += blockDim.x) {
    xk[j] = xs[kpos[j]];
    yk[j] = ys[kpos[j]];
  }
  __syncthreads();
  spline_notaknot(
      nk, [&](int j) { return xk[j]; }, [&](int j) { return yk[j]; }, M, scratch);
  double emax = 0.0;
  for (int v = threadIdx.x; v < nv; v += blockDim.x) {
    const int e = vpos[v];
    const double xv = xs[e];
    int lo = 0, hi = nk - 1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (xv < xk[mid]) hi = mid; else lo = mid;
    }
    emax = fmax(emax, fabs(ys[e] - spline_eval(xk[lo], xk[lo + 1], yk[lo], yk[lo + 1], M[lo], M[lo + 1], xv)));
  }
  for (int o = 16; o; o >>= 1) {
    emax = fmax(emax, __shfl_down_sync(0xffffffffu, emax, o));
    smax = fmax(smax, __shfl_down_sync(0xffffffffu, smax, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red_e[threadIdx.x >> 5] = emax;
    red_s[threadIdx.x >> 5] = smax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double e = 0, sx = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      e = fmax(e, red_e[w]);
      sx = fmax(sx, red_s[w]);
    }
    colerr[2 * col] = e;
    colerr[2 * col + 1] = sx;
  }
}

// Decision and fill-in, one CTA per real column: accepted when the largest
// column error <= tol x the largest |remainder| (every CTA reaches the same
// decision; CTA 0 records it in flag / err_out). When accepted, the table's
// other radii ir[] get network + a not-a-knot spline of the residual through
// all ne integrated radii (a denser spline than the judged one), which is
// solved beside the judge's, before the wait for its verdict. Shared memory:
// 10 ne doubles.
__global__ void __launch_bounds__(256) sur_fill_kernel(int NC, const double* __restrict__ rho, int ne,
                                                       const int* __restrict__ ie, int nr, const int* __restrict__ ir,
                                                       const float* __restrict__ Y, const double* __restrict__ scale,
                                                       const double* colerr, double tol,
                                                       zd* __restrict__ res, int* __restrict__ flag,
                                                       double* __restrict__ err_out) {
  extern __shared__ double sm[];
  __shared__ int accepted;
  const int ncol = 2 * NC, col = blockIdx.x;
  double* xs = sm;
  double* ys = xs + ne;
  double* M = ys + ne;
  double* scratch = M + ne;
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    const int i = ie[e];
    const zd v = res[(int64_t)i * NC + (col >> 1)];
    xs[e] = rho[i];
    ys[e] = ((col & 1) ? v.im : v.re) - scale[col] * (double)Y[(int64_t)i * ncol + col];
  }
  __syncthreads();
  spline_notaknot(
      ne, [&](int e) { return xs[e]; }, [&](int e) { return ys[e]; }, M, scratch);
  grid_wait();  // the judge's errors
  if (threadIdx.x == 0) {
    double e = 0, sx = 0;
    for (int c = 0; c < ncol; ++c) {
      e = fmax(e, __ldcg(colerr + 2 * c));  // written by the kernel before, beside which this one started
      sx = fmax(sx, __ldcg(colerr + 2 * c + 1));
    }
    const double rel = sx > 0 ? e / sx : INFINITY;
    accepted = rel <= tol ? 1 : 0;
    if (blockIdx.x == 0) {
      *flag = accepted;
      *err_out = rel;
    }
  }
  __syncthreads();
  if (!accepted) return;
  for (int r = threadIdx.x; r < nr; r += blockDim.x) {
    const int i = ir[r];
    const double xv = rho[i];
    int lo = 0, hi = ne - 1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (xv < xs[mid]) hi = mid; else lo = mid;
    }
    const double v = scale[col] * (double)Y[(int64_t)i * ncol + col] +
                     spline_eval(xs[lo], xs[lo + 1], ys[lo], ys[lo + 1], M[lo], M[lo + 1], xv);
    double* out = reinterpret_cast<double*>(res + (int64_t)i * NC + (col >> 1));
    out[col & 1] = v;
  }
}

// shared memory of the two kernels above, and its limit
inline size_t sur_judge_smem(int ne, int nk) { return sizeof(double) * (2 * (size_t)ne + 10 * (size_t)nk); }
inline size_t sur_fill_smem(int ne) { return sizeof(double) * 10 * (size_t)ne; }
constexpr size_t kSurSmemMax = 200 * 1024;

int mlp_forward_device(const m25_mlp* m, int n, const float* X, float* Y, cudaStream_t st);  // mlp.cu
int mlp_dims(const m25_mlp* m, int* n_in, int* n_out);

}  // namespace m25

using namespace m25;

extern "C" int m25_greens_create(m25_ctx* ctx, const m25_greens_desc* d, m25_greens** out) {
  if (!ctx || !d || !out) {
    set_error("m25_greens_create: null argument");
    return M25_ERR_VALUE;
  }
  if (d->nlayer < 1 || d->nlayer > kMaxLayers || d->nlev < 1 || d->nlev > kMaxLev || d->nrho < 4 ||
      d->nk_c < 1 || d->nk_r < 1 || (d->single && (d->nlayer != 1 || d->nlev != 1))) {
    set_error("m25_greens_create: unsupported stack (1-8 layers, 1-3 metal levels, >= 4 radii)");
    return M25_ERR_VALUE;
  }
  for (int l = 0; l < d->nlev; ++l)
    if (d->lev_iface[l] < 1 || d->lev_iface[l] > d->nlayer || (d->top_pec && d->lev_iface[l] == d->nlayer)) {
      set_error("m25_greens_create: level interface out of range (or on the PEC cover)");
      return M25_ERR_VALUE;
    }
  if (d->top_pec && (d->single || d->nlayer < 2)) {
    set_error("m25_greens_create: a PEC cover needs a layer above the metal");
    return M25_ERR_VALUE;
  }
  M25_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  StackDev S{};
  S.nlayer = d->nlayer;
  S.nlev = d->nlev;
  S.single = d->single;
  S.top_pec = d->top_pec ? 1 : 0;
  double omega = 2.0 * kPi * d->freq;
  S.k0 = omega / kC0;
  S.h = d->stack_h;
  for (int n = 0; n < d->nlayer; ++n) {
    S.t[n] = d->layer_t[n];
    S.epsc[n] = zd(d->layer_eps[n], 0.0) * zd(1.0, -d->layer_tand[n]);
    S.kk[n] = csqrt(S.epsc[n]) * S.k0;
  }
  for (int l = 0; l < d->nlev; ++l) {
    S.il[l] = d->lev_iface[l];
    S.zl[l] = d->lev_z[l];
  }
  const int L = d->nlev, NC = 3 * L * L;
  m25_greens* g = new m25_greens();
  g->ctx = ctx;
  g->nlev = L;
  g->nrho = d->nrho;
  g->single = d->single;
  g->freq = d->freq;
  g->omega = omega;
  g->stack_h = d->stack_h;
  g->rho_h.assign(d->rho, d->rho + d->nrho);
  int rc = M25_OK;
  StackDev* Sd = nullptr;
  double *kc = nullptr, *wc = nullptr, *kr = nullptr, *wr = nullptr;
  zd *cc = nullptr, *cr = nullptr, *res = nullptr;
  std::vector<void*> tmp;
  const int n = d->nrho;
  double rmax = 0, kcmax = 0, krmax = 0;
  for (int i = 0; i < n; ++i) rmax = std::max(rmax, d->rho[i]);
  for (int q = 0; q < d->nk_c; ++q) kcmax = std::max(kcmax, d->kc[2 * q]);
  for (int q = 0; q < d->nk_r; ++q) krmax = std::max(krmax, d->kr[q]);
  const int rows_r = j0_rows(rmax * krmax, kJ0Step, kJ0Rows), rows_a = j0_rows(rmax * kcmax, kJ0ArcStep, kJ0ArcRows);
#define TRY(x)         \
  do {                 \
    rc = (x);          \
    if (rc) goto fail; \
  } while (0)
  // learned remainder: which radii get the Sommerfeld integral first
  std::vector<int> ie, kpos, vpos, ir, lists;
  if (d->surrogate) {
    int nin = 0, nout = 0;
    mlp_dims(d->surrogate, &nin, &nout);
    if (nin != 2 || nout != 2 * NC || d->sur_stride < 2 || d->sur_stride > 64 || !(d->sur_near >= 0) ||
        !d->sur_scale || !(d->sur_fmax > d->sur_fmin) || !(d->sur_a > 0) || !(d->sur_rho_ref > 0)) {
      set_error("m25_greens_create: surrogate does not match the stack (2 inputs, 2 NC outputs, stride 2-64)");
      delete g;
      return M25_ERR_VALUE;
    }
    std::vector<int> knots;
    int n0 = 0;
    while (n0 < n && d->rho[n0] < d->sur_near) knots.push_back(n0++);
    for (int i = n0; i < n; i += d->sur_stride) knots.push_back(i);
    if (knots.back() != n - 1) knots.push_back(n - 1);
    std::vector<char> exact(n, 0), val(n, 0);
    for (int i : knots) exact[i] = 1;
    for (size_t j = 0; j + 1 < knots.size(); ++j)
      if (knots[j + 1] - knots[j] >= 2) val[(knots[j] + knots[j + 1]) / 2] = 1;
    for (int i = 0; i < n; ++i) {
      if (exact[i] || val[i]) {
        if (exact[i]) kpos.push_back((int)ie.size());
        if (val[i]) vpos.push_back((int)ie.size());
        ie.push_back(i);
      } else {
        ir.push_back(i);
      }
    }
    if (kpos.size() < 4 || vpos.empty() || ir.empty() ||
        std::max(sur_judge_smem((int)ie.size(), (int)kpos.size()), sur_fill_smem((int)ie.size())) >
            kSurSmemMax) {  // the plain tabulation
      ie.clear();
      kpos.clear();
      vpos.clear();
      ir.clear();
    }
  }
  for (const std::vector<int>* l : {&ie, &kpos, &vpos, &ir}) lists.insert(lists.end(), l->begin(), l->end());
  const int ne = (int)ie.size();
  // One block for what outlives this call and one for what does not, each
  // carved up at multiples of 256 bytes, and the inputs in one copy.
  size_t keep = 0, scratch = 0;
  auto carve = [](size_t& total, size_t bytes) {
    const size_t at = total;
    total += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t o_stack = carve(keep, sizeof(StackDev)), o_rho = carve(keep, sizeof(double) * n),
               o_kc = carve(keep, sizeof(double) * 2 * d->nk_c), o_wc = carve(keep, sizeof(double) * 2 * d->nk_c),
               o_kr = carve(keep, sizeof(double) * d->nk_r), o_wr = carve(keep, sizeof(double) * d->nk_r),
               o_lists = carve(keep, sizeof(int) * lists.size()), o_scl = carve(keep, sizeof(double) * (ne ? 2 * NC : 0)),
               n_in = keep,
               o_res = carve(keep, sizeof(zd) * (size_t)n * NC), o_sur = carve(keep, 16),
               o_rho32 = carve(keep, sizeof(float) * n), o_S = carve(keep, sizeof(zd) * (size_t)NC * n),
               o_coef = carve(keep, sizeof(zd) * (size_t)L * L * (n - 1) * 12),
               o_coef32 = carve(keep, sizeof(zf) * (size_t)L * L * (n - 1) * 12);
  const int nsa = som_split_arc(d->nk_c), nsr = som_split_real(d->nk_r);
  const size_t o_cc = carve(scratch, sizeof(zd) * (size_t)d->nk_c * NC),
               o_cr = carve(scratch, sizeof(zd) * (size_t)d->nk_r * NC), o_gbig = carve(scratch, sizeof(zd) * NC),
               o_j0r = carve(scratch, sizeof(double) * kJ0Row * (size_t)rows_r),
               o_j0a = carve(scratch, sizeof(double) * kJ0ArcRow * (size_t)rows_a),
               o_part = carve(scratch, sizeof(zd) * (size_t)(nsa + nsr) * n * NC),
               o_X = carve(scratch, ne ? sizeof(float) * 2 * (size_t)n : 0),
               o_Y = carve(scratch, ne ? sizeof(float) * 2 * NC * (size_t)n : 0),
               o_colerr = carve(scratch, ne ? sizeof(double) * 2 * 2 * NC : 0);
  std::vector<char> in(n_in);
  memcpy(in.data() + o_stack, &S, sizeof(StackDev));
  memcpy(in.data() + o_rho, d->rho, sizeof(double) * n);
  memcpy(in.data() + o_kc, d->kc, sizeof(double) * 2 * d->nk_c);
  memcpy(in.data() + o_wc, d->wc, sizeof(double) * 2 * d->nk_c);
  memcpy(in.data() + o_kr, d->kr, sizeof(double) * d->nk_r);
  memcpy(in.data() + o_wr, d->wr, sizeof(double) * d->nk_r);
  if (ne) {
    memcpy(in.data() + o_lists, lists.data(), sizeof(int) * lists.size());
    memcpy(in.data() + o_scl, d->sur_scale, sizeof(double) * 2 * NC);
  }
  char *kb = nullptr, *sb = nullptr;
  zd* gbig = nullptr;
  double *j0r = nullptr, *j0a = nullptr, *part = nullptr;
  TRY(alloc_async(g->allocs, (void**)&kb, keep, st));
  TRY(alloc_async(tmp, (void**)&sb, scratch, st));
  Sd = reinterpret_cast<StackDev*>(kb + o_stack);
  g->rho = reinterpret_cast<double*>(kb + o_rho);
  kc = reinterpret_cast<double*>(kb + o_kc);
  wc = reinterpret_cast<double*>(kb + o_wc);
  kr = reinterpret_cast<double*>(kb + o_kr);
  wr = reinterpret_cast<double*>(kb + o_wr);
  g->res = res = reinterpret_cast<zd*>(kb + o_res);
  g->sur = kb + o_sur;
  g->rho32 = reinterpret_cast<float*>(kb + o_rho32);
  g->S = reinterpret_cast<decltype(g->S)>(kb + o_S);
  g->coef = reinterpret_cast<decltype(g->coef)>(kb + o_coef);
  g->coef32 = reinterpret_cast<float*>(kb + o_coef32);
  g->lead = reinterpret_cast<decltype(g->lead)>(Sd);
  cc = reinterpret_cast<zd*>(sb + o_cc);
  cr = reinterpret_cast<zd*>(sb + o_cr);
  gbig = reinterpret_cast<zd*>(sb + o_gbig);
  j0r = reinterpret_cast<double*>(sb + o_j0r);
  j0a = reinterpret_cast<double*>(sb + o_j0a);
  part = reinterpret_cast<double*>(sb + o_part);
  M25_CUDA(cudaMemcpyAsync(kb, in.data(), n_in, cudaMemcpyHostToDevice, st));
  if (d->surrogate) M25_CUDA(cudaMemsetAsync(g->sur, 0, 16, st));
  {
  const SurFeatures sf{ne ? n : 0,   g->rho,     d->sur_a,   d->sur_rho_ref,
                       d->freq,      d->sur_fmin, d->sur_fmax, reinterpret_cast<float*>(sb + o_X)};
  StageTimer tm(ctx, ST_GREENS);
  {
    const int lanes = d->single ? d->nk_c + d->nk_r : 2 * (d->nk_c + d->nk_r + 1), nb = (lanes + 63) / 64;
    spectral_g_kernel<<<nb + j0_ctas(rows_r, rows_a) + (sf.n + 63) / 64, 64, 0, st>>>(Sd, d->nk_c, kc, d->nk_r, kr, d->kbig, cc, cr,
                                                                       gbig, nb, j0r, rows_r, j0a, rows_a, sf);
    leading_kernel<<<1, 32 * L * L, 0, st>>>(Sd, d->kbig, gbig);
    spectral_coef_kernel<<<dim3((d->nk_c + d->nk_r + 63) / 64, L * L), 64, 0, st>>>(Sd, d->nk_c, kc, wc, d->nk_r, kr,
                                                                                    wr, cc, cr);
  }
  {
    // the Sommerfeld integral at the radii rho[idx[e]], e < ne (idx NULL:
    // all n) into res; skip: see sommerfeld_kernel
    auto sommerfeld = [&](int ne, const int* idx, const int* skip, bool chained = false) {
      if (ne <= 0) return;
      auto launch = [&](void (*kernel)(SomArgs), dim3 grid, const SomArgs& a) {
        if (chained)
          launch_chained(kernel, grid, 128, 0, st, a);
        else
          kernel<<<grid, 128, 0, st>>>(a);
      };
      const dim3 grid(nsa + nsr, (ne + 31) / 32);
      const SomArgs a{ne, idx, g->rho, nsa, nsr, d->nk_c, kc, cc, d->nk_r, kr, cr, j0r, j0a, rows_r, rows_a, part, skip};
      switch (NC) {
        case 3: launch(sommerfeld_kernel<3>, grid, a); break;
        case 12: launch(sommerfeld_kernel<12>, grid, a); break;
        default: launch(sommerfeld_kernel<27>, grid, a); break;
      }
      sommerfeld_sum_kernel<<<(2 * ne * NC + 31) / 32, 256, 0, st>>>(ne, NC, idx, nsa + nsr, part, res, skip);
    };
    if (!ie.empty()) {
      // the network at every radius, the Sommerfeld integral at the knots and
      // validation radii, the judge, then the integral at the other radii
      // unless the judge accepted
      const int nk = (int)kpos.size(), nv = (int)vpos.size(), nr = (int)ir.size();
      const int* dl = reinterpret_cast<const int*>(kb + o_lists);
      const double* scl = reinterpret_cast<const double*>(kb + o_scl);
      double* colerr = reinterpret_cast<double*>(sb + o_colerr);
      float* Y = reinterpret_cast<float*>(sb + o_Y);
      const int *d_ie = dl, *d_kpos = dl + ne, *d_vpos = dl + ne + nk, *d_ir = dl + ne + nk + nv;
      TRY(mlp_forward_device(d->surrogate, n, sf.X, Y, st));
      sommerfeld(ne, d_ie, nullptr, true);
      int* flag = static_cast<int*>(g->sur);
      double* err = reinterpret_cast<double*>(static_cast<char*>(g->sur) + 8);
      static const bool smem_attr =
          cudaFuncSetAttribute(sur_judge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSurSmemMax) ==
              cudaSuccess &&
          cudaFuncSetAttribute(sur_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSurSmemMax) ==
              cudaSuccess;
      if (!smem_attr) {
        set_error("m25_greens_create: the learned remainder's shared memory could not be reserved");
        rc = M25_ERR_CUDA;
        goto fail;
      }
      sur_judge_kernel<<<2 * NC, 256, sur_judge_smem(ne, nk), st>>>(NC, g->rho, ne, d_ie, nk, d_kpos, nv, d_vpos, Y,
                                                                    scl, res, colerr);
      launch_chained(sur_fill_kernel, dim3(2 * NC), dim3(256), sur_fill_smem(ne), st, NC, g->rho, ne, d_ie, nr, d_ir, Y, scl,
                     colerr, d->sur_tol, res, flag, err);
      sommerfeld(nr, d_ir, flag);  // the integral at the other radii unless the judge accepted
      g->sur_planned = ne;
    } else {
      sommerfeld(n, nullptr, nullptr);
    }
  }
  table_kernel<<<(NC * n + 127) / 128, 128, 0, st>>>(Sd, n, g->rho, res, omega, zd(d->zs_ground_re, d->zs_ground_im),
                                                   reinterpret_cast<zd*>(g->S));
  {
    const bool pcr = spline_smem_pcr(n) <= 200 * 1024;
    if (!pcr && spline_smem(n) > 200 * 1024) {
      set_error("m25_greens_create: too many tabulation radii for the spline in shared memory");
      rc = M25_ERR_VALUE;
      goto fail;
    }
    static const bool spline_attr =
        cudaFuncSetAttribute(spline_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) ==
            cudaSuccess &&
        cudaFuncSetAttribute(spline_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) ==
            cudaSuccess;
    if (!spline_attr) {
      set_error("m25_greens_create: the spline's shared memory could not be reserved");
      rc = M25_ERR_CUDA;
      goto fail;
    }
    if (pcr)
      spline_kernel<true><<<NC, 128, spline_smem_pcr(n), st>>>(L, n, g->rho, reinterpret_cast<zd*>(g->S),
                                                               reinterpret_cast<zd*>(g->coef));
    else
      spline_kernel<false><<<NC, 128, spline_smem(n), st>>>(L, n, g->rho, reinterpret_cast<zd*>(g->S),
                                                            reinterpret_cast<zd*>(g->coef));
  }
  {
    const int64_t nc = (int64_t)L * L * (n - 1) * 12 * 2;
    to_f32_kernel<<<(unsigned)((nc + n + 255) / 256), 256, 0, st>>>(g->coef, g->coef32, nc, g->rho, g->rho32, n);
  }
  }
  M25_CHECK_LAUNCH();
  // temporaries are released once the stream has consumed them
  free_all_async(tmp, st);
  {
    StackDev h;
    M25_CUDA(cudaMemcpyAsync(&h, g->lead, sizeof(StackDev), cudaMemcpyDeviceToHost, st));
    M25_CUDA(cudaStreamSynchronize(st));
    g->lead_h.resize(3 * L * L);
    g->dz_h.resize(L * L);
    for (int m = 0; m < 3; ++m)
      for (int i = 0; i < L; ++i)
        for (int j = 0; j < L; ++j) g->lead_h[(m * L + i) * L + j] = h.lead_c[m][i][j];
    for (int i = 0; i < L; ++i)
      for (int j = 0; j < L; ++j) g->dz_h[i * L + j] = h.dz[i][j];
  }
  if (d->surrogate) {
    char hs[16];
    M25_CUDA(cudaMemcpy(hs, g->sur, 16, cudaMemcpyDeviceToHost));  // the stream is idle here
    int acc;
    memcpy(&acc, hs, sizeof(int));
    memcpy(&g->sur_info[1], hs + 8, sizeof(double));
    g->sur_info[0] = acc;
    g->sur_info[2] = acc ? g->sur_planned : n;
  } else {
    g->sur_info[2] = n;
  }
  *out = g;
  return M25_OK;
fail:
  cudaStreamSynchronize(st);
  free_all_async(tmp, st);
  free_all_async(g->allocs, st);
  delete g;
  return rc;
#undef TRY
}

extern "C" int m25_greens_destroy(m25_greens* g) {
  if (!g) return M25_OK;
  free_all_async(g->allocs, g->ctx->stream);
  delete g;
  return M25_OK;
}

extern "C" int m25_greens_remainder(m25_greens* g, double* res, double* info) {
  if (!g) {
    set_error("m25_greens_remainder: null greens");
    return M25_ERR_VALUE;
  }
  M25_CUDA(cudaStreamSynchronize(g->ctx->stream));
  if (res)
    M25_CUDA(cudaMemcpy(res, g->res, sizeof(zd) * (size_t)g->nrho * 3 * g->nlev * g->nlev, cudaMemcpyDeviceToHost));
  if (info) {
    info[0] = g->sur_info[0];
    info[1] = g->sur_info[1];
    info[2] = g->sur_info[2];
  }
  return M25_OK;
}

extern "C" int m25_greens_tables(m25_greens* g, double* S, double* c, double* coef) {
  if (!g) {
    set_error("m25_greens_tables: null greens");
    return M25_ERR_VALUE;
  }
  const int L = g->nlev, n = g->nrho;
  M25_CUDA(cudaStreamSynchronize(g->ctx->stream));
  if (S) M25_CUDA(cudaMemcpy(S, g->S, sizeof(zd) * 3 * L * L * n, cudaMemcpyDeviceToHost));
  if (c)
    for (int k = 0; k < 3 * L * L; ++k) {
      c[2 * k] = g->lead_h[k].re;
      c[2 * k + 1] = g->lead_h[k].im;
    }
  if (coef) M25_CUDA(cudaMemcpy(coef, g->coef, sizeof(zd) * (size_t)L * L * (n - 1) * 12, cudaMemcpyDeviceToHost));
  return M25_OK;
}
