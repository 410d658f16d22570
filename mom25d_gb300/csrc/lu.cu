// Dense complex LU with partial pivoting and the triangular solves, the
// GPU replacement of mom25d's _dense_solve (Engine/mom25d/solver.py:11-23,
// LAPACK zgetrf / zgetrs through scipy).
//
// Right-looking blocked factorisation of a row-major matrix, per block of
// columns (64 of complex128, 128 of complex64 with tensor cores):
//   lu_panel.cu    the block's panel on one cluster of CTAs, in strips
//   panel_kernel   taller panels (above 8192 rows): cooperative grid, each CTA
//                  keeps a slice of the panel rows in shared memory; one
//                  bounded grid barrier per column (pivot search |re| + |im|
//                  as izamax, swap, scale, rank-1 update of the panel)
//   swap_trsm_kernel  the block's row interchanges on the other columns,
//                  composed into one gather, fused with U12 = L11^-1 A12
//   lu_oz.cu       complex128: A22 -= L21 U12 from exact integer slices
//   lu_tc.cu       complex64: the same in 3xTF32, in super-blocks of 256
//                  columns (the trailing matrix is read and written once per
//                  256 columns, which bounds the update)
//   gemm_kernel    complex64 without tensor cores (SIMT)
// Solve: permutation, blocked forward / backward substitution. The mixed
// path refines in fp64: r = B - Z X, X += LU32^-1 r.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "m25_internal.h"
#include "m25_lu.h"

namespace m25 {

constexpr long long kBarrierSpinLimit = 1LL << 25;  // ~1 s of polling, then give up

// Grid-wide barrier for a cooperative launch. Every wait is bounded: on
// timeout the CTA raises *err and the caller returns.
__device__ inline bool grid_sync(unsigned* count, unsigned* gen, unsigned nblocks, int* err) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* vgen = gen;
    unsigned g0 = *vgen;
    __threadfence();
    unsigned arrived = atomicAdd(count, 1u);
    if (arrived == nblocks - 1) {
      atomicExch(count, 0u);
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      long long it = 0;
      while (*vgen == g0) {
        if (++it > kBarrierSpinLimit || *(volatile int*)err) {
          atomicExch(err, 1);
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *(volatile int*)err == 0;
}

template <class T>
struct PanelArgs {
  cx<T>* A;
  int64_t lda;
  int n, k0, nb, rows_per_cta;
  int32_t* ipiv;      // absolute pivot row per factored row
  cx<T>* cand;        // (2, G, nb) candidate pivot rows
  T* candval;         // (2, G)
  int* candidx;       // (2, G)
  cx<T>* rowj;        // (2, nb) row k0+j before the swap
  unsigned* bar;      // count, generation
  int* err;           // barrier timeout
  int* info;          // first zero pivot (1-based), 0 if none
};

template <class T>
__global__ void __launch_bounds__(256) panel_kernel(PanelArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G = gridDim.x, g = blockIdx.x, nb = a.nb;
  const int r0 = a.k0 + g * a.rows_per_cta;
  const int r1 = min(a.n, r0 + a.rows_per_cta);
  const int R = max(0, r1 - r0);
  cx<T>* P = reinterpret_cast<cx<T>*>(smem_raw);      // (rows_per_cta, nb)
  cx<T>* urow = P + (size_t)a.rows_per_cta * nb;        // (nb)
  __shared__ T red_v[8];
  __shared__ int red_i[8];
  __shared__ int red_g[8];
  __shared__ int piv_sh;
  for (int e = threadIdx.x; e < R * nb; e += blockDim.x) {
    int r = e / nb, c = e % nb;
    P[e] = a.A[(int64_t)(r0 + r) * a.lda + a.k0 + c];
  }
  __syncthreads();
  for (int j = 0; j < nb; ++j) {
    const int row_j = a.k0 + j;
    const int par = j & 1;
    // local pivot candidate: max |re|+|im|, first index on ties
    T best = T(-1);
    int bi = -1;
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
      if (r0 + r < row_j) continue;
      T v = cabs1(P[r * nb + j]);
      if (v > best) {
        best = v;
        bi = r0 + r;
      }
    }
    for (int o = 16; o; o >>= 1) {
      T ov = __shfl_down_sync(0xffffffffu, best, o);
      int oi = __shfl_down_sync(0xffffffffu, bi, o);
      if (oi >= 0 && (ov > best || (ov == best && (bi < 0 || oi < bi)))) {
        best = ov;
        bi = oi;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      red_v[threadIdx.x >> 5] = best;
      red_i[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      T bv = T(-1);
      int bidx = -1;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        int oi = red_i[w];
        T ov = red_v[w];
        if (oi >= 0 && (ov > bv || (ov == bv && (bidx < 0 || oi < bidx)))) {
          bv = ov;
          bidx = oi;
        }
      }
      a.candval[par * G + g] = bv;
      a.candidx[par * G + g] = bidx;
      piv_sh = bidx;
    }
    __syncthreads();
    {
      int bidx = piv_sh;
      if (bidx >= 0)
        for (int c = threadIdx.x; c < nb; c += blockDim.x)
          a.cand[((size_t)par * G + g) * nb + c] = P[(bidx - r0) * nb + c];
      if (row_j >= r0 && row_j < r1)
        for (int c = threadIdx.x; c < nb; c += blockDim.x) a.rowj[par * nb + c] = P[(row_j - r0) * nb + c];
    }
    if (!grid_sync(a.bar, a.bar + 1, G, a.err)) return;
    // global pivot: all threads read the G candidates, then a block reduction
    {
      T bv = T(-1);
      int bidx = -1, bg = -1;
      for (int q = threadIdx.x; q < G; q += blockDim.x) {
        int oi = *(volatile int*)&a.candidx[par * G + q];
        T ov = *(volatile T*)&a.candval[par * G + q];
        if (oi >= 0 && (ov > bv || (ov == bv && (bidx < 0 || oi < bidx)))) {
          bv = ov;
          bidx = oi;
          bg = q;
        }
      }
      for (int o = 16; o; o >>= 1) {
        T ov = __shfl_down_sync(0xffffffffu, bv, o);
        int oi = __shfl_down_sync(0xffffffffu, bidx, o);
        int og = __shfl_down_sync(0xffffffffu, bg, o);
        if (oi >= 0 && (ov > bv || (ov == bv && (bidx < 0 || oi < bidx)))) {
          bv = ov;
          bidx = oi;
          bg = og;
        }
      }
      if ((threadIdx.x & 31) == 0) {
        red_v[threadIdx.x >> 5] = bv;
        red_i[threadIdx.x >> 5] = bidx;
        red_g[threadIdx.x >> 5] = bg;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      T bv = T(-1);
      int bidx = -1, bg = -1;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        int oi = red_i[w];
        T ov = red_v[w];
        if (oi >= 0 && (ov > bv || (ov == bv && (bidx < 0 || oi < bidx)))) {
          bv = ov;
          bidx = oi;
          bg = red_g[w];
        }
      }
      if (bidx < 0 || bv == T(0)) {
        if (g == 0 && *a.info == 0) *a.info = row_j + 1;
        bidx = row_j;
        bg = -1;
      }
      piv_sh = bidx;
      red_i[0] = bg;
      if (g == 0) a.ipiv[row_j] = bidx;
    }
    __syncthreads();
    const int p = piv_sh, pg = red_i[0];
    for (int c = threadIdx.x; c < nb; c += blockDim.x) {
      if (pg >= 0) {
        volatile cx<T>* src = &a.cand[((size_t)par * G + pg) * nb + c];
        urow[c] = cx<T>(src->re, src->im);
      } else if (row_j >= r0 && row_j < r1) {
        urow[c] = P[(row_j - r0) * nb + c];
      }
    }
    __syncthreads();
    if (pg < 0 && !(row_j >= r0 && row_j < r1)) {
      // zero pivot owned elsewhere: take the row from the published copy
      for (int c = threadIdx.x; c < nb; c += blockDim.x) {
        volatile cx<T>* src = &a.rowj[par * nb + c];
        urow[c] = cx<T>(src->re, src->im);
      }
      __syncthreads();
    }
    if (p != row_j) {
      if (p >= r0 && p < r1)
        for (int c = threadIdx.x; c < nb; c += blockDim.x) {
          volatile cx<T>* src = &a.rowj[par * nb + c];
          P[(p - r0) * nb + c] = cx<T>(src->re, src->im);
        }
      if (row_j >= r0 && row_j < r1)
        for (int c = threadIdx.x; c < nb; c += blockDim.x) P[(row_j - r0) * nb + c] = urow[c];
    }
    __syncthreads();
    const cx<T> piv = urow[j];
    const bool zero = piv.re == T(0) && piv.im == T(0);
    // multipliers, then the rank-1 update of the panel's remaining columns
    if (!zero)
      for (int r = threadIdx.x; r < R; r += blockDim.x)
        if (r0 + r > row_j) P[r * nb + j] = P[r * nb + j] / piv;
    __syncthreads();
    const int w = nb - j - 1;
    if (w > 0)
      for (int e = threadIdx.x; e < R * w; e += blockDim.x) {
        int r = e / w, c = j + 1 + e % w;
        if (r0 + r > row_j) P[r * nb + c] -= P[r * nb + j] * urow[c];
      }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < R * nb; e += blockDim.x) {
    int r = e / nb, c = e % nb;
    a.A[(int64_t)(r0 + r) * a.lda + a.k0 + c] = P[e];
  }
}

__device__ __forceinline__ float tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// The panel's row interchanges applied to the columns outside it, fused with
// U12 = L11^-1 A12 on the columns to its right (L11 unit lower). A CTA owns NC
// columns: it gathers the rows the interchanges touch into shared memory,
// writes them to their final rows, and on the right-hand columns runs the
// forward substitution with LPC lanes per column, each lane holding W / LPC of
// the w <= W panel rows (rows l, l + LPC, ...): at step t the lane of row t
// passes x[t] to the others by a shuffle. Every element takes its
// subtractions in the order t = 0, 1, ... as in LAPACK's ztrsm.
// complex64: 32 columns, 8 lanes each. complex128: 8 columns, 16 lanes each, as
// a warp's fp64 instruction holds its unit for 64 cycles: four times as many
// CTAs share the columns and a lane has four rows (N = 546 / 1085 / 2434 / 5943,
// all launches of a factorisation: 0.27 / 0.55 / 1.66 / 8.34 ms; 1.07 / 2.15 /
// 5.1 / 20.5 ms with 32 columns, 8 lanes and six fp64 operations per product).
// The interchanges are composed, not replayed: the rows touched are the w
// panel rows and the pivot rows below the panel, and the original row that
// ends in position x is found by applying the swaps to x in reverse order.
// (LAPACK zgetrf applies the same swaps one by one through zlaswp.)
// The CTAs cover the columns vc_begin <= vc < vc_end counted without the
// panel's (vc < k0: column vc, else column vc + w). W = 128 serves a block
// of two 64-column panels whose interchanges and L11 are taken together.
constexpr int kSwapMaxW = 64;
constexpr int kLsLd = 65;  // row stride of a 64 x 64 block of L11 in shared memory (complex elements)

template <class T>
struct SwapShape {
  static constexpr int LPC = sizeof(T) == 4 ? 8 : 16, NC = sizeof(T) == 4 ? 32 : 8;
  static constexpr int kThreads = LPC * NC;
};

// shared memory: W / 64 blocks of L11 (64 x 64, transposed) and the W gathered rows
template <class T, int W = kSwapMaxW>
__host__ __device__ constexpr size_t swap_trsm_smem() {
  return sizeof(cx<T>) * ((size_t)(W / 64) * 64 * kLsLd + (size_t)W * (SwapShape<T>::NC + 1));
}

// Lb[t * kLsLd + r] = L11[r0 + r][c0 + t] for r0 + r < w (strictly below the
// diagonal on a diagonal block), zero elsewhere; rows of A read coalesced
template <class T>
__device__ __forceinline__ void load_l_block(cx<T>* Lb, const cx<T>* A, int64_t lda, int k0, int w, int r0, int c0) {
  constexpr int kThreads = SwapShape<T>::kThreads;
#pragma unroll
  for (int b = 0; b < 64 * 64 / (16 * kThreads); ++b) {
    cx<T> v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int e = threadIdx.x + kThreads * (16 * b + k), t = e & 63, r = e >> 6;
      const bool keep = r0 + r < w && (r0 != c0 || t < r);
      v[k] = keep ? A[(int64_t)(k0 + r0 + r) * lda + k0 + c0 + t] : cx<T>();
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int e = threadIdx.x + kThreads * (16 * b + k), t = e & 63, r = e >> 6;
      Lb[t * kLsLd + r] = v[k];
    }
  }
}

// ipiv null: no interchanges (the rows are in place already); solve false:
// the interchanges alone, no U12 (and no B2). B2 rows are 2 P floats long
// ([hi | lo] planes of width P); this call writes K positions koff ..
// koff + 2 W - 1 of each plane.
template <class T, int W = kSwapMaxW>
__global__ void __launch_bounds__(SwapShape<T>::kThreads)
    swap_trsm_kernel(cx<T>* A, int64_t lda, int n, int k0, int w, const int32_t* __restrict__ ipiv,
                     float* __restrict__ B2, int P, int vc_begin, int vc_end, int koff, bool solve) {
  static_assert(W == 64 || W == 128, "panel blocks of 64 or 128 columns");
  constexpr int LPC = SwapShape<T>::LPC, NC = SwapShape<T>::NC, kLd = NC + 1;
  static_assert(W <= SwapShape<T>::kThreads, "a pivot per thread");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // L11 in 64 x 64 blocks, transposed: for W = 128 first [L11 of rows and
  // columns 0..63 | rows 64..127 x columns 0..63], then rows and columns 64..127
  // in the first buffer
  cx<T>* Ls = reinterpret_cast<cx<T>*>(smem_raw);
  cx<T>* Ls1 = Ls + (W / 64 - 1) * 64 * kLsLd;
  cx<T>* V = Ls + (W / 64) * 64 * kLsLd;  // the w panel rows of the CTA's columns [W][kLd]
  __shared__ int piv[W], dst[2 * W], src[2 * W];
  __shared__ int nd_s;
  grid_wait();
  grid_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kend = k0 + w;
  const int vc0 = vc_begin + blockIdx.x * NC;  // first column of the CTA, counted without the panel's
  // positions touched: the panel rows, then each pivot row below the panel
  // once (its first occurrence among the panel's pivots, in order); one
  // pivot per thread of the first W / 32 warps
  __shared__ int wcnt[W / 32];
  int pj = -1;
  if (threadIdx.x < W) {
    pj = (int)threadIdx.x < w ? (ipiv ? ipiv[k0 + threadIdx.x] : k0 + (int)threadIdx.x) : -1;
    piv[threadIdx.x] = pj;
  }
  __syncthreads();
  bool fst = false;
  if (threadIdx.x < W && pj >= kend) {
    fst = true;
    for (int q = 0; q < (int)threadIdx.x; ++q)
      if (piv[q] == pj) {
        fst = false;
        break;
      }
  }
  const unsigned fb = __ballot_sync(~0u, fst);
  if (warp < W / 32 && lane == 0) wcnt[warp] = __popc(fb);
  for (int i = threadIdx.x; i < w; i += blockDim.x) dst[i] = k0 + i;
  __syncthreads();
  if (fst) {
    int off = 0;
    for (int u = 0; u < warp; ++u) off += wcnt[u];
    dst[w + off + __popc(fb & ((1u << lane) - 1u))] = pj;
  }
  if (threadIdx.x == 0) {
    int nx = 0;
#pragma unroll
    for (int u = 0; u < W / 32; ++u) nx += wcnt[u];
    nd_s = w + nx;
  }
  // the CTA's columns vc0 .. vc0 + NC - 1 map to vc (< k0) or vc + w (right of the panel)
  const bool any_right = solve && kend < n && min(vc0 + NC - 1, vc_end - 1) >= k0;
  if (any_right) {
    load_l_block(Ls, A, lda, k0, w, 0, 0);
    if (W == 128) load_l_block(Ls1, A, lda, k0, w, 64, 0);
  }
  __syncthreads();
  const int nd = nd_s;
  // the original row of each touched position: the swaps applied to it in
  // reverse order, one position per thread
  for (int i = threadIdx.x; i < nd; i += blockDim.x) {
    int y = dst[i];
#pragma unroll 4
    for (int j = w - 1; j >= 0; --j) {
      const int r = k0 + j, p = piv[j];
      y = y == r ? p : (y == p ? r : y);
    }
    src[i] = y;
  }
  __syncthreads();
  const int ci = threadIdx.x % NC, ri = threadIdx.x / NC;  // rows ri, ri + LPC, ... of column ci
  const int vc = vc0 + ci;
  const bool valid = vc < vc_end;
  const int c = vc < k0 ? vc : vc + w;
  const bool right = solve && c >= kend;
  {
    // every row of the CTA's columns is read before any is written (the
    // barrier), as rows move between threads
    cx<T> v[2 * W / LPC];
#pragma unroll
    for (int j = 0; j < 2 * W / LPC; ++j) {
      const int i = ri + LPC * j;
      v[j] = valid && i < nd ? A[(int64_t)src[i] * lda + c] : cx<T>();
    }
    if (any_right)
#pragma unroll
      for (int j = 0; j < 2 * W / LPC; ++j) {
        const int i = ri + LPC * j;
        if (i < w) V[i * kLd + ci] = v[j];
      }
    __syncthreads();
    // rows that are not solved go straight to their final rows
#pragma unroll
    for (int j = 0; j < 2 * W / LPC; ++j) {
      const int i = ri + LPC * j;
      if (valid && i < nd && (i >= w || !right) && src[i] != dst[i]) A[(int64_t)dst[i] * lda + c] = v[j];
    }
  }
  if (!any_right) return;
  {
    constexpr int R = W / LPC, RB = 64 / LPC;  // rows per lane, of which in the first 64
    const int l = lane % LPC, col = threadIdx.x / LPC;
    cx<T> x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = l + LPC * k < w ? V[(l + LPC * k) * kLd + col] : cx<T>();
    // rows 0..63 (and, for W = 128, rows 64..127 take their products with
    // them); the loops over a lane's registers are unrolled, the LPC steps
    // within a group of rows are not (a fully unrolled substitution is
    // thousands of instructions, and the warps then wait on instruction fetch)
#pragma unroll
    for (int kb = 0; kb < RB; ++kb)
#pragma unroll 1
      for (int j = 0; j < LPC; ++j) {
        const int t = LPC * kb + j;
        cx<T> xt;
        xt.re = __shfl_sync(~0u, x[kb].re, (lane & ~(LPC - 1)) | j);
        xt.im = __shfl_sync(~0u, x[kb].im, (lane & ~(LPC - 1)) | j);
        // L11 rows >= w and on / above the diagonal are zero in Ls
#pragma unroll
        for (int k = kb; k < RB; ++k)
          if (k > kb || l > j) x[k] = fnma(x[k], ldc(Ls + t * kLsLd + l + LPC * k), xt);
#pragma unroll
        for (int k = RB; k < R; ++k) x[k] = fnma(x[k], ldc(Ls1 + t * kLsLd + l + LPC * (k - RB)), xt);
      }
    if (W == 128) {
      // rows 64..127 with their own diagonal block, loaded over the first one
      __syncthreads();
      load_l_block(Ls, A, lda, k0, w, 64, 64);
      __syncthreads();
#pragma unroll
      for (int kb = RB; kb < R; ++kb)
#pragma unroll 1
        for (int j = 0; j < LPC; ++j) {
          const int t = LPC * (kb - RB) + j;
          cx<T> xt;
          xt.re = __shfl_sync(~0u, x[kb].re, (lane & ~(LPC - 1)) | j);
          xt.im = __shfl_sync(~0u, x[kb].im, (lane & ~(LPC - 1)) | j);
#pragma unroll
          for (int k = kb; k < R; ++k)
            if (k > kb || l > j) x[k] = fnma(x[k], ldc(Ls + t * kLsLd + l + LPC * (k - RB)), xt);
        }
    }
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (l + LPC * k < w) V[(l + LPC * k) * kLd + col] = x[k];
  }
  __syncthreads();
  if (valid && right)
#pragma unroll
    for (int j = 0; j < W / LPC; ++j) {
      const int i = ri + LPC * j;
      if (i < w) A[(int64_t)(k0 + i) * lda + c] = V[i * kLd + ci];
    }
  if constexpr (sizeof(T) == 4)
    if (B2) {
      // U12 as the tensor-core update's B operand: for trailing column cc the
      // rows 2 cc (re, im) and 2 cc + 1 (im, -re) of (U, -iU), K-major, split
      // into tf32 hi and lo planes P floats apart, zero beyond 2 w
      for (int row = warp; row < 64; row += 8) {  // row = 2 x (column of the CTA) + part
        const int cl = row >> 1, part = row & 1;
        const int vcl = vc0 + cl;
        if (vcl >= vc_end || vcl < k0) continue;  // not a trailing column
        const int cc = vcl - k0;                  // = (vcl + w) - kend
        for (int jj = lane; jj < 2 * W; jj += 32) {
          const int t = jj >> 1, f = jj & 1;
          float hi = 0.f, lo = 0.f;
          if (t < w) {
            const cx<T> U = V[t * kLd + cl];
            const float v = part == 0 ? (f == 0 ? (float)U.re : (float)U.im) : (f == 0 ? (float)U.im : -(float)U.re);
            hi = tf32_rna(v);
            lo = tf32_rna(v - hi);
          }
          B2[(int64_t)(2 * cc + part) * 2 * P + koff + jj] = hi;
          B2[(int64_t)(2 * cc + part) * 2 * P + P + koff + jj] = lo;
        }
      }
    }
}

// C[r][c] -= sum_t Lp[r][t] Up[t][c] over rows / cols >= off, t < nb:
// 64 x 64 tile per CTA, 4 x 4 complex outputs per thread.
template <class T>
__global__ void __launch_bounds__(256) gemm_kernel(cx<T>* A, int64_t lda, int n, int k0, int nb) {
  const int off = k0 + nb;
  const int row0 = off + blockIdx.y * 64, col0 = off + blockIdx.x * 64;
  __shared__ cx<T> As[16][64 + 1];
  __shared__ cx<T> Bs[16][64];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  cx<T> acc[4][4];
  for (int t0 = 0; t0 < nb; t0 += 16) {
    for (int e = threadIdx.x; e < 16 * 64; e += 256) {
      int r = e >> 4, t = e & 15;  // As[t][r] = L[row0 + r][k0 + t0 + t]
      int gr = row0 + r, gt = t0 + t;
      As[t][r] = (gr < n && gt < nb) ? A[(int64_t)gr * lda + k0 + gt] : cx<T>();
      int t2 = e >> 6, c = e & 63;  // Bs[t][c] = U[k0 + t0 + t][col0 + c]
      int gc = col0 + c, gt2 = t0 + t2;
      Bs[t2][c] = (gc < n && gt2 < nb) ? A[(int64_t)(k0 + gt2) * lda + gc] : cx<T>();
    }
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < 16; ++t) {
      cx<T> a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[t][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[t][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j].re += a[i].re * b[j].re - a[i].im * b[j].im;
          acc[i][j].im += a[i].re * b[j].im + a[i].im * b[j].re;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int r = row0 + ty + 16 * i, c = col0 + tx + 16 * j;
      if (r < n && c < n) A[(int64_t)r * lda + c] -= acc[i][j];
    }
}

// perm[i] = the original row that the interchanges (0 p_0), (1 p_1), ... bring to
// position i (p_t >= t). Undone from the last to the first, they take position
// i to p_i and from there, at the largest s < i with p_s = p_i, to s; a row at
// s goes on to the largest r < s with p_r = s, and so on. The second kind of step is
// the same for every i: last[s], by an atomic maximum in shared memory. For the
// first each thread looks through the list once. Composing the swaps forward
// instead is one chain through shared memory (N = 5943: 235 us, here 32 us).
// STAGE: the list in shared memory too (n <= 25600).
constexpr int kPermThreads = 128;
template <bool STAGE>
__global__ void __launch_bounds__(kPermThreads) perm_kernel(int n, const int32_t* __restrict__ ipiv,
                                                            int32_t* __restrict__ perm) {
  extern __shared__ __align__(16) int perm_smem[];
  int* last = perm_smem;
  int* ps = last + ((n + 3) & ~3);
  for (int t = threadIdx.x; t < n; t += kPermThreads) last[t] = -1;
  __syncthreads();
  for (int t = threadIdx.x; t < n; t += kPermThreads) {
    const int p = ipiv[t];
    if (STAGE) ps[t] = p;
    if (p > t && p < n) atomicMax(&last[p], t);
  }
  __syncthreads();
  const int i = blockIdx.x * kPermThreads + threadIdx.x;
  if (i >= n) return;
  const int* pl = STAGE ? ps : ipiv;
  const int pi = pl[i], i0 = i & ~31;
  int x = pi > i && pi < n ? pi : i, s = -1;
  if (STAGE) {
    const int4* p4 = reinterpret_cast<const int4*>(ps);
#pragma unroll 4
    for (int t = 0; t < i0; t += 4) {
      const int4 v = p4[t >> 2];
      if (v.x == x) s = t;
      if (v.y == x) s = t + 1;
      if (v.z == x) s = t + 2;
      if (v.w == x) s = t + 3;
    }
  } else {
#pragma unroll 8
    for (int t = 0; t < i0; ++t)
      if (ipiv[t] == x) s = t;
  }
  for (int t = i0; t < i; ++t)
    if (pl[t] == x) s = t;
  for (; s >= 0; s = last[s]) x = s;
  perm[i] = x;
}

// Bp[i] = B[perm[i]] for every right-hand side
template <class T>
__global__ void gather_rows_kernel(int n, int nrhs, const int32_t* __restrict__ perm, const cx<T>* __restrict__ B,
                                   cx<T>* __restrict__ Bp) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * nrhs) return;
  int i = int(e / nrhs), c = int(e % nrhs);
  Bp[e] = B[(int64_t)perm[i] * nrhs + c];
}

// ----------------------------------------------------------------- drivers
// lu_tc.cu
int lu_tc_prepare(m25_ctx* ctx, int n);
int lu_tc_buffers(m25_ctx* ctx, int n, float** A3, float** B3, float** Ai, float** Bi);
int lu_tc_pack_a(m25_ctx* ctx, const zf* A, int64_t lda, int k0, int w, int row0, int m, int P, int pw, int koff,
                 float* A3);
int lu_tc_update(m25_ctx* ctx, zf* A, int64_t lda, int r0, int c0, int m, int nc, int P, int pw, const float* A3,
                 const float* B3, int slot);
int lu_tc_error(m25_ctx* ctx, int* flag);
bool lu_tc_available();

template <class T>
int lu_factor(m25_ctx* ctx, cx<T>* A, int64_t lda, int n, int32_t* ipiv, int nb, bool use_tc, int* info_host) {
  cudaStream_t st = ctx->stream;
  // the tensor-core update reduces into C through a TMA tensor map: rows of
  // a multiple of 16 bytes and a 16-byte aligned matrix (else SIMT updates)
  // complex128: the update by integer slices (lu_oz.cu), which needs the
  // context's operand buffer and 16-byte aligned elements
  const bool use_oz = use_tc && std::is_same<T, double>::value && !ctx->ext_scratch &&
                      reinterpret_cast<uintptr_t>(A) % 16 == 0 && nb == kSwapMaxW && n > nb;
  use_tc = use_tc && std::is_same<T, float>::value && lda % 2 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
           nb == kSwapMaxW;
  // panel workspace
  size_t panel_smem = 0;
  int G = 0;
  const size_t extra = (size_t)nb * sizeof(cx<T>);
  // pick the widest grid whose slices fit: rows_per_cta = ceil(m / G)
  auto fits = [&](int g, int m, size_t& smem) {
    int rpc = (m + g - 1) / g;
    smem = (size_t)rpc * nb * sizeof(cx<T>) + extra;
    return smem <= 200 * 1024;
  };
  M25_CUDA(cudaFuncSetAttribute(panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
  if (nb > kSwapMaxW) {
    set_error("dense LU: panel width above 64");
    return M25_ERR_VALUE;
  }
  M25_CUDA(cudaFuncSetAttribute(swap_trsm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)swap_trsm_smem<T>()));
  if constexpr (std::is_same<T, float>::value)
    M25_CUDA(cudaFuncSetAttribute(swap_trsm_kernel<T, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)swap_trsm_smem<T, 128>()));
  int Gmax = ctx->ext_scratch ? ctx->ext_gmax : 4 * ctx->num_sms;
  char* base = ctx->ext_scratch;
  if (!base) {
    int rc = ctx->scratch.ensure(sizeof(cx<T>) * 2 * (size_t)Gmax * nb + sizeof(T) * 2 * Gmax +
                                 sizeof(int) * 2 * Gmax + sizeof(cx<T>) * 2 * nb + 64);
    if (rc) return rc;
    base = ctx->scratch.as<char>();
  }
  unsigned* bar = reinterpret_cast<unsigned*>(base);
  int* err = reinterpret_cast<int*>(base + 8);
  int* info = reinterpret_cast<int*>(base + 12);
  cx<T>* cand = reinterpret_cast<cx<T>*>(base + 64);
  T* candval = reinterpret_cast<T*>(cand + 2 * (size_t)Gmax * nb);
  int* candidx = reinterpret_cast<int*>(candval + 2 * Gmax);
  cx<T>* rowj = reinterpret_cast<cx<T>*>(candidx + 2 * Gmax);
  M25_CUDA(cudaMemsetAsync(base, 0, 64, st));
  if (use_tc || use_oz) {
    int rc = use_tc ? lu_tc_prepare(ctx, n) : lu_oz_prepare(ctx, n);
    if (rc) return rc;
  }
  // blocks of up to strip_rows rows are factored by one cluster (lu_panel.cu), taller ones panel by
  // panel on a cooperative grid
  const int strip_rows = lu_strip_rows<T>(ctx);
  // M25_PANEL_CLUSTER_MIN: the smallest cluster size used (4, 8 or 16; a tuning knob)
  static const int cl_min_env = [] {
    const char* e = getenv("M25_PANEL_CLUSTER_MIN");
    const int v = e ? atoi(e) : 8;
    return v >= 16 ? 16 : v >= 8 ? 8 : 4;
  }();
  // the context's setting (m25_ctx_set_tuning) over the process default
  const int cl_min = ctx->tune_cluster_min >= 16 ? 16
                     : ctx->tune_cluster_min >= 8 ? 8
                     : ctx->tune_cluster_min > 0  ? 4
                                                  : cl_min_env;
  // one panel of w <= nb columns at k0 over the rows k0 .. n - 1 on a cooperative grid
  auto run_panel = [&](int k0, int w) -> int {
    const int m = n - k0;
    // grid size: as many CTAs as can be co-resident, each with >= 1 row
    int occ = 0;
    G = std::min(std::min(m, ctx->num_sms), Gmax);
    // M25_PANEL_CTAS: fixed panel grid (a tuning knob; 0 or unset = automatic)
    static const int forced = getenv("M25_PANEL_CTAS") ? atoi(getenv("M25_PANEL_CTAS")) : 0;
    if (forced > 0) G = std::min(std::min(m, forced), Gmax);
    fits(G, m, panel_smem);
    // fewest CTAs (one per SM) whose row slices fit: the per-column barrier
    // and pivot reduction cost grow with the grid
    for (int bps = 1; bps <= 4 && forced <= 0; ++bps) {
      int g = std::min(m, bps * ctx->num_sms);
      size_t smem;
      if (g > Gmax || !fits(g, m, smem)) continue;
      M25_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, panel_kernel<T>, 256, smem));
      if (occ * ctx->num_sms >= g) {
        G = g;
        panel_smem = smem;
        break;
      }
    }
    if (!fits(G, m, panel_smem)) {
      set_error("dense LU: matrix too large for the panel slices in shared memory");
      return M25_ERR_VALUE;
    }
    M25_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, panel_kernel<T>, 256, panel_smem));
    if (occ * ctx->num_sms < G) {
      set_error("dense LU: cooperative panel grid does not fit on the device");
      return M25_ERR_VALUE;
    }
    PanelArgs<T> pa;
    pa.A = A;
    pa.lda = lda;
    pa.n = n;
    pa.k0 = k0;
    pa.nb = w;
    pa.rows_per_cta = (m + G - 1) / G;
    pa.ipiv = ipiv;
    pa.cand = cand;
    pa.candval = candval;
    pa.candidx = candidx;
    pa.rowj = rowj;
    pa.bar = bar;
    pa.err = err;
    pa.info = info;
    void* args[] = {&pa};
    StageTimer tm(ctx, ST_PANEL);
    M25_CUDA(cudaLaunchCooperativeKernel((void*)panel_kernel<T>, dim3(G), dim3(256), args, panel_smem, st));
    return M25_OK;
  };
  // interchanges of the panel at k0 (width w) on the columns vc_begin <= vc <
  // vc_end (counted without the panel's), U12 on those right of it
  auto swap_trsm = [&](int k0, int w, int vc_begin, int vc_end, float* B2, int P2) -> int {
    if (vc_end <= vc_begin) return M25_OK;
    StageTimer tm(ctx, ST_TRSM);
    using Sw = SwapShape<T>;
    M25_CUDA(launch_chained(swap_trsm_kernel<T, kSwapMaxW>, dim3((vc_end - vc_begin + Sw::NC - 1) / Sw::NC), Sw::kThreads,
                            swap_trsm_smem<T>(), st, A, lda, n, k0, w, (const int32_t*)ipiv, B2, P2, vc_begin, vc_end,
                            0, true));
    return M25_OK;
  };
  // the same for a block of w <= 128 columns (two panels' interchanges and a
  // 128-row L11 at once): piv null skips the interchanges, solve false skips
  // U12; B planes of width P at K offset koff
  auto swap_trsm128 = [&](int k0, int w, int vc_begin, int vc_end, float* B2, int P, int koff, const int32_t* piv,
                          bool solve) -> int {
    if (vc_end <= vc_begin) return M25_OK;
    StageTimer tm(ctx, ST_TRSM);
    using Sw = SwapShape<T>;
    M25_CUDA(launch_chained(swap_trsm_kernel<T, 128>, dim3((vc_end - vc_begin + Sw::NC - 1) / Sw::NC), Sw::kThreads,
                            swap_trsm_smem<T, 128>(), st, A, lda, n, k0, w, piv, B2, P, vc_begin, vc_end, koff, solve));
    return M25_OK;
  };
  int rc = M25_OK;
  if (!use_tc) {
    // right-looking: panel, interchanges and U12, update of the trailing matrix
    for (int k0 = 0; k0 < n; k0 += nb) {
      const int w = std::min(nb, n - k0);
      if (n - k0 <= strip_rows) rc = lu_strip_block<T>(ctx, A, lda, n, k0, w, ipiv, info, err, cand, cl_min);
      else rc = run_panel(k0, w);
      if (rc) return rc;
      if ((rc = swap_trsm(k0, w, 0, n - w, nullptr, 0))) return rc;
      if (k0 + w >= n) break;
      if constexpr (std::is_same<T, double>::value) {
        // nb = 64 here: k0 + w < n
        if ((rc = use_oz ? lu_oz_update(ctx, A, lda, n, k0) : lu_oz_update_simt(ctx, A, lda, n, k0, cand))) return rc;
      } else {
        const int ncol = n - k0 - w;
        StageTimer tm(ctx, ST_GEMM);
        dim3 grid((ncol + 63) / 64, (ncol + 63) / 64);
        gemm_kernel<T><<<grid, 256, 0, st>>>(A, lda, n, k0, w);
        M25_CHECK_LAUNCH();
      }
    }
  } else if constexpr (std::is_same<T, float>::value) {
    // super-blocks of 256 columns: two blocks a, b of 128, each factored as
    // two panels of 64 (the first panel's rank-64 update of the second's
    // columns). Block a's interchanges and U_a = L_aa^-1 A_a go to every
    // column right of it, its rank-128 update only to block b's columns;
    // block b is factored; on the trailing columns then block b's
    // interchanges, its rows minus L_ba U_a, U_b = L_bb^-1 of those rows, and
    // one rank-256 update of the trailing matrix: its read-modify-write of C,
    // the bound of the update, once per 256 columns. B3 holds U_a at K
    // 0..255 and U_b at K 256..511 of planes 512 floats wide, for the columns
    // from the first right of block a (block b's, then the trailing ones).
    float *A3, *B3, *Ai, *Bi;
    if ((rc = lu_tc_buffers(ctx, n, &A3, &B3, &Ai, &Bi))) return rc;
    constexpr int kHalf = kSwapMaxW, kBlock = 2 * kSwapMaxW, kSuper = 2 * kBlock, kPW = 2 * kSuper;
    int slot = 0;
    // one block of W <= 128 columns at c0. By one cluster: *left false, its
    // interchanges are still to be applied to every other column. Taller
    // ones: both panels, the first one's U12 and rank-64 update on the second
    // one's columns, each panel's interchanges on every column left of it
    // (none on columns right of the block), *left true
    auto factor_block = [&](int c0, int W, bool* left) -> int {
      *left = n - c0 > strip_rows;
      if (!*left) return lu_strip_block<T>(ctx, A, lda, n, c0, W, ipiv, info, err, cand, cl_min);
      const int w1 = std::min(kHalf, W), w2 = W - w1;
      int r;
      if ((r = run_panel(c0, w1))) return r;
      if (w2 == 0) return swap_trsm(c0, w1, 0, c0, nullptr, 0);
      if ((r = swap_trsm(c0, w1, 0, c0 + w2, Bi, 128))) return r;
      const int m1 = n - c0 - w1;
      if ((r = lu_tc_pack_a(ctx, A, lda, c0, w1, c0 + w1, m1, 128, 128, 0, Ai))) return r;
      if ((r = lu_tc_update(ctx, A, lda, c0 + w1, c0 + w1, m1, w2, 128, 128, Ai, Bi, slot++))) return r;
      if ((r = run_panel(c0 + w1, w2))) return r;
      return swap_trsm(c0 + w1, w2, 0, c0 + w1, nullptr, 0);
    };
    for (int k0 = 0; k0 < n; k0 += kSuper) {
      const int SW = std::min(kSuper, n - k0), wa = std::min(kBlock, SW), wb = SW - wa;
      bool left;
      if ((rc = factor_block(k0, wa, &left))) return rc;
      const int ra = k0 + wa;  // first column (and row) right of block a
      // block a's interchanges (on the columns left of it too, where they are
      // still due) and U_a on every column right of it
      if ((rc = swap_trsm128(k0, wa, left ? k0 : 0, n - wa, B3, kPW, 0, ipiv, true))) return rc;
      if (ra >= n) break;  // (then wb = 0)
      // block a's rank-128 update of block b's columns
      if ((rc = lu_tc_pack_a(ctx, A, lda, k0, wa, ra, n - ra, 2 * kBlock, kPW, 0, A3))) return rc;
      if ((rc = lu_tc_update(ctx, A, lda, ra, ra, n - ra, wb, 2 * kBlock, kPW, A3, B3, slot++))) return rc;
      if ((rc = factor_block(ra, wb, &left))) return rc;
      const int t0 = k0 + SW, nt = n - t0;  // the trailing columns
      float* Bt = B3 + (size_t)2 * wb * 2 * kPW;  // B rows of the trailing columns
      // block b's interchanges on the other columns
      if ((rc = swap_trsm128(ra, wb, left ? ra : 0, ra + nt, nullptr, 0, 0, ipiv, false))) return rc;
      if (nt <= 0) continue;
      // block b's rows of the trailing columns minus L_ba U_a
      if ((rc = lu_tc_pack_a(ctx, A, lda, k0, wa, ra, wb, 2 * kBlock, kPW, 0, A3))) return rc;
      if ((rc = lu_tc_update(ctx, A, lda, ra, t0, wb, nt, 2 * kBlock, kPW, A3, Bt, slot++))) return rc;
      // U_b = L_bb^-1 of those rows, its B planes at K 256..511
      if ((rc = swap_trsm128(ra, wb, ra, ra + nt, Bt, kPW, 2 * kBlock, nullptr, true))) return rc;
      // the rank-256 update of the trailing matrix
      if ((rc = lu_tc_pack_a(ctx, A, lda, k0, SW, t0, nt, kPW, kPW, 0, A3))) return rc;
      if ((rc = lu_tc_update(ctx, A, lda, t0, t0, nt, nt, kPW, kPW, A3, Bt, slot++))) return rc;
    }
  }
  int hflags[3];
  M25_CUDA(cudaMemcpyAsync(hflags, base + 8, 8, cudaMemcpyDeviceToHost, st));
  M25_CUDA(cudaStreamSynchronize(st));
  if (hflags[0]) {
    set_error("dense LU: a wait of the panel factorisation ran out");
    return M25_ERR_CUDA;
  }
  if (use_tc || use_oz) {
    int tcerr = 0;
    int rc = lu_tc_error(ctx, &tcerr);
    if (rc) return rc;
    if (tcerr) {
      set_error("dense LU: a wait of the tensor-core update ran out");
      return M25_ERR_CUDA;
    }
  }
  *info_host = hflags[1];
  return M25_OK;
}

constexpr long long kFlagSpinLimit = 1LL << 24;  // bounded wait on a block's ready flag

template <class TF, class TV>
struct WaveArgs {
  const cx<TF>* A;
  int64_t lda;
  int n, nrhs, upper;
  cx<TV>* X;       // in: permuted right-hand sides; out: the solution of this sweep
  int* flags;      // (nblk) == epoch once block k of X is final (complex128 vectors)
  int epoch;
  int* err;        // a wait ran out
  long long spins; // polls per wait before it gives up
  // complex64 vectors: the solved values published with the sweep's epoch in
  // every 8-byte word, (epoch << 32) | bits of re, then the same for im, so
  // a reader can poll the data itself (aligned 8-byte accesses are single-copy
  // atomic); replaces the ready flags and their fences
  unsigned long long* Yt;
};

// asynchronous global -> shared copy of one element (8 or 16 bytes); a
// column outside the matrix is zero-filled without reading global memory
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* dst, const void* src, bool valid) {
  unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  int n = valid ? BYTES : 0;
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Rows of a block of the triangular sweeps. complex64: 64, as a step's latencies (the flag, the
// barriers) bound the chain. complex128: 32, as the fp64 operations on the chain do - the
// substitution and the last tile's product, both of which halve per row - and the
// rest of a block's products runs beside it (N = 546 / 1085 / 2434 / 5943, all sweeps of a solve with
// two right-hand sides: 0.49 / 0.91 / 2.03 / 5.1 ms, 0.63 / 1.19 / 2.71 / 6.45 ms with 64).
template <class TV>
__host__ __device__ constexpr int wave_b() { return sizeof(TV) == 8 ? 32 : 64; }
template <int B>
constexpr int kTileLd = B + 1;  // padded row of a tile in shared memory

// fetch the w x B tile at (r0, c0) (columns >= wc zero) into a (B, B + 1) shared buffer; one commit group
template <int B, class TF>
__device__ __forceinline__ void fetch_tile(cx<TF>* dst, const cx<TF>* A, int64_t lda, int r0, int c0, int w, int wc) {
  for (int e = threadIdx.x; e < w * B; e += blockDim.x) {
    int r = e / B, c = e % B;
    const cx<TF>* src = A + (int64_t)(r0 + r) * lda + c0 + (c < wc ? c : 0);
    cp_async_elem<sizeof(cx<TF>)>(&dst[r * kTileLd<B> + c], src, c < wc);
  }
  cp_async_commit();
}

// the diagonal w x w tile at (r0, r0), transposed: DgT[c * (B + 1) + r] = A[r0 + r][r0 + c]; one commit group
template <int B, class TF>
__device__ __forceinline__ void fetch_diag_t(cx<TF>* DgT, const cx<TF>* A, int64_t lda, int r0, int w) {
  for (int e = threadIdx.x; e < w * B; e += blockDim.x) {
    int r = e / B, c = e % B;
    const cx<TF>* src = A + (int64_t)(r0 + r) * lda + r0 + (c < w ? c : 0);
    cp_async_elem<sizeof(cx<TF>)>(&DgT[c * kTileLd<B> + r], src, c < w);
  }
  cp_async_commit();
}

// Substitution on the diagonal block by one warp for one right-hand side c,
// in registers: lane l owns the rows 2l and 2l + 1, so each round the owner of
// a pair of rows solves both locally and broadcasts them with one round of
// shuffles (32 rounds for 64 rows). DgT is the transposed diagonal tile
// already masked to the triangle of this sweep (zeros elsewhere and outside
// the block), dinv the reciprocal diagonal (zero outside the block), so the
// rounds load factors without any test. Lower: unit diagonal, forward; upper:
// backward. acc (rows x P) in and out, column c.
// The rounds have no test for the owner: its own factors are zero on and
// beyond the diagonal, so that its rows take the right subtractions too (and
// are scaled by the reciprocal diagonal at the end); a select per round made it
// divergent, 180 cycles a round against 83. Rounds beyond the block's rows
// change nothing.
template <class TF>
__device__ __forceinline__ void diag_solve1(int lane, int w, int P, int c, int upper, const cx<TF>* DgT,
                                            const zf* dinv, zf* acc) {
  using TV = float;
  const int ra = 2 * lane, rb = ra + 1;
  cx<TV> va = ra < w ? acc[ra * P + c] : cx<TV>();
  cx<TV> vb = rb < w ? acc[rb * P + c] : cx<TV>();
  auto bcast = [](cx<TV> v, int k) { return cx<TV>(__shfl_sync(0xffffffffu, v.re, k), __shfl_sync(0xffffffffu, v.im, k)); };
  const cx<TV> da = upper ? ldc(dinv + ra) : cx<TV>(), db = upper ? ldc(dinv + rb) : cx<TV>();
  if (!upper) {
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
      const cx<TF>*ca = DgT + (2 * k) * kTileLd<64>, *cb = ca + kTileLd<64>;  // columns 2 k, 2 k + 1
      const cx<TV> aA(ca[ra]), bA(ca[rb]), aB(cb[ra]), bB(cb[rb]);
      // owner (lane k): x_2k is final, x_2k+1 = v_2k+1 - L[2k+1][2k] x_2k
      const cx<TV> xa = bcast(va, k), xb = bcast(fnma(vb, bA, va), k);
      va = fnma(fnma(va, aA, xa), aB, xb);
      vb = fnma(fnma(vb, bA, xa), bB, xb);
    }
  } else {
#pragma unroll 4
    for (int k = 31; k >= 0; --k) {
      const cx<TF>*ca = DgT + (2 * k) * kTileLd<64>, *cb = ca + kTileLd<64>;
      const cx<TV> aA(ca[ra]), bA(ca[rb]), aB(cb[ra]), bB(cb[rb]);
      // owner: x_2k+1 = v_2k+1 / d, then x_2k = (v_2k - U[2k][2k+1] x_2k+1) / d
      const cx<TV> ob = vb * db, oa = fnma(va, aB, ob) * da;
      const cx<TV> xa = bcast(oa, k), xb = bcast(ob, k);
      va = fnma(fnma(va, aB, xb), aA, xa);
      vb = fnma(fnma(vb, bB, xb), bA, xa);
    }
  }
  if (upper) {
    va = va * da;
    vb = vb * db;
  }
  if (ra < w) acc[ra * P + c] = va;
  if (rb < w) acc[rb * P + c] = vb;
}

// complex128, 32 rows: lane l owns row l, a column per round (the fp64 operations bound it: four a round, eight
// for the upper factor, whose solved value every lane forms).
template <class TF>
__device__ __forceinline__ void diag_solve1(int lane, int w, int P, int c, int upper, const cx<TF>* DgT,
                                            const zd* dinv, zd* acc) {
  zd v = lane < w ? acc[lane * P + c] : zd();
  auto bcast = [](zd u, int k) { return zd(__shfl_sync(0xffffffffu, u.re, k), __shfl_sync(0xffffffffu, u.im, k)); };
  const zd d = upper ? ldc(dinv + lane) : zd();
  if (!upper) {
#pragma unroll 4
    for (int k = 0; k < 32; ++k) v = fnma(v, zd(DgT[k * kTileLd<32> + lane]), bcast(v, k));
  } else {
#pragma unroll 4
    for (int k = 31; k >= 0; --k) v = fnma(v, zd(DgT[k * kTileLd<32> + lane]), bcast(v * d, k));
    v = v * d;
  }
  if (lane < w) acc[lane * P + c] = v;
}

// tiles in flight per CTA: 4 complex64 or 2 complex128 tiles
template <class TF>
constexpr int wave_stages() {
  return sizeof(cx<TF>) == 8 ? 4 : 2;
}
constexpr int kYtWords = 64 * 8 * 2;  // tagged words of one block of y (64 rows, up to 8 right-hand sides)
template <class TF, class TV>
constexpr size_t wave_smem() {
  constexpr int B = wave_b<TV>();
  return sizeof(cx<TF>) * B * kTileLd<B> * (1 + wave_stages<TF>()) + sizeof(cx<TV>) * (B * 8 * 2 + B) +
         (sizeof(TV) == 4 ? sizeof(unsigned long long) * kYtWords * wave_stages<TF>() : 0);
}

// One triangular sweep as a dependency wavefront (no grid barriers): CTA g
// owns the blocks g, g + G, ... of wave_b rows. For its block i it subtracts the
// tile products A_ij y_j of the blocks j it depends on (j < i for the unit
// lower factor, j > i for the upper one, in the order they become final) as
// soon as block j is flagged final, solves the diagonal block by
// substitution, publishes y_i and raises flag i. The off-diagonal tiles
// stream through a ring of cp.async stages so that a CTA's backlog of tiles
// never holds up the chain; the chain step itself is the flag round trip,
// one tile product and the substitution, which one warp runs in
// registers (complex64: lane l owns rows 2l and 2l + 1; each solved pair is broadcast with
// shuffles; the upper sweep multiplies by the reciprocal diagonal). It is
// bound by that chain, not by the factors' bytes: all sweeps of a solve, two
// right-hand sides, N = 1085 / 3789 / 5943 in complex64 0.35 / 1.85 / 1.69 ms
// (0.46 / 2.51 / 2.33 ms with a select per round and one lane per row of the
// tile product), N = 546 / 2434 / 5943 in complex128 0.49 / 2.03 / 5.1 ms (0.90 /
// 3.96 / 9.6 ms, and blocks of 64 rows). Every
// wait is bounded; blocks only wait on blocks solved earlier, and the
// cooperative launch keeps all CTAs resident, so the order cannot deadlock.
template <class TF, class TV>
__global__ void __launch_bounds__(256, 1) trsv_wave_kernel(WaveArgs<TF, TV> a) {
  constexpr int S = wave_stages<TF>(), B = wave_b<TV>(), LD = kTileLd<B>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<TF>* Dg = reinterpret_cast<cx<TF>*>(smem_raw);  // (B, B + 1) diagonal tile, transposed
  cx<TF>* ring = Dg + B * LD;                   // S x (B, B + 1) off-diagonal tiles
  cx<TV>* acc = reinterpret_cast<cx<TV>*>(ring + S * B * LD);  // (B, P)
  cx<TV>* y = acc + B * 8;                                            // (B, P)
  cx<TV>* dinv = y + B * 8;                                           // (B) reciprocal diagonal
  constexpr bool kTagged = sizeof(TV) == 4;
  unsigned long long* yring = reinterpret_cast<unsigned long long*>(dinv + B);  // S x kYtWords (tagged)
  const unsigned tag = (unsigned)a.epoch;
  __shared__ int fail;
  const int G = gridDim.x, P = a.nrhs, tid = threadIdx.x;
  const int nblk = (a.n + B - 1) / B;
  if (tid == 0) fail = 0;
  __syncthreads();
  for (int q = blockIdx.x; q < nblk; q += G) {
    const int i = a.upper ? nblk - 1 - q : q;
    const int r0 = i * B, w = min(B, a.n - r0);
    // dependencies in the order they become final: j = 0 .. i-1 (lower) or nblk-1 .. i+1 (upper)
    const int ndep = a.upper ? nblk - 1 - i : i;
    auto dep = [&](int d) { return a.upper ? nblk - 1 - d : d; };
    // the tile of dependency d (and, for tagged vectors, the published y_j as
    // it stands now) into ring slot d % S; one commit group per dependency
    auto fetch_dep = [&](int d) {
      const int j = dep(d), wj = min(B, a.n - j * B);
      if constexpr (kTagged) {
        unsigned long long* ys = yring + (d % S) * kYtWords;
        for (int e = threadIdx.x; e < wj * P; e += blockDim.x)  // 16 bytes = one complex value, L2 only
          cp_async_elem<16>(ys + 2 * e, a.Yt + ((int64_t)j * B * P + e) * 2, true);
      }
      fetch_tile<B>(ring + (d % S) * B * LD, a.A, a.lda, r0, j * B, w, wj);
    };
    // commit groups: the diagonal tile, then one per dependency (dependency d is group d + 1)
    fetch_diag_t<B>(Dg, a.A, a.lda, r0, w);
    for (int d = 0; d < S; ++d) {
      if (d < ndep) fetch_dep(d);
      else cp_async_commit();
    }
    for (int e = tid; e < w * P; e += blockDim.x) acc[e] = a.X[(int64_t)r0 * P + e];
    // reciprocal diagonal (zero outside the block), then the tile masked to
    // this sweep's triangle (zero elsewhere); the first step's barrier
    // separates the two, the next barrier publishes the result
    auto prep_diag = [&]() {
      if (tid < B) {
        cx<TV> di;
        if (a.upper && tid < w) {
          const cx<TV> dd(Dg[tid * LD + tid]);
          const TV m2 = dd.re * dd.re + dd.im * dd.im;
          di = cx<TV>(dd.re / m2, -dd.im / m2);
        }
        dinv[tid] = di;
      }
      __syncthreads();
      for (int e = tid; e < B * B; e += blockDim.x) {
        const int col = e / B, r = e % B;
        const bool keep = r < w && col < w && (a.upper ? r < col : r > col);
        if (!keep) Dg[col * LD + r] = cx<TF>();
      }
    };
    for (int d = 0; d < ndep; ++d) {
      const int j = dep(d), c0 = j * B, wj = min(B, a.n - c0);
      const cx<TF>* T = ring + (d % S) * B * LD;
      if constexpr (kTagged) {
        cp_async_wait<S - 1>();  // tile d and the prefetched y_j have landed
        __syncthreads();
        if (d == 0) prep_diag();  // the diagonal tile (group 0) is in: mask it while the chain runs
        // words of y_j not yet final when prefetched are polled until they carry this sweep's tag
        const unsigned long long* ys = yring + (d % S) * kYtWords;
        bool bad = false;
        for (int e = tid; e < B * P * 2; e += blockDim.x) {
          float f = 0.f;
          if (e < wj * P * 2) {
            unsigned long long v = ys[e];
            if ((unsigned)(v >> 32) != tag) {
              const volatile unsigned long long* g = a.Yt + (int64_t)j * B * P * 2 + e;
              long long it = 0;
              while (true) {
                v = *g;
                if ((unsigned)(v >> 32) == tag) break;
                if (++it > a.spins || *(volatile int*)a.err) {
                  bad = true;
                  break;
                }
                __nanosleep(20);
              }
            }
            f = __uint_as_float((unsigned)v);
          }
          if (e & 1) y[e >> 1].im = f;
          else y[e >> 1].re = f;
        }
        if (__syncthreads_or(bad)) {
          if (tid == 0) atomicExch(a.err, 1);
          cp_async_wait<0>();
          return;
        }
      } else {
        if (tid == 0) {
          long long it = 0;
          while (*(volatile int*)&a.flags[j] != a.epoch) {
            if (++it > a.spins || *(volatile int*)a.err) {
              atomicExch(a.err, 1);
              fail = 1;
              break;
            }
            __nanosleep(32);
          }
          __threadfence();
        }
        cp_async_wait<S - 1>();  // tile d has landed
        __syncthreads();
        if (d == 0) prep_diag();
        if (fail) {
          cp_async_wait<0>();
          return;
        }
        for (int e = tid; e < B * P; e += blockDim.x) {
          if (e < wj * P) {
            volatile cx<TV>* src = &a.X[(int64_t)c0 * P + e];
            y[e] = cx<TV>(src->re, src->im);
          } else {
            y[e] = cx<TV>();
          }
        }
        __syncthreads();
      }
      // the tile's product: kL lanes per row, kC columns each, two right-hand
      // sides at a time. The lanes start at different columns so that a half
      // warp's loads fall into different banks
      {
        constexpr int kL = 256 / B, kC = B / kL;
        const int part = tid & (kL - 1), r = (unsigned)tid / kL;
        const cx<TF>* Tr = T + r * LD + kC * part;
        for (int c = 0; c < P; c += 2) {
          const bool two = c + 1 < P;
          const cx<TV>* yc = y + kC * part * P + c;
          cx<TV> s[2][2];  // minus the product, in two sums per right-hand side
#pragma unroll 8
          for (int i = 0; i < kC; ++i) {
            const int t = (i + 4 * part) & (kC - 1);
            const cx<TV> tv(ldc(Tr + t));
            s[0][i & 1] = fnma(s[0][i & 1], tv, ldc(yc + t * P));
            if (two) s[1][i & 1] = fnma(s[1][i & 1], tv, ldc(yc + t * P + 1));
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (q && !two) break;
            cx<TV> v = s[q][0] + s[q][1];
#pragma unroll
            for (int o = 1; o < kL; o <<= 1) {
              v.re += __shfl_xor_sync(0xffffffffu, v.re, o);
              v.im += __shfl_xor_sync(0xffffffffu, v.im, o);
            }
            if (part == 0 && r < w) acc[r * P + c + q] += v;
          }
        }
      }
      __syncthreads();  // the stage of tile d is free again
      if (d + S < ndep) fetch_dep(d + S);
      else cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();
    if (ndep == 0) {
      prep_diag();
      __syncthreads();
    }
    // diagonal block: warp c solves right-hand side c (P <= 8 warps in parallel)
    const int warp = tid >> 5, lane = tid & 31;
    if (warp < P) diag_solve1(lane, w, P, warp, a.upper, Dg, dinv, acc);
    __syncthreads();
    // publish y_i (warp 0)
    if (tid < 32) {
      if constexpr (kTagged) {
        // publish first (the chain waits on it), then the plain copy for the next sweep
        const unsigned long long hi = (unsigned long long)tag << 32;
        volatile unsigned long long* yt = a.Yt + (int64_t)r0 * P * 2;
        for (int e = lane; e < w * P; e += 32) {
          const cx<TV> v = acc[e];
          yt[2 * e] = hi | __float_as_uint((float)v.re);
          yt[2 * e + 1] = hi | __float_as_uint((float)v.im);
        }
      }
      for (int e = lane; e < w * P; e += 32) a.X[(int64_t)r0 * P + e] = acc[e];
      if constexpr (!kTagged) __threadfence();
    }
    __syncthreads();
    if constexpr (!kTagged) {
      if (tid == 0) atomicExch(&a.flags[i], a.epoch);
    }
  }
}

// perm (n ints, device) of the interchanges in ipiv; once per factorisation
int lu_make_perm(m25_ctx* ctx, int n, const int32_t* ipiv, int32_t* perm) {
  if ((size_t)n * sizeof(int) > 200 * 1024) {
    set_error("dense solve: n <= 51200");
    return M25_ERR_VALUE;
  }
  static const bool attr =
      cudaFuncSetAttribute(perm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 201 * 1024) ==
          cudaSuccess &&
      cudaFuncSetAttribute(perm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 201 * 1024) ==
          cudaSuccess;
  if (!attr) {
    set_error("dense solve: the permutation kernel's shared memory could not be reserved");
    return M25_ERR_CUDA;
  }
  const size_t sm = sizeof(int) * ((size_t)(n + 3) & ~(size_t)3);
  const unsigned g = (unsigned)((n + kPermThreads - 1) / kPermThreads);
  if (2 * sm <= 200 * 1024)
    perm_kernel<true><<<g, kPermThreads, 2 * sm, ctx->stream>>>(n, ipiv, perm);
  else
    perm_kernel<false><<<g, kPermThreads, sm, ctx->stream>>>(n, ipiv, perm);
  M25_CHECK_LAUNCH();
  return M25_OK;
}

// X = (LU)^-1 P B: the permutation (from ipiv, or the precomputed perm when
// given), then one wavefront launch per factor. wide: on as many CTAs as there
// are blocks, whatever the cap.
template <class TF, class TV>
int lu_solve_wave(m25_ctx* ctx, const cx<TF>* A, int64_t lda, int n, const int32_t* ipiv, const cx<TV>* B, int nrhs,
                  cx<TV>* X, const int32_t* perm, bool wide) {
  cudaStream_t st = ctx->stream;
  if (nrhs > 8 || (size_t)n * sizeof(int) > 200 * 1024) {
    set_error("dense solve: at most 8 right-hand sides and n <= 51200");
    return M25_ERR_VALUE;
  }
  constexpr int kB = wave_b<TV>();
  const int nblk = (n + kB - 1) / kB;
  // layout: [0] wait error, [16 ..] ready flag per block, then the
  // permutation when it is built here; zeroed whenever the buffer is
  // (re)allocated (a caller-provided buffer comes zeroed)
  // then (complex64 vectors) the tagged copy of y, 16 bytes per value
  const bool tagged = sizeof(TV) == 4;
  const size_t yt_off = ((sizeof(int) * (nblk + 16 + n)) + 255) / 256 * 256;
  int* err = ctx->ext_flags;
  if (tagged && err) {
    set_error("dense solve: complex64 vectors need the context's flag buffer");
    return M25_ERR_VALUE;
  }
  if (!err) {
    void* before = ctx->flags.p;
    int rc = ctx->flags.ensure(yt_off + (tagged ? sizeof(unsigned long long) * 2 * (size_t)n * 8 : 0));
    if (rc) return rc;
    if (ctx->flags_fresh || ctx->flags.p != before) {
      M25_CUDA(cudaMemsetAsync(ctx->flags.p, 0, ctx->flags.bytes, st));
      ctx->flags_fresh = false;
      ctx->epoch = 0;
    }
    err = ctx->flags.as<int>();
  }
  int* flags = err + 16;
  unsigned long long* Yt =
      tagged ? reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(err) + yt_off) : nullptr;
  if (!Yt && ctx->yt_off && sizeof(int) * (nblk + 16 + n) > ctx->yt_off)
    ctx->yt_off = 0;  // this call's permutation reaches into the tagged copy of an earlier one
  if (Yt && ctx->yt_off != yt_off) {
    // the tagged copy moved (another n): what the buffer held there before
    // (permutations, flags) must not pass for a tag of this sweep
    M25_CUDA(cudaMemsetAsync(Yt, 0, sizeof(unsigned long long) * 2 * (size_t)n * 8, st));
    ctx->yt_off = yt_off;
  }
  if (!ctx->ext_flags) {
    // what another order's permutation or tagged copy left where this one's flags lie must not pass for a flag
    if (!tagged && ctx->flags_nblk != nblk) M25_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * nblk, st));
    ctx->flags_nblk = tagged ? -1 : nblk;
  }
  const size_t sm = wave_smem<TF, TV>();
  M25_CUDA(cudaFuncSetAttribute(trsv_wave_kernel<TF, TV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  int occ = 0;
  M25_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, trsv_wave_kernel<TF, TV>, 256, sm));
  if (occ < 1) {
    set_error("dense solve: the triangular-solve kernel does not fit on an SM");
    return M25_ERR_CUDA;
  }
  // M25_WAVE_CTAS: at most this many CTAs (a tuning knob; 0 or unset = one per block up to the device's fill)
  static const int wave_cap_env = getenv("M25_WAVE_CTAS") ? atoi(getenv("M25_WAVE_CTAS")) : 0;
  const int wave_cap = wide ? 0 : ctx->tune_wave_ctas > 0 ? ctx->tune_wave_ctas : wave_cap_env;
  const int G = std::min(std::min(nblk, ctx->num_sms * occ), wave_cap > 0 ? wave_cap : nblk);
  StageTimer tm(ctx, ST_TRSV);
  if (!perm) {
    if (ctx->ext_flags) {  // no room for a permutation in a caller-provided flag buffer
      set_error("dense solve: a precomputed permutation is required here");
      return M25_ERR_VALUE;
    }
    int32_t* pbuf = flags + nblk;
    int rc = lu_make_perm(ctx, n, ipiv, pbuf);
    if (rc) return rc;
    perm = pbuf;
  }
  {
    const int64_t tot = (int64_t)n * nrhs;
    gather_rows_kernel<TV><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(n, nrhs, perm, B, X);
  }
  for (int upper = 0; upper < 2; ++upper) {
    if (++ctx->epoch <= 0) {  // wrapped: start the flags (and tags) afresh
      M25_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * nblk, st));
      if (Yt) M25_CUDA(cudaMemsetAsync(Yt, 0, sizeof(unsigned long long) * 2 * (size_t)n * 8, st));
      ctx->epoch = 1;
    }
    WaveArgs<TF, TV> wa{A, lda, n, nrhs, upper, X, flags, ctx->epoch, err,
                        ctx->wave_spins > 0 ? ctx->wave_spins : kFlagSpinLimit, Yt};
    void* args[] = {&wa};
    M25_CUDA(cudaLaunchCooperativeKernel((void*)trsv_wave_kernel<TF, TV>, dim3(G), dim3(256), args, sm, st));
  }
  M25_CHECK_LAUNCH();
  return M25_OK;
}

// clear the wait flag of the triangular solves before a solve: a solve whose
// wait ran out left it set, and every later sweep would give up at once
int lu_wave_reset(m25_ctx* ctx) {
  if (ctx->ext_flags) return M25_OK;  // a caller-provided flag buffer is cleared by its owner
  if (ctx->flags.p) M25_CUDA(cudaMemsetAsync(ctx->flags.p, 0, sizeof(int), ctx->stream));
  return M25_OK;
}

// the wait flag of the last sweeps (0: every wait ended in time)
int lu_wave_error(m25_ctx* ctx, int n, int* flag) {
  *flag = 0;
  (void)n;
  const int* src = ctx->ext_flags ? ctx->ext_flags : ctx->flags.as<int>();
  if (!src) return M25_OK;
  M25_CUDA(cudaMemcpyAsync(flag, src, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  M25_CUDA(cudaStreamSynchronize(ctx->stream));
  return M25_OK;
}

template int lu_solve_wave<double, double>(m25_ctx*, const zd*, int64_t, int, const int32_t*, const zd*, int, zd*,
                                           const int32_t*, bool);
template int lu_solve_wave<float, float>(m25_ctx*, const zf*, int64_t, int, const int32_t*, const zf*, int, zf*,
                                         const int32_t*, bool);

template int lu_factor<double>(m25_ctx*, zd*, int64_t, int, int32_t*, int, bool, int*);
template int lu_factor<float>(m25_ctx*, zf*, int64_t, int, int32_t*, int, bool, int*);

// ------------------------------------------------ GMRES iterative refinement
// Right-hand sides are handled in lockstep (one column per rhs).

// ---- fp64-accurate products on the fp32 pipes. GB300's fp64 rate makes an
// fp64 matrix-vector product arithmetic-bound (~0.8 ms at N = 5943); here
// Z is held as two complex64 planes, Z = Zh + Zl (Zl = fp32(Z - Zh)), the
// vectors likewise, and the dot products use the error-free transforms of
// Ogita, Rump & Oishi ("Accurate sum and dot product", 2005): the FMA
// two-product and Knuth's two-sum, with the cross terms Zh Xl + Zl Xh and the
// rounding errors summed in fp32. The result is as accurate as a dot product
// in about 2^-48 relative precision, read from the same HBM bytes as the
// complex128 matrix.
__device__ __forceinline__ void dot2_acc(float& s, float& c, float ah, float al, float bh, float bl) {
  const float p = ah * bh;
  const float ep = fmaf(ah, bh, -p);
  const float t = s + p;
  const float z = t - s;
  const float es = (s - (t - z)) + (p - z);
  s = t;
  c += (ep + es) + fmaf(ah, bl, al * bh);
}

// Y = Z X, a row per warp; Zl may be absent (LO false: Z is exact in complex64). Each lane has the loads of four
// column steps (eight of eight bytes) in flight before it uses the first. Bound by the fp32 operations (some 120
// per element and two columns), then by the matrix's bytes: N = 5943, two columns 168 us (3.4 TB/s; 183 us with one
// step in flight; packed fp32 operations, 194 - 282 us, lose more in moves than they save).
template <int P, bool LO>
__global__ void __launch_bounds__(256) matvec_df_kernel(int n, const zf* __restrict__ Zh, const zf* __restrict__ Zl,
                                                        int64_t ldz, const zf* __restrict__ Xh,
                                                        const zf* __restrict__ Xl, zd* __restrict__ Y) {
  constexpr int D = 4;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= n) return;
  float s[P][2], cc[P][2];
#pragma unroll
  for (int c = 0; c < P; ++c) s[c][0] = s[c][1] = cc[c][0] = cc[c][1] = 0.f;
  const zf *zhp = Zh + (int64_t)row * ldz, *zlp = LO ? Zl + (int64_t)row * ldz : nullptr;
  auto step = [&](int t, zf zh, zf zl) {
#pragma unroll
    for (int c = 0; c < P; ++c) {
      const zf xh = Xh[(int64_t)t * P + c], xl = Xl[(int64_t)t * P + c];
      dot2_acc(s[c][0], cc[c][0], zh.re, zl.re, xh.re, xl.re);
      dot2_acc(s[c][0], cc[c][0], zh.im, zl.im, -xh.im, -xl.im);
      dot2_acc(s[c][1], cc[c][1], zh.re, zl.re, xh.im, xl.im);
      dot2_acc(s[c][1], cc[c][1], zh.im, zl.im, xh.re, xl.re);
    }
  };
  int t = lane;
  for (; t + 32 * (D - 1) < n; t += 32 * D) {
    zf zh[D], zl[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      zh[d] = zhp[t + 32 * d];
      if (LO) zl[d] = zlp[t + 32 * d];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) step(t + 32 * d, zh[d], zl[d]);
  }
  for (; t < n; t += 32) step(t, zhp[t], LO ? zlp[t] : zf());
#pragma unroll
  for (int c = 0; c < P; ++c) {
    double v[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float a = s[c][q], e = cc[c][q];
      for (int o = 16; o; o >>= 1) {
        const float b = __shfl_down_sync(0xffffffffu, a, o), f = __shfl_down_sync(0xffffffffu, e, o);
        const float u = a + b, z = u - a;
        e += f + ((a - (u - z)) + (b - z));
        a = u;
      }
      v[q] = (double)a + (double)e;
    }
    if (lane == 0) Y[(int64_t)row * P + c] = zd(v[0], v[1]);
  }
}

// hi / lo complex64 planes of complex128 values: hi = fp32(x), lo = fp32(x - hi)
__device__ __forceinline__ void split_z64(zd x, zf& h, zf& l) {
  const float hr = (float)x.re, hi = (float)x.im;
  h = zf(hr, hi);
  l = zf((float)(x.re - (double)hr), (float)(x.im - (double)hi));
}
__global__ void split_z64_kernel(int64_t n, const zd* __restrict__ X, zf* __restrict__ Xh, zf* __restrict__ Xl) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) split_z64(X[e], Xh[e], Xl[e]);
}

// the same for an n x m block of a matrix (leading dimensions lda / ldb),
// also writing the hi plane to a second destination (the LU's input, ldlu)
// Row equilibration of the mixed solve: rs[r] = 2^-e with max_c |Z[r][c]|
// (|re| + |im|) in [2^(e-1), 2^e): scaling by powers of two is exact, and
// rows of very different size (the via unknowns' rows next to the RWG rows)
// no longer hide the RWG rows' residuals in the normwise backward error.
__global__ void row_scale_kernel(int n, const zd* __restrict__ a, int64_t lda, double* __restrict__ rs) {
  const int r = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (r >= n) return;
  double mx = 0.0;
  for (int c = lane; c < n; c += 32) {
    const zd x = a[(int64_t)r * lda + c];
    mx = fmax(mx, fabs(x.re) + fabs(x.im));
  }
  for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) {
    int e = 0;
    frexp(mx, &e);
    rs[r] = mx > 0.0 && isfinite(mx) ? ldexp(1.0, -e) : 1.0;
  }
}

__global__ void scale_rows_kernel(int64_t n, int P, const double* __restrict__ rs, zd* __restrict__ B) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * P) return;
  const double s = rs[e / P];
  B[e] = zd(B[e].re * s, B[e].im * s);
}

__global__ void split_matrix_kernel(const zd* __restrict__ a, int64_t lda, zf* __restrict__ lu, int64_t ldlu,
                                    zf* __restrict__ h, zf* __restrict__ l, int64_t ldb, int n, int m,
                                    const double* __restrict__ rs) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * m) return;
  const int64_t r = e / m, c = e % m;
  zd x = a[r * lda + c];
  if (rs) x = zd(x.re * rs[r], x.im * rs[r]);
  const float hr = (float)x.re, hi = (float)x.im;
  const zf hv(hr, hi);
  lu[r * ldlu + c] = hv;
  h[r * ldb + c] = hv;
  l[r * ldb + c] = zf((float)(x.re - (double)hr), (float)(x.im - (double)hi));
}

// Y = (Zh + Zl) X in fp64-level accuracy; Xh + Xl: the split X (n P complex64 each)
void matvec_df(int n, int P, const zf* Zh, const zf* Zl, int64_t ldz, const zf* Xh, const zf* Xl, zd* Y,
               cudaStream_t st) {
  const unsigned g = (unsigned)(((size_t)n * 32 + 255) / 256);
#define M25_MVDF(PP)                                                                \
  case PP:                                                                          \
    if (Zl)                                                                         \
      matvec_df_kernel<PP, true><<<g, 256, 0, st>>>(n, Zh, Zl, ldz, Xh, Xl, Y);     \
    else                                                                            \
      matvec_df_kernel<PP, false><<<g, 256, 0, st>>>(n, Zh, Zl, ldz, Xh, Xl, Y);    \
    break
  switch (P) {
    M25_MVDF(1);
    M25_MVDF(2);
    M25_MVDF(3);
    M25_MVDF(4);
    M25_MVDF(5);
    M25_MVDF(6);
    M25_MVDF(7);
    M25_MVDF(8);
    default: break;  // 1 <= P <= 8 is checked by the callers
  }
#undef M25_MVDF
}

// The vector kernels of a GMRES step. Sums over the rows are formed in a
// fixed order: by kDotSplit CTAs (the dot products) or by the CTAs of 256 elements (the
// norms), whose partial sums the next kernel adds up. (One CTA per dot product
// or norm took 32 and 19 us at N = 5943 with two columns, its fp64
// operations and latencies on one SM; the host then scaled the vector between two synchronisations.)
constexpr int kDotSplit = 8;
constexpr int kMaxGmres = 30;  // restart length
// A solve that takes more steps than this is the long pole of a sweep (the LPF's and the via transition's lowest
// frequencies: 12 and 46 steps against 2 to 5): the CTA cap, which leaves room to points beside it, ends there.
// Eight points in flight, via transition: 63 ms a sweep of eight, 72 ms with the cap throughout.
constexpr int kCappedSteps = 4;

// sum of v over the CTA (256 threads), on thread 0
__device__ __forceinline__ double cta_sum(double v, double* red) {
  for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < 8; ++w) s += red[w];
  return s;
}

// hp[k][i][c] = sum over the rows of part k of conj(V_i[t][c]) W[t][c], i < nvec; grid (nvec, kDotSplit)
__global__ void __launch_bounds__(256) dots_kernel(int n, int P, const zd* __restrict__ V, int64_t vstride,
                                                   const zd* __restrict__ W, zd* __restrict__ hp, int hcap) {
  const int i = blockIdx.x, k = blockIdx.y;
  const int t0 = (int)((int64_t)n * k / kDotSplit), t1 = (int)((int64_t)n * (k + 1) / kDotSplit);
  const zd* Vi = V + (int64_t)i * vstride;
  __shared__ double red[8];
  for (int c = 0; c < P; ++c) {
    zd acc;
    for (int t = t0 + threadIdx.x; t < t1; t += 256) {
      const zd v = Vi[(int64_t)t * P + c], w = W[(int64_t)t * P + c];
      acc.re = fma(v.re, w.re, fma(v.im, w.im, acc.re));
      acc.im = fma(v.re, w.im, fma(-v.im, w.re, acc.im));
    }
    const double re = cta_sum(acc.re, red), im = cta_sum(acc.im, red);
    if (threadIdx.x == 0) hp[(size_t)k * hcap + i * P + c] = zd(re, im);
  }
}

// part[b][c] = the squared 2-norm of CTA b's elements of column c (one element per thread)
__device__ __forceinline__ void norm_parts(int64_t e, int64_t np, int P, zd v, double* red, double* part) {
  const double q = e < np ? norm2(v) : 0.0;
  const int col = (int)(e % P);
  for (int c = 0; c < P; ++c) {
    const double s = cta_sum(c == col ? q : 0.0, red);
    if (threadIdx.x == 0) part[(size_t)blockIdx.x * P + c] = s;
  }
}

// W[t][c] -= sum_{i < nvec} V_i[t][c] h[i][c], h the sum of the parts hp, which CTA 0 also writes to hout; with
// part: the partial norms of the new W, and *mx = 0 for col_scale_kernel
__global__ void __launch_bounds__(256) orth_update_kernel(int n, int P, int nvec, const zd* __restrict__ V,
                                                          int64_t vstride, const zd* __restrict__ hp, int hcap,
                                                          zd* __restrict__ hout, zd* __restrict__ W,
                                                          double* __restrict__ part,
                                                          unsigned long long* __restrict__ mx) {
  __shared__ zd h[kMaxGmres * 8];
  __shared__ double red[8];
  for (int j = threadIdx.x; j < nvec * P; j += 256) {
    zd a;
    for (int k = 0; k < kDotSplit; ++k) a += hp[(size_t)k * hcap + j];
    h[j] = a;
    if (blockIdx.x == 0) hout[j] = a;
  }
  if (mx && blockIdx.x == 0 && threadIdx.x == 0) *mx = 0;
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x, np = (int64_t)n * P;
  zd v;
  if (e < np) {
    const int c = int(e % P);
    v = W[e];
    for (int i = 0; i < nvec; ++i) v = fnma(v, V[(int64_t)i * vstride + e], h[i * P + c]);
    W[e] = v;
  }
  if (part) norm_parts(e, np, P, v, red, part);
}

// R = B - W (W = Z X), the partial norms of R, X and B, and *mx = 0
__global__ void __launch_bounds__(256) residual_kernel(int n, int P, const zd* __restrict__ B,
                                                       const zd* __restrict__ W, const zd* __restrict__ X,
                                                       zd* __restrict__ R, double* __restrict__ pr,
                                                       double* __restrict__ px, double* __restrict__ pb,
                                                       unsigned long long* __restrict__ mx) {
  __shared__ double red[8];
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x, np = (int64_t)n * P;
  if (blockIdx.x == 0 && threadIdx.x == 0) *mx = 0;
  zd b, r, x;
  if (e < np) {
    b = B[e];
    x = X[e];
    r = b - W[e];
    R[e] = r;
  }
  norm_parts(e, np, P, r, red, pr);
  norm_parts(e, np, P, x, red, px);
  norm_parts(e, np, P, b, red, pb);
}

// out = in / |in| per column (0 for a zero column) from the partial norms; *mx
// = the largest |re| + |im| of out (the preconditioner's scale) and, from
// CTA 0, norms[c] = |in|
__global__ void __launch_bounds__(256) col_scale_kernel(int64_t np, int P, const zd* __restrict__ in, int nparts,
                                                        const double* __restrict__ part, zd* __restrict__ out,
                                                        double* __restrict__ norms,
                                                        unsigned long long* __restrict__ mx) {
  __shared__ double inv[8];
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < P; c += 8) {
    double s = 0;
    for (int b = lane; b < nparts; b += 32) s += part[(size_t)b * P + c];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const double r = sqrt(s);
      inv[c] = r > 0 ? 1.0 / r : 0.0;
      if (blockIdx.x == 0) norms[c] = r;
    }
  }
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  double m = 0;
  if (e < np) {
    const zd v = in[e] * inv[e % P];
    out[e] = v;
    m = cabs1(v);
  }
  for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) atomicMax(mx, (unsigned long long)__double_as_longlong(m));  // m >= 0: bit order = value order
}

// X[t][c] += sum_i V_i[t][c] y[i][c]
__global__ void combine_kernel(int n, int P, int nvec, const zd* __restrict__ V, int64_t vstride,
                               const zd* __restrict__ y, zd* __restrict__ X) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * P) return;
  int c = int(e % P);
  zd s(0.0);
  for (int i = 0; i < nvec; ++i) s += V[(int64_t)i * vstride + e] * y[i * P + c];
  X[e] += s;
}

// max over rows of sum |Z[t][k]| (infinity norm; it only scales the stopping
// test, so fp32 from the hi plane), one warp per row + atomicMax on the bits
__global__ void rownorm_kernel(int n, const zf* __restrict__ Z, int64_t ldz, unsigned long long* __restrict__ out) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  const zf* row = Z + (int64_t)warp * ldz;
  float s = 0;
  int t = lane;
  for (; t + 7 * 32 < n; t += 8 * 32) {
    zf z[8];
#pragma unroll
    for (int d = 0; d < 8; ++d) z[d] = row[t + 32 * d];
#pragma unroll
    for (int d = 0; d < 8; ++d) s += sqrtf(z[d].re * z[d].re + z[d].im * z[d].im);
  }
  for (; t < n; t += 32) s += sqrtf(row[t].re * row[t].re + row[t].im * row[t].im);
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) atomicMax(out, (unsigned long long)__double_as_longlong((double)s));  // s >= 0: bit order = value order
}

// o = a / s and back, s = *sp (a device scalar; 1 when it is not positive)
__global__ void z64_to_z32_scaled(int64_t n, const zd* __restrict__ a, const double* __restrict__ sp,
                                  zf* __restrict__ o) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const double s = *sp > 0 ? 1.0 / *sp : 1.0;
  if (e < n) o[e] = zf(float(a[e].re * s), float(a[e].im * s));
}
// the second with the hi / lo planes of o for the product that follows
__global__ void z32_to_z64_scaled(int64_t n, const zf* __restrict__ a, const double* __restrict__ sp,
                                  zd* __restrict__ o, zf* __restrict__ oh, zf* __restrict__ ol) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const double s = *sp > 0 ? *sp : 1.0;
  const zd x(double(a[e].re) * s, double(a[e].im) * s);
  o[e] = x;
  split_z64(x, oh[e], ol[e]);
}
// *out = max |re| + |im| (*out starts at 0)
__global__ void __launch_bounds__(256) maxabs_kernel(int64_t n, const zd* __restrict__ a,
                                                     unsigned long long* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  double m = e < n ? cabs1(a[e]) : 0.0;
  for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// Restarted flexible GMRES in fp64 on Z x = B, right-preconditioned by the
// complex64 LU applied in fp32 arithmetic (GMRES-based iterative refinement,
// Carson & Higham 2017, in its flexible form so that the rounding of the
// fp32 triangular solves does not break the Arnoldi relation: fp64 on this
// GPU is too slow for the serial substitution chains). Orthogonalisation and
// the iterate stay in fp64; the matrix-vector products use Z = Zh + Zl, two
// complex64 planes, with fp64-level accuracy on the fp32 pipes (matvec_df;
// Zl absent when Z is itself complex64). Stops when the normwise backward
// error |r| / (|Z| |x| + |b|) of every column <= tol; max_iter bounds the
// total number of GMRES steps.
int refine(m25_ctx* ctx, int n, int P, const zf* Zh, const zf* Zl, int64_t ldz, const zf* LU, int64_t ldlu,
           const int32_t* ipiv, const zd* B, zd* X, double tol, int max_iter, int* steps) {
  cudaStream_t st = ctx->stream;
  const int m = std::min(kMaxGmres, std::max(1, max_iter));
  const size_t np = (size_t)n * P;
  const unsigned g1 = (unsigned)((np + 255) / 256);
  const int hcap = m * P;
  int rc = ctx->Rw.ensure(sizeof(zd) * np * (2 * m + 3) + sizeof(zf) * np * 4 + sizeof(double) * (64 + 3 * (size_t)g1 * P) +
                          sizeof(zd) * (size_t)hcap * (kDotSplit + 3) + sizeof(int32_t) * n);
  if (rc) return rc;
  zd* V = ctx->Rw.as<zd>();           // (m+1) Arnoldi vectors
  zd* Zp = V + np * (m + 1);          // (m) preconditioned directions
  zd* W = Zp + np * m;                // work vector
  zd* R = W + np;                     // residual
  zf* r32 = reinterpret_cast<zf*>(R + np);
  zf* d32 = r32 + np;
  zf* xh = d32 + np;                                        // hi / lo planes of a vector
  zf* xl = xh + np;
  zd* hp = reinterpret_cast<zd*>(xl + np);                  // partial dot products
  zd* ydev = hp + (size_t)hcap * kDotSplit;
  zd* hout = ydev + hcap;                                   // the step's results for the host: two passes of dot products, norms
  double* wnorm = reinterpret_cast<double*>(hout + 2 * (size_t)hcap);
  double* pscale = wnorm + 48;
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(pscale);
  double* parts = wnorm + 64;                               // partial norms: 3 x (g1, P)
  const size_t nparts = (size_t)g1 * P;
  int32_t* perm = reinterpret_cast<int32_t*>(parts + 3 * nparts);  // row permutation of the LU
  const unsigned gw = (unsigned)(((size_t)n * 32 + 255) / 256);
  StageTimer tm(ctx, ST_REFINE);
  int total = 0;  // GMRES steps
  // out = (LU32)^-1 in, in fp32 with the input scaled to O(1) by its
  // largest entry *mx (kept on the device: no host round trip), and out's planes
  auto precond = [&](const zd* in, zd* out) -> int {
    z64_to_z32_scaled<<<g1, 256, 0, st>>>((int64_t)np, in, pscale, r32);
    int r = lu_solve_wave<float, float>(ctx, LU, ldlu, n, ipiv, r32, P, d32, perm, total >= kCappedSteps);
    if (r) return r;
    z32_to_z64_scaled<<<g1, 256, 0, st>>>((int64_t)np, d32, pscale, out, xh, xl);
    return M25_OK;
  };
  auto set_col_scalars = [&](const std::vector<zd>& v) -> int {
    M25_CUDA(cudaMemcpyAsync(ydev, v.data(), sizeof(zd) * v.size(), cudaMemcpyHostToDevice, st));
    return M25_OK;
  };
  if ((rc = lu_make_perm(ctx, n, ipiv, perm))) return rc;
  unsigned long long* zb = mx + 1;
  M25_CUDA(cudaMemsetAsync(mx, 0, 2 * sizeof(unsigned long long), st));
  rownorm_kernel<<<gw, 256, 0, st>>>(n, Zh, ldz, zb);
  // start from the fp32 solution x0 = M^-1 B
  maxabs_kernel<<<g1, 256, 0, st>>>((int64_t)np, B, mx);
  if ((rc = precond(B, X))) return rc;
  double prev_worst = INFINITY, znorm = 0;
  std::vector<double> rn(P), xn(P), bn(P), hparts(64 + 3 * nparts), step(4 * (size_t)hcap + P);
  std::vector<zd> hh((size_t)(m + 2) * P), H((size_t)(m + 1) * m * P), g((size_t)(m + 1) * P), cs(m * P), sn(m * P);
  for (int outer = 0; outer < 50; ++outer) {
    // R = B - Z X
    if (outer) split_z64_kernel<<<g1, 256, 0, st>>>((int64_t)np, X, xh, xl);
    matvec_df(n, P, Zh, Zl, ldz, xh, xl, W, st);
    residual_kernel<<<g1, 256, 0, st>>>(n, P, B, W, X, R, parts, parts + nparts, parts + 2 * nparts, mx);
    M25_CUDA(cudaMemcpyAsync(hparts.data(), wnorm, sizeof(double) * hparts.size(), cudaMemcpyDeviceToHost, st));
    M25_CUDA(cudaStreamSynchronize(st));
    znorm = hparts[49];  // zb
    for (int c = 0; c < P; ++c) {
      double q[3] = {};
      for (int k = 0; k < 3; ++k)
        for (unsigned b = 0; b < g1; ++b) q[k] += hparts[64 + k * nparts + (size_t)b * P + c];
      rn[c] = sqrt(q[0]);
      xn[c] = sqrt(q[1]);
      bn[c] = sqrt(q[2]);
    }
    double worst = 0;
    std::vector<double> target(P);
    bool finite = std::isfinite(znorm);
    for (int c = 0; c < P; ++c) {
      double den = znorm * xn[c] + bn[c];
      target[c] = tol * den;
      finite = finite && std::isfinite(rn[c]) && std::isfinite(xn[c]);
      worst = std::max(worst, den > 0 ? rn[c] / den : 0.0);
    }
    if (!finite) {  // an overflow in the complex64 factors or solves: never "converged"
      set_error("mixed solve: non-finite residual or solution (complex64 LU overflow?)");
      return M25_ERR_NUMERIC;
    }
    if (worst <= tol) break;
    const bool stalled = worst > 0.5 * prev_worst;
    if (total >= max_iter || stalled) {
      if (worst <= 1e3 * tol && outer > 0) break;  // at the fp64 floor
      char msg[160];
      snprintf(msg, sizeof msg,
               "mixed solve: GMRES refinement stopped at backward error %.3e (tolerance %.1e) after %d steps",
               worst, tol, total);
      set_error(msg);
      return M25_ERR_NUMERIC;
    }
    prev_worst = worst;
    // V0 = R / |R|
    col_scale_kernel<<<g1, 256, 0, st>>>((int64_t)np, P, R, (int)g1, parts, V, wnorm, mx);
    std::fill(g.begin(), g.end(), zd(0.0));
    for (int c = 0; c < P; ++c) g[c] = zd(rn[c]);
    int k = 0;
    for (; k < m && total < max_iter; ++k, ++total) {
      zd* zk = Zp + np * k;
      if ((rc = precond(V + np * k, zk))) return rc;
      matvec_df(n, P, Zh, Zl, ldz, xh, xl, W, st);
      // classical Gram-Schmidt, twice; then V_{k+1} = W / |W|
      for (int pass = 0; pass < 2; ++pass) {
        dots_kernel<<<dim3(k + 1, kDotSplit), 256, 0, st>>>(n, P, V, (int64_t)np, W, hp, hcap);
        orth_update_kernel<<<g1, 256, 0, st>>>(n, P, k + 1, V, (int64_t)np, hp, hcap, hout + (size_t)pass * hcap, W,
                                               pass ? parts : nullptr, pass ? mx : nullptr);
      }
      col_scale_kernel<<<g1, 256, 0, st>>>((int64_t)np, P, W, (int)g1, parts, V + np * (k + 1), wnorm, mx);
      M25_CUDA(cudaMemcpyAsync(step.data(), hout, sizeof(double) * step.size(), cudaMemcpyDeviceToHost, st));
      M25_CUDA(cudaStreamSynchronize(st));
      for (int i = 0; i < (k + 1) * P; ++i)
        hh[i] = zd(step[2 * i], step[2 * i + 1]) + zd(step[2 * (hcap + i)], step[2 * (hcap + i) + 1]);
      const double* wn = step.data() + 4 * (size_t)hcap;
      bool done = true;
      for (int c = 0; c < P; ++c) {
        // column k of the Hessenberg matrix, rotated by the previous Givens rotations
        std::vector<zd> col(k + 2);
        for (int i = 0; i <= k; ++i) col[i] = hh[(size_t)i * P + c];
        col[k + 1] = zd(wn[c]);
        for (int i = 0; i < k; ++i) {
          zd x0 = col[i], x1 = col[i + 1];
          zd cI = cs[(size_t)i * P + c], sI = sn[(size_t)i * P + c];
          col[i] = conj(cI) * x0 + conj(sI) * x1;
          col[i + 1] = -sI * x0 + cI * x1;
        }
        double r = sqrt(norm2(col[k]) + norm2(col[k + 1]));
        zd cN = r > 0 ? col[k] / zd(r) : zd(1.0), sN = r > 0 ? col[k + 1] / zd(r) : zd(0.0);
        cs[(size_t)k * P + c] = cN;
        sn[(size_t)k * P + c] = sN;
        col[k] = zd(r);
        col[k + 1] = zd(0.0);
        for (int i = 0; i <= k; ++i) H[((size_t)i * m + k) * P + c] = col[i];
        zd gk = g[(size_t)k * P + c];
        g[(size_t)k * P + c] = conj(cN) * gk;
        g[(size_t)(k + 1) * P + c] = -sN * gk;
        // right preconditioning: |g_{k+1}| estimates the true residual
        if (cabs(g[(size_t)(k + 1) * P + c]) > 0.25 * target[c]) done = false;
      }
      if (done) {
        ++k;
        ++total;
        break;
      }
    }
    // y = H^-1 g (upper triangular), X += Zp y
    std::vector<zd> y((size_t)k * P, zd(0.0));
    for (int c = 0; c < P; ++c)
      for (int i = k - 1; i >= 0; --i) {
        zd sacc = g[(size_t)i * P + c];
        for (int j = i + 1; j < k; ++j) sacc -= H[((size_t)i * m + j) * P + c] * y[(size_t)j * P + c];
        zd d = H[((size_t)i * m + i) * P + c];
        y[(size_t)i * P + c] = (d.re != 0 || d.im != 0) ? sacc / d : zd(0.0);
      }
    if (k > 0) {
      if ((rc = set_col_scalars(y))) return rc;
      combine_kernel<<<g1, 256, 0, st>>>(n, P, k, Zp, (int64_t)np, ydev, X);
    }
  }
  *steps = total;
  M25_CHECK_LAUNCH();
  return M25_OK;
}



// rs (n doubles, device) or null: the rows are equilibrated by powers of two
// (row_scale_kernel), and the right-hand sides B (n x P) with them
void split_to_z32(m25_ctx* ctx, const zd* a, int64_t lda, zf* lu, int64_t ldlu, zf* h, zf* l, int64_t ldb, int n,
                  int m, double* rs, zd* B, int P) {
  int64_t tot = (int64_t)n * m;
  if (rs) {
    row_scale_kernel<<<(unsigned)(((int64_t)n * 32 + 255) / 256), 256, 0, ctx->stream>>>(n, a, lda, rs);
    scale_rows_kernel<<<(unsigned)(((int64_t)n * P + 255) / 256), 256, 0, ctx->stream>>>(n, P, rs, B);
  }
  split_matrix_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, ctx->stream>>>(a, lda, lu, ldlu, h, l, ldb, n, m, rs);
}

}  // namespace m25

// ------------------------------------------------- allocation-free solve
// Scratch of m25_dense_solve_noalloc: one file-scope device array that every
// GPU loading this library holds until the process exits. Layout: [0, 64)
// barrier words of the panel factorisation, then its candidate pivot rows for
// up to kNoAllocGmax CTAs of 64 columns, then the ready flags of the
// triangular solves, then the row permutation of the factorisation.
namespace {
constexpr int kNoAllocGmax = 192;
constexpr size_t kNoAllocPanelBytes = 64 + sizeof(m25::zd) * 2 * kNoAllocGmax * 64 + sizeof(double) * 2 * kNoAllocGmax +
                                      sizeof(int) * 2 * kNoAllocGmax + sizeof(m25::zd) * 2 * 64;
constexpr size_t kNoAllocFlagsOffset = (kNoAllocPanelBytes + 255) / 256 * 256;
constexpr size_t kNoAllocPermOffset =
    (kNoAllocFlagsOffset + sizeof(int) * (16 + M25_NOALLOC_MAX_N / m25::wave_b<double>() + 1) + 255) / 256 * 256;
static_assert(kNoAllocPermOffset + sizeof(int) * M25_NOALLOC_MAX_N <= M25_NOALLOC_SCRATCH_BYTES,
              "scratch too small for the declared maximum size");
std::mutex g_noalloc_mu;
constexpr int kMaxDevices = 64;
void* g_noalloc_addr[kMaxDevices] = {};
}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[M25_NOALLOC_SCRATCH_BYTES];

extern "C" int m25_dense_solve_noalloc(int32_t n, int32_t nrhs, void* Z, const void* B, void* X, int32_t* ipiv,
                                       void* stream, int32_t* info) {
  using namespace m25;
  if (!Z || !B || !X || !ipiv || n < 1 || nrhs < 1 || nrhs > 8) {
    set_error("m25_dense_solve_noalloc: null pointer, n < 1 or nrhs outside 1..8");
    return M25_ERR_VALUE;
  }
  if (n > M25_NOALLOC_MAX_N) {
    set_error("m25_dense_solve_noalloc: n = " + std::to_string(n) + " exceeds the maximum " +
              std::to_string(M25_NOALLOC_MAX_N) + " of the static scratch; use m25_dense_solve");
    return M25_ERR_VALUE;
  }
  int dev = 0;
  M25_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("m25_dense_solve_noalloc: device index out of range");
    return M25_ERR_VALUE;
  }
  void* addr = nullptr;
  {
    // once per device, with that device current: the device address of the
    // array (its host-side name is only a stand-in, not a device pointer)
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        set_error(std::string("m25_dense_solve_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        return M25_ERR_CUDA;
      }
      g_noalloc_addr[dev] = p;
    }
    addr = g_noalloc_addr[dev];
  }
  m25_ctx c;  // borrowed stream, no workspace of its own
  c.device = dev;
  c.stream = static_cast<cudaStream_t>(stream);
  M25_CUDA(cudaDeviceGetAttribute(&c.num_sms, cudaDevAttrMultiProcessorCount, dev));
  if (c.num_sms > kNoAllocGmax) {
    set_error("m25_dense_solve_noalloc: more SMs than the static panel scratch covers");
    return M25_ERR_VALUE;
  }
  char* base = static_cast<char*>(addr);
  c.ext_scratch = base;
  c.ext_gmax = kNoAllocGmax;
  c.ext_flags = reinterpret_cast<int*>(base + kNoAllocFlagsOffset);
  // the array keeps the previous call's contents: clear the barrier words
  // (lu_factor clears its header) and the ready flags
  M25_CUDA(cudaMemsetAsync(c.ext_flags, 0, sizeof(int) * (16 + n / m25::wave_b<double>() + 1), c.stream));
  int zinfo = 0;
  int rc = lu_factor<double>(&c, static_cast<zd*>(Z), n, n, ipiv, 64, false, &zinfo);
  if (rc) return rc;
  if (info) {
    info[0] = 0;
    info[1] = zinfo;
  }
  if (zinfo) {
    set_error("m25_dense_solve_noalloc: exactly singular matrix (zero pivot)");
    return M25_ERR_NUMERIC;
  }
  int32_t* perm = reinterpret_cast<int32_t*>(base + kNoAllocPermOffset);
  if ((rc = lu_make_perm(&c, n, ipiv, perm))) return rc;
  rc = lu_solve_wave<double, double>(&c, static_cast<const zd*>(Z), n, n, ipiv, static_cast<const zd*>(B), nrhs,
                                     static_cast<zd*>(X), perm, false);
  if (rc) return rc;
  int werr = 0;
  if ((rc = lu_wave_error(&c, n, &werr))) return rc;
  if (werr) {
    set_error("m25_dense_solve_noalloc: a wait of the triangular solve ran out");
    return M25_ERR_CUDA;
  }
  return M25_OK;
}
