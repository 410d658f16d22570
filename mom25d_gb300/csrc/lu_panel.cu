// The panel of the dense LU (lu.cu): one block of columns is factored strip by
// strip (32 columns of complex64, 16 of complex128), each strip by
//   strip_panel_kernel   one cluster of up to 16 CTAs, the strip's rows in registers
//   strip_update_kernel  U12 of the block's columns right of the strip and their
//                        rank-W update, on the whole GPU
// The panel is a chain of column steps (pivot search, exchange, rank-1
// update), so what bounds it is the latency of a step and, in complex128, the
// rate of fp64 multiply-adds of the SMs that hold the rows (two per clock and
// SM). Hence:
//  - one row per thread (complex128 with few rows: on two or four), its W columns in registers: a step reads only the
//    pivot row from shared memory, and has one CTA barrier and one wait for the
//    cluster's exchange;
//  - rows are not moved while the strip is factored: a thread follows the
//    position of its row through the interchanges and writes it there at the
//    end, so the row at position k0 + j need not be sent around;
//  - narrow strips: the rank-1 updates of a step cost W / 2 columns on
//    average, and the products between strips go to the whole GPU.
//  - complex128: two warps without rows do the division of the reciprocal
//    pivot and send the candidate's row, while the warps with rows run the
//    multiply-adds of the step before (kAhead below).
// Measured on GB300 (one factorisation alone, sum over its panels):
//   complex128, N = 546 / 1085 / 2434 / 5943: 1.4 / 3.0 / 8.0 / 27.8 ms (1.75 / 3.5 / 8.6 / 28.4 ms with one lane per
//   row throughout; 1.9 / 3.9 / 9.4 / 30.6 ms with every step finished before the next one's search, too;
//   7.95 / 20.0 / 53.0 / 96.6 ms for 64-column panels in shared memory, with the row k0 + j sent around and both
//   divisions on the chain)
//   complex64, N = 1085 / 5943: 1.6 / 10.1 ms (2.5 / 21.1 ms, and 0.2 / 2.1 ms for the products between
//   the two panels of a block)
// A column step of complex64 takes about 1 us, of which 0.45 us are the exchange's
// flight; one of complex128 with one lane per row 2.5 us: search 0.35, the candidate's staging 0.4, the
// multiply-adds 1.0 (half with two lanes per row), the wait 0.2, multiplier and next column 0.5.
#include <algorithm>
#include <string>

#include "m25_internal.h"
#include "m25_lu.h"

namespace m25 {

namespace {

constexpr long long kStripSpinLimit = 1LL << 25;
constexpr int kStripThreads = 512;  // rows of a CTA at the most
constexpr int kStripMaxCl = 16;
constexpr int kGrp = 8;             // columns factored between two shifts of the registers

// strip width
template <class T>
constexpr int strip_w() { return sizeof(T) == 4 ? 32 : 16; }

// a CTA's candidate for the pivot of a column
template <class T>
struct alignas(16) StripCand;
template <>
struct alignas(16) StripCand<float> {
  unsigned key;  // bits of |re| + |im| plus one; 0: no row
  int pos;
  float rre, rim;  // reciprocal pivot
};
template <>
struct alignas(16) StripCand<double> {
  unsigned long long key;
  long long pos;
  double rre, rim;
};

template <class T>
struct StripArgs {
  cx<T>* A;
  int64_t lda;
  int n, k0, w;        // rows k0 .. n - 1, columns k0 .. k0 + w - 1
  int blk0, blk1;      // the block's columns: the strip's interchanges are applied to all of them
  int rows_per_cta;
  int32_t* ipiv;
  cx<T>* Ub;           // (w, blk1 - k0 - w): the pivot rows' columns right of the strip (input of strip_update_kernel)
  int* info;
  int* err;
};

__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
// the address of a shared variable of this CTA in the shared memory of cluster CTA rank
__device__ __forceinline__ uint32_t cl_map(const void* p, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// 16-byte remote store that completes its bytes on the destination CTA's mbarrier
__device__ __forceinline__ void cl_put(uint32_t a, uint4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(a),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(count));
}
__device__ __forceinline__ void bar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}
// bounded wait (iterations and wall clock) for the phase of the given parity
// of a barrier completed by remote transactions; a wait that runs out raises
// *fail, and every later wait of the CTA then returns at once
__device__ __forceinline__ void bar_wait(uint64_t* bar, uint32_t parity, volatile int* fail) {
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(bar);
  unsigned long long t0 = 0;
  for (long long it = 0; it < kStripSpinLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return;
    if ((it & 63) != 63) continue;  // the clock is slow to read: seldom
    if (*fail) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    if (t0 == 0) t0 = t;
    if (t - t0 > 500ull * 1000 * 1000) break;
  }
  *fail = 1;
}

// larger value first, then the smaller position; over the lanes of a warp
__device__ __forceinline__ unsigned warp_best(unsigned key, unsigned& pos) {
  const unsigned k = __reduce_max_sync(~0u, key);
  pos = __reduce_min_sync(~0u, key == k ? pos : ~0u);
  return k;
}
__device__ __forceinline__ unsigned long long warp_best(unsigned long long key, unsigned& pos) {
  const unsigned hi = __reduce_max_sync(~0u, (unsigned)(key >> 32));
  const bool top = (unsigned)(key >> 32) == hi;
  const unsigned lo = __reduce_max_sync(~0u, top ? (unsigned)key : 0u);
  pos = __reduce_min_sync(~0u, top && (unsigned)key == lo ? pos : ~0u);
  return ((unsigned long long)hi << 32) | lo;
}
// bits of v + 1 (ordered as v for v >= 0), 0 for a NaN, which is never chosen
__device__ __forceinline__ unsigned val_key(float v) { return v >= 0.f ? __float_as_uint(v) + 1u : 0u; }
__device__ __forceinline__ unsigned long long val_key(double v) {
  // a sum of magnitudes: not negative; the comparison as integers (a NaN's bits exceed infinity's), off the fp64 pipe
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b <= 0x7ff0000000000000ull ? b + 1ull : 0ull;
}
// whether a sum of two squares has neither overflowed nor lost bits below the normal range (2^-960 .. 2^1024,
// 2^-96 .. 2^128; by the bits, off the fp64 pipe)
__device__ __forceinline__ bool square_in_range(double m2) {
  return (unsigned)(__double2hiint(m2) - ((1023 - 960) << 20)) < (unsigned)((2047 - (1023 - 960)) << 20);
}
__device__ __forceinline__ bool square_in_range(float m2) {
  return (unsigned)(__float_as_int(m2) - ((127 - 96) << 23)) < (unsigned)((255 - (127 - 96)) << 23);
}
// a power of two that brings the squares of such a value into it
__device__ __forceinline__ double pivot_scale(cx<double> v) { return cabs1(v) >= 1.0 ? 0x1p-600 : 0x1p600; }
__device__ __forceinline__ float pivot_scale(cx<float> v) { return cabs1(v) >= 1.f ? 0x1p-70f : 0x1p70f; }
template <class T>
using KeyOf = decltype(val_key(T(0)));

// A thread's row of the strip, from column jb on (a multiple of kGrp) at index
// 0. complex64 columns go in pairs, real and imaginary parts apart, for the
// packed fp32 multiply-add (two per lane and instruction). (A row that moves one
// column to the front with every update, so that the loop over the columns
// needs no unrolling, is half the code and 5 to 10 % slower: it spills.)
// complex128 rows may lie on TPR = 2 or 4 neighbouring lanes, lane h of them
// with the columns h, h + TPR, ...; get(i) and the update of one column are for the lane that has it.
template <class T, int TPR>
struct StripRow;
template <int TPR>
struct StripRow<double, TPR> {
  static constexpr int W = strip_w<double>(), N = W / TPR, G = kGrp / TPR;
  cx<double> x[N];
  __device__ __forceinline__ cx<double> get(int i) const { return x[i / TPR]; }
  __device__ __forceinline__ void set(int i, cx<double> v) { x[i / TPR] = v; }
  __device__ __forceinline__ void load(const cx<double>* row, int h) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = row[TPR * i + h];
  }
  // the columns from i0 on to row (from column jb)
  __device__ __forceinline__ void store(int i0, int jb, cx<double>* row, int h) const {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (TPR * i + h >= i0 && jb + TPR * i < W) row[TPR * i + h] = x[i];
  }
  static __device__ __forceinline__ uint4 pack(cx<double> v) {
    return make_uint4((unsigned)__double2loint(v.re), (unsigned)__double2hiint(v.re), (unsigned)__double2loint(v.im),
                      (unsigned)__double2hiint(v.im));
  }
  // the columns from i0 on as they are sent (16 bytes each; u: from column jb)
  __device__ __forceinline__ void stage(int i0, int jb, uint4* u, int h) const {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (TPR * i + TPR > i0 && jb + TPR * i < W) u[TPR * i + h] = pack(x[i]);
  }
  static __device__ __forceinline__ cx<double> sent(const uint4* u, int c) {
    return *reinterpret_cast<const cx<double>*>(u + c);
  }
  // x_i -= l u_i for i >= i0 and jb + i < W (u: the pivot row's chunks from column jb)
  __device__ __forceinline__ void update(int i0, int jb, cx<double> l, const uint4* u, int h) {
#pragma unroll
    for (int i = 0; i < G; ++i)
      if (TPR * i >= i0) {
        x[i] = fnma(x[i], l, sent(u, TPR * i + h));
      } else if (TPR * i + TPR > i0) {
        if (TPR * i + h >= i0) x[i] = fnma(x[i], l, sent(u, TPR * i + h));
      }
    if (jb + kGrp < W)  // no fp64 operation for nothing
#pragma unroll
      for (int i = G; i < N; ++i)
        if (TPR * i >= i0) {
          x[i] = fnma(x[i], l, sent(u, TPR * i + h));
        } else if (TPR * i + h >= i0) {
          x[i] = fnma(x[i], l, sent(u, TPR * i + h));
        }
  }
  __device__ __forceinline__ void shift() {
#pragma unroll
    for (int i = 0; i + G < N; ++i) x[i] = x[i + G];
  }
};
template <>
struct StripRow<float, 1> {
  static constexpr int W = strip_w<float>();
  float4 x[W / 2];  // columns 2 k, 2 k + 1: (re, re, im, im)
  __device__ __forceinline__ cx<float> get(int i) const {
    return (i & 1) ? cx<float>(x[i / 2].y, x[i / 2].w) : cx<float>(x[i / 2].x, x[i / 2].z);
  }
  __device__ __forceinline__ void set(int i, cx<float> v) {
    if (i & 1) {
      x[i / 2].y = v.re;
      x[i / 2].w = v.im;
    } else {
      x[i / 2].x = v.re;
      x[i / 2].z = v.im;
    }
  }
  __device__ __forceinline__ void load(const cx<float>* row, int) {
#pragma unroll
    for (int c = 0; c < W; ++c) set(c, row[c]);
  }
  __device__ __forceinline__ void store(int i0, int jb, cx<float>* row, int) const {
#pragma unroll
    for (int i = 0; i < W; ++i)
      if (i >= i0 && jb + i < W) row[i] = get(i);
  }
  __device__ __forceinline__ void stage(int i0, int jb, uint4* u, int) const {
#pragma unroll
    for (int k = 0; k < W / 2; ++k)
      if (k >= i0 / 2 && jb / 2 + k < W / 2)
        u[k] = make_uint4(__float_as_uint(x[k].x), __float_as_uint(x[k].y), __float_as_uint(x[k].z),
                          __float_as_uint(x[k].w));
  }
  static __device__ __forceinline__ cx<float> sent(const uint4* u, int c) {
    const float* f = reinterpret_cast<const float*>(u + c / 2) + (c & 1);
    return cx<float>(f[0], f[2]);
  }
  static __device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    union {
      float2 f;
      unsigned long long u;
    } x = {a}, y = {b}, z = {c}, r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r.u) : "l"(x.u), "l"(y.u), "l"(z.u));
    return r.f;
  }
  // Columns beyond the strip's end are updated too, with whatever lies behind
  // the pivot row (within the exchange's memory): the packed multiply-adds cost
  // less than the branches around them, which would expose the loads' latency
  // once per group.
  __device__ __forceinline__ void update(int i0, int jb, cx<float> l, const uint4* u, int) {
    const float2 nr = make_float2(-l.re, -l.re), ni = make_float2(-l.im, -l.im), pi = make_float2(l.im, l.im);
    auto pair = [&](int k) {
      const float4 v = *reinterpret_cast<const float4*>(u + k);
      const float2 ur = make_float2(v.x, v.y), ui = make_float2(v.z, v.w);
      const float2 re = fma2(pi, ui, fma2(nr, ur, make_float2(x[k].x, x[k].y)));
      const float2 im = fma2(ni, ur, fma2(nr, ui, make_float2(x[k].z, x[k].w)));
      x[k] = make_float4(re.x, re.y, im.x, im.y);
    };
    if (i0 & 1) {  // the pair's second column alone
      const float4 v = *reinterpret_cast<const float4*>(u + i0 / 2);
      set(i0, fnma(get(i0), l, cx<float>(v.y, v.w)));
    }
#pragma unroll
    for (int k = 0; k < W / 4; ++k)
      if (2 * k >= i0) pair(k);
    if (jb < W / 2)
#pragma unroll
      for (int k = W / 4; k < W / 2; ++k) pair(k);
  }
  __device__ __forceinline__ void shift() {
#pragma unroll
    for (int i = 0; i + kGrp / 2 < W / 2; ++i) x[i] = x[i + kGrp / 2];
  }
};

// complex128: a step updates only the next column before its pivot is
// searched; the others follow while the exchange is under way (up to 3800
// cycles of fp64 multiply-adds a step, half that on average). The candidate's
// row, whose other columns are a step behind in its registers, is brought up
// to date by half a warp, a column per lane, on its way out.
template <class T>
constexpr bool kAhead = sizeof(T) == 8;

// What the cluster's CTAs send one another, at the start of the dynamic shared
// memory: per column parity the barrier, every CTA's candidate and its row.
template <class T, int CL>
struct StripShared {
  static constexpr int kCh = strip_w<T>() * (int)sizeof(cx<T>) / 16;  // 16-byte chunks of a row
  static constexpr int kBuf = kAhead<T> ? 3 : 2;  // a pivot row is read until the next one has been sent
  uint64_t colbar[2];
  StripCand<T> cand[2][CL];
  uint4 crow[kBuf][CL][kCh];
  uint4 stage[kCh];  // this CTA's candidate row; behind crow, see StripRow<float>::update
};

template <class T, int CL>
__host__ __device__ constexpr size_t strip_smem(int R, int nother) {
  constexpr int W = strip_w<T>();
  // the exchange, the rows (padded to an even count of elements), the moved rows' other columns
  return sizeof(StripShared<T, CL>) + sizeof(cx<T>) * (((size_t)R * (W + 1) + 1) / 2 * 2 + (size_t)2 * W * nother);
}

template <class T, int CL, int TPR>
__global__ void __launch_bounds__(kStripThreads, 1) strip_panel_kernel(StripArgs<T> a) {
  using Row = StripRow<T, TPR>;
  constexpr int W = strip_w<T>(), LD = W + 1;
  constexpr int kVec = 16 / (int)sizeof(cx<T>);  // columns of a chunk
  using Sh = StripShared<T, CL>;
  static_assert(Sh::kCh == 16, "half a warp sends a row");
  using Key = KeyOf<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int q = (int)cl_rank(), R = a.rows_per_cta, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = tid / TPR, h = tid % TPR;  // this thread's row and its place in it
  const int nwarp = blockDim.x >> 5;
  const int w = a.w, k0 = a.k0;
  // this CTA's rows k0 + q, k0 + q + CL, ...: dealt out one by one, so that the
  // pivot rows (the first ones) and their columns are spread over the cluster
  const int Rq = max(0, (a.n - k0 - q + CL - 1) / CL);
  auto row = [&](int i) { return k0 + q + CL * i; };
  const int nother = a.blk1 - a.blk0 - w, nleft = k0 - a.blk0;
  Sh& sh = *reinterpret_cast<Sh*>(smem_raw);
  cx<T>* S = reinterpret_cast<cx<T>*>(smem_raw + sizeof(Sh));  // (R, LD): the strip's rows
  cx<T>* mv = S + ((size_t)R * LD + 1) / 2 * 2;                // (<= 2 W, nother) moved rows
  __shared__ Key wkey[2][kStripThreads / 32];
  __shared__ unsigned wpos[2][kStripThreads / 32];
  __shared__ cx<T> wval[2][kStripThreads / 32];
  __shared__ int fpos[kStripThreads];
  __shared__ int mlist[2 * W];
  __shared__ int nmoved, fail_s;
  __shared__ cx<T> stage_l;
  volatile int* fail = &fail_s;
  if (tid == 0) {
    bar_init(&sh.colbar[0], 1);
    bar_init(&sh.colbar[1], 1);
    nmoved = 0;
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  grid_wait();  // what the previous kernel on the stream wrote
  for (int e0 = tid; e0 < Rq * W; e0 += 8 * blockDim.x) {  // eight loads in flight per thread
    cx<T> v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + i * blockDim.x, r = e / W, c = e % W;
      v[i] = r < Rq && c < w ? a.A[(int64_t)row(r) * a.lda + k0 + c] : cx<T>();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + i * blockDim.x, r = e / W, c = e % W;
      if (r < Rq) S[r * LD + c] = v[i];
    }
  }
  // the peers a lane sends to: its half-warp's chunks go to CTAs (lane / 16),
  // that + 2, ...; the candidates to CTA lane
  uint32_t peer[CL / 2];
#pragma unroll
  for (int i = 0; i < CL / 2; ++i) peer[i] = cl_map(&sh, (lane >> 4) + 2 * i);
  const uint32_t cpeer = cl_map(&sh, lane < CL ? lane : 0), self = (uint32_t)__cvta_generic_to_shared(&sh);
  auto off = [&](const void* p) { return (uint32_t)__cvta_generic_to_shared(p) - self; };
  __syncthreads();
  Row x;
  if (r < Rq) x.load(S + r * LD, h);
  unsigned pos = (unsigned)row(r);
  bool live = r < Rq;  // not yet a pivot row
  cl_sync();             // every CTA runs, with its barriers set up, before the first push
  cx<T> lp;                      // kAhead: this row's multiplier of the step before,
  const uint4* pu = nullptr;     // its pivot row,
  bool pend = false;             // and whether the columns after the next are still to be updated with them
  int buf = 0;
  const int hw = kAhead<T> && blockDim.x >= (unsigned)(TPR * R) + 64 ? nwarp - 2 : -1;  // the first of two warps without rows
  // the staged row to all CTAs, a half warp for half of them; l: kAhead, its multiplier of the step before
  auto put_row = [&](int j, int par, cx<T> l) {
    const int c = lane & 15;
    if (c < j / kVec) return;
    uint4 v = sh.stage[c];
    if constexpr (kAhead<T>)
      if (pend && c > j) v = Row::pack(fnma(Row::sent(sh.stage, c), l, Row::sent(pu, c)));
    const uint32_t oc = off(&sh.crow[buf][q][c]), ob = off(&sh.colbar[par]);
#pragma unroll
    for (int i = 0; i < CL / 2; ++i) cl_put(peer[i] + oc, v, peer[i] + ob);
  };
  // the candidate with the reciprocal pivot, both parts in one division: the even lanes the real, the odd ones the
  // imaginary part
  auto reciprocal = [&](cx<T> pv) {
    T m2 = pv.re * pv.re + pv.im * pv.im, f = T(1);
    const bool plain = square_in_range(m2);  // the same in the whole warp
    if (!plain) {
      f = pivot_scale(pv);
      pv = pv * f;
      m2 = pv.re * pv.re + pv.im * pv.im;
    }
    const T half = ((lane & 1) ? -pv.im : pv.re) / m2;
    return plain ? half : half * f;
  };
  auto put_candidate = [&](T half, Key key, unsigned p, int par) {
    union {
      uint4 v[sizeof(StripCand<T>) / 16];
      StripCand<T> c;
    } u;
    u.c.key = key;
    u.c.pos = (int)p;
    u.c.rre = __shfl_sync(~0u, half, 0);
    u.c.rim = __shfl_sync(~0u, half, 1);
    if (lane < CL) {
      const uint32_t b = cpeer + off(&sh.colbar[par]), d = cpeer + off(&sh.cand[par][q]);
#pragma unroll
      for (int i = 0; i < (int)sizeof(StripCand<T>) / 16; ++i) cl_put(d + 16 * i, u.v[i], b);
    }
  };
#pragma unroll 1
  for (int jb = 0; jb < w; jb += kGrp) {
#pragma unroll
    for (int jj = 0; jj < kGrp; ++jj) {
      const int j = jb + jj;
      if (j >= w) break;
      const int row_j = k0 + j, par = j & 1;
      if (tid == 0)
        bar_expect(&sh.colbar[par], CL * (uint32_t)(sizeof(StripCand<T>) + 16 * (Sh::kCh - j / kVec)));
      // this CTA's candidate: over the warp, then over the warps
      const bool has = TPR == 1 || h == jj % TPR;  // this thread has column jj of its row
      Key key = live && has ? val_key(cabs1(x.get(jj))) : Key(0);
      unsigned p = key ? pos : ~0u;
      key = warp_best(key, p);
      if (lane == 0) {
        wkey[par][warp] = key;
        wpos[par][warp] = p;
      }
      if (hw >= 0 && live && has && key != 0 && pos == p) wval[par][warp] = x.get(jj);
      __syncthreads();
      key = lane < nwarp ? wkey[par][lane] : Key(0);
      p = key ? wpos[par][lane] : ~0u;
      key = warp_best(key, p);
      // its owner stages the row's remaining columns; the owner's warp, or the
      // warps without rows, send them and the candidate to all CTAs
      const bool own = live && key != 0 && pos == p;
      const unsigned ob = __ballot_sync(~0u, own);
      const bool owns = key ? ob != 0 : warp == 0;  // the warp whose lane has the candidate
      if (owns && own) {
        x.stage(jj, jb, sh.stage + jb / kVec, h);
        if (hw >= 0 && h == 0) stage_l = lp;
      }
      if (hw < 0) {
        if (owns) {
          const int lo = key ? __ffs(ob) - 1 + jj % TPR : 0;
          const cx<T> xj = x.get(jj);
          const cx<T> pv(__shfl_sync(~0u, xj.re, lo), __shfl_sync(~0u, xj.im, lo));
          cx<T> l;
          if (kAhead<T>) l = cx<T>(__shfl_sync(~0u, lp.re, lo), __shfl_sync(~0u, lp.im, lo));
          __syncwarp();
          put_row(j, par, l);
          put_candidate(reciprocal(pv), key, p, par);
        }
      } else if (warp == hw) {
        const unsigned wb = __ballot_sync(~0u, lane < nwarp && wpos[par][lane < nwarp ? lane : 0] == p);
        const cx<T> pv = wval[par][key ? __ffs(wb) - 1 : 0];
        put_candidate(reciprocal(pv), key, p, par);
      } else if (warp == hw + 1) {
        if (key) asm volatile("bar.sync 1, 64;\n" ::: "memory");
        put_row(j, par, stage_l);
      } else if (key && owns) {
        asm volatile("bar.arrive 1, 64;\n" ::: "memory");
      }
      if constexpr (kAhead<T>)
        if (pend && (hw < 0 || warp < hw)) x.update(jj + 1, jb, lp, pu + jb, h);
      bar_wait(&sh.colbar[par], (j >> 1) & 1, fail);
      // the pivot among the CTAs' candidates (each warp for itself)
      key = lane < CL ? sh.cand[par][lane < CL ? lane : 0].key : Key(0);
      p = key ? (unsigned)sh.cand[par][lane < CL ? lane : 0].pos : ~0u;
      const unsigned mine = p;
      key = warp_best(key, p);
      if (key <= 1) {  // zero (or not a number) column: no interchange, no scaling
        if (q == 0 && tid == 0) {
          if (*a.info == 0) *a.info = row_j + 1;
          a.ipiv[row_j] = row_j;
        }
        if (live) {
          if (pos == (unsigned)row_j) {
            x.store(jj, jb, S + r * LD + jb, h);
            live = false;
          } else if (has) {
            S[r * LD + j] = x.get(jj);
          }
        }
        pend = false;
        buf = buf + 1 == Sh::kBuf ? 0 : buf + 1;
        continue;
      }
      const int src = __ffs(__ballot_sync(~0u, mine == p)) - 1;  // positions are distinct: one CTA
      if (q == 0 && tid == 0) a.ipiv[row_j] = p < (unsigned)a.n ? (int)p : row_j;
      cx<T> xj = x.get(jj);
      if (TPR > 1) {
        const int from = (lane & ~(TPR - 1)) | jj % TPR;
        xj = cx<T>(__shfl_sync(~0u, xj.re, from), __shfl_sync(~0u, xj.im, from));
      }
      if (live) {
        if (pos == p) {
          pos = (unsigned)row_j;
          live = false;
        } else {
          if (pos == (unsigned)row_j) pos = p;
          const cx<T> rp(sh.cand[par][src].rre, sh.cand[par][src].rim);
          const cx<T> l = xj * rp;
          if (has) S[r * LD + j] = l;
          if constexpr (kAhead<T>) {
            lp = l;
            if (j + 1 < W && (TPR == 1 || h == (jj + 1) % TPR)) x.set(jj + 1, fnma(x.get(jj + 1), l, Row::sent(sh.crow[buf][src], j + 1)));
          } else {
            x.update(jj + 1, jb, l, &sh.crow[buf][src][jb / kVec], h);
          }
        }
      }
      // the pivot row's columns from j on, final now, from the exchange to its place (its owner's warp)
      if (src == q && ob != 0 && lane >= j && lane < W)
        S[(warp * 32 + __ffs(ob) - 1) / TPR * LD + lane] = Row::sent(sh.crow[buf][src], lane);
      pend = true;
      pu = sh.crow[buf][src];
      buf = buf + 1 == Sh::kBuf ? 0 : buf + 1;
    }
    x.shift();
  }
  grid_trigger();
  // rows to their positions; rows that moved or became pivot rows take the
  // block's other columns along
  if (r < Rq && h == 0) {
    fpos[r] = (int)pos;
    if (nother > 0 && (pos != (unsigned)row(r) || pos < (unsigned)(k0 + w))) {
      const int i = atomicAdd(&nmoved, 1);
      if (i < 2 * W) mlist[i] = r;
    }
  }
  __syncthreads();
  const int nm = min(nmoved, 2 * W), ne = nm * nother;
  auto other = [&](int c) { return c < nleft ? a.blk0 + c : a.blk0 + w + c; };
  const bool dead = *fail != 0;
  // all threads on all moved rows, eight loads in flight each
  for (int e0 = tid; e0 < ne; e0 += 8 * blockDim.x) {
    cx<T> v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = min(e0 + i * (int)blockDim.x, ne - 1), m = e / nother;
      v[i] = a.A[(int64_t)row(mlist[m]) * a.lda + other(e - m * nother)];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (e0 + i * (int)blockDim.x < ne) mv[e0 + i * blockDim.x] = v[i];
  }
  if (!dead)
#pragma unroll 4
    for (int e = tid; e < Rq * W; e += blockDim.x) {
      const int r = e / W, c = e % W, fp = fpos[r];
      if (c < w && fp >= k0 && fp < a.n) a.A[(int64_t)fp * a.lda + k0 + c] = S[r * LD + c];
    }
  // every moved row has been read, and no CTA leaves while a peer may still store into its shared memory
  cl_sync();
  if (dead) {
    if (tid == 0) atomicExch(a.err, 1);
    return;
  }
#pragma unroll 4
  for (int e = tid; e < ne; e += blockDim.x) {
    const int m = e / nother, c = e - m * nother, fp = fpos[mlist[m]];
    if (fp < k0 || fp >= a.n) continue;
    const cx<T> v = mv[e];
    a.A[(int64_t)fp * a.lda + other(c)] = v;
    if (fp < k0 + w && c >= nleft) a.Ub[(int64_t)(fp - k0) * (nother - nleft) + c - nleft] = v;
  }
}

// After a strip of W columns at k0: on the columns c0 .. c0 + nc - 1 right of
// it (c0 = k0 + W) U12 = L11^-1 Ub, and A22 -= L21 U12. A CTA takes TR rows and
// CG columns and solves for its columns' U12 itself (W^2 / 2 products for each
// of its CG columns against the TR W ones of the update; 8 lanes per column as
// in swap_trsm_kernel); the first row of CTAs stores it.
template <class T>
struct StripUpd {
  static constexpr int W = strip_w<T>(), CG = sizeof(T) == 4 ? 32 : 16, TR = sizeof(T) == 4 ? 64 : 16;
};

template <class T>
__global__ void __launch_bounds__(256) strip_update_kernel(cx<T>* __restrict__ A, int64_t lda, int n, int k0, int nc,
                                                           const cx<T>* __restrict__ Ub) {
  constexpr int W = StripUpd<T>::W, CG = StripUpd<T>::CG, TR = StripUpd<T>::TR;
  __shared__ __align__(16) cx<T> Lt[W][W + 1];   // Lt[t][r] = L11[r][t] below the diagonal
  __shared__ __align__(16) cx<T> V[W][CG + 1];
  __shared__ __align__(16) cx<T> L[TR][W + 1];
  const int tid = threadIdx.x, c0 = k0 + W;
  const int cb = blockIdx.x * CG, rb = c0 + blockIdx.y * TR;
  grid_wait();
  grid_trigger();
  // outputs of this thread: column tc, rows tr + i * kRs
  constexpr int kRs = 256 / CG, kOut = TR / kRs;
  const int tc = tid % CG, tr = tid / CG;
  cx<T> c[kOut];
#pragma unroll
  for (int i = 0; i < kOut; ++i) {
    const int r = rb + tr + i * kRs;
    c[i] = r < n && cb + tc < nc ? A[(int64_t)r * lda + c0 + cb + tc] : cx<T>();
  }
  for (int e = tid; e < W * W; e += 256) {
    const int r = e / W, t = e % W;
    Lt[t][r] = t < r ? A[(int64_t)(k0 + r) * lda + k0 + t] : cx<T>();
  }
  for (int e = tid; e < W * CG; e += 256) {
    const int t = e / CG, k = e % CG;
    V[t][k] = cb + k < nc ? Ub[(int64_t)t * nc + cb + k] : cx<T>();
  }
  for (int e = tid; e < TR * W; e += 256) {
    const int r = e / W, t = e % W;
    L[r][t] = rb + r < n ? A[(int64_t)(rb + r) * lda + k0 + t] : cx<T>();
  }
  __syncthreads();
  if (tid < 8 * CG) {  // whole warps
    const int lane = tid & 31, l8 = lane & 7, col = tid >> 3;
    constexpr int kR = W / 8;
    cx<T> x[kR];
#pragma unroll
    for (int k = 0; k < kR; ++k) x[k] = V[l8 + 8 * k][col];
#pragma unroll
    for (int kb = 0; kb < kR; ++kb)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int t = 8 * kb + j;
        cx<T> xt;
        xt.re = __shfl_sync(~0u, x[kb].re, (lane & ~7) | j);
        xt.im = __shfl_sync(~0u, x[kb].im, (lane & ~7) | j);
#pragma unroll
        for (int k = kb; k < kR; ++k)
          if (k > kb || l8 > j) x[k] = fnma(x[k], ldc(&Lt[t][l8 + 8 * k]), xt);
      }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kR; ++k) V[l8 + 8 * k][col] = x[k];
  }
  __syncthreads();
  if (blockIdx.y == 0)
    for (int e = tid; e < W * CG; e += 256) {
      const int t = e / CG, k = e % CG;
      if (cb + k < nc) A[(int64_t)(k0 + t) * lda + c0 + cb + k] = V[t][k];
    }
#pragma unroll 8
  for (int t = 0; t < W; ++t) {
    const cx<T> u = ldc(&V[t][tc]);
#pragma unroll
    for (int i = 0; i < kOut; ++i) c[i] = fnma(c[i], ldc(&L[tr + i * kRs][t]), u);
  }
#pragma unroll
  for (int i = 0; i < kOut; ++i) {
    const int r = rb + tr + i * kRs;
    if (r < n && cb + tc < nc) A[(int64_t)r * lda + c0 + cb + tc] = c[i];
  }
}

// whether clusters of 16 CTAs with the panel's shared memory can be launched (decided once per element type)
template <class T>
bool strip_available(int device) {
  static const bool ok = [device] {
    int optin = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return false;
    const int smem = (int)strip_smem<T, 16>(kStripThreads, 128 - strip_w<T>());
    const char* off = getenv("M25_NO_CLUSTER_PANEL");
    bool yes = !(off && *off == '1') && smem + 8192 <= optin &&
               cudaFuncSetAttribute(strip_panel_kernel<T, 16, 1>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(strip_panel_kernel<T, 16, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(strip_panel_kernel<T, 8, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
                   cudaSuccess;
    if constexpr (sizeof(T) == 4)
      yes = yes && cudaFuncSetAttribute(strip_panel_kernel<T, 4, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        smem) == cudaSuccess;
    if constexpr (sizeof(T) == 8) {
      const auto set = [&](auto kernel, bool wide) {
        yes = yes && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
              (!wide || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
      };
      set(strip_panel_kernel<T, 8, 2>, false);
      set(strip_panel_kernel<T, 8, 4>, false);
      set(strip_panel_kernel<T, 16, 2>, true);
      set(strip_panel_kernel<T, 16, 4>, true);
    }
    if (yes) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 16;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(16);
      cfg.blockDim = dim3(kStripThreads);
      cfg.dynamicSmemBytes = smem;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nclusters = 0;
      yes = cudaOccupancyMaxActiveClusters(&nclusters, strip_panel_kernel<T, 16, 1>, &cfg) == cudaSuccess && nclusters > 0;
    }
    cudaGetLastError();  // a refused attribute only means: no cluster panel
    return yes;
  }();
  return ok;
}

template <class T, int CL, int TPR = 1>
cudaError_t launch_strip(const StripArgs<T>& a, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(CL);
  const int rows = (TPR * a.rows_per_cta + 31) / 32 * 32;
  cfg.blockDim = dim3(kAhead<T> && rows + 64 <= kStripThreads ? rows + 64 : std::max(64, rows));
  cfg.dynamicSmemBytes = strip_smem<T, CL>(a.rows_per_cta, a.blk1 - a.blk0 - a.w);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, strip_panel_kernel<T, CL, TPR>, a);
}

// complex128: as many lanes per row as give the four sub-partitions of the SM a warp each, as each has its own fp64
// unit (panel of N = 546 / 1085: 1.75 / 3.52 -> 1.43 / 2.98 ms). Beyond 64 rows the warps of single lanes already share
// them out: two lanes each would only double the warps.
template <class T, int CL>
cudaError_t launch_rows(const StripArgs<T>& a, cudaStream_t st) {
  if constexpr (sizeof(T) == 8) {
    if (a.rows_per_cta <= 32) return launch_strip<T, CL, 4>(a, st);
    if (a.rows_per_cta <= 64) return launch_strip<T, CL, 2>(a, st);
  }
  return launch_strip<T, CL>(a, st);
}

}  // namespace

// rows a block's panel can have (0: clusters are not available)
template <class T>
int lu_strip_rows(m25_ctx* ctx) {
  return strip_available<T>(ctx->device) ? kStripThreads * kStripMaxCl : 0;
}

template <class T>
size_t lu_strip_scratch() {
  return sizeof(cx<T>) * strip_w<T>() * 128;
}

// The block of columns b0 .. b0 + bw - 1 (bw <= 128) of the rows b0 .. n - 1,
// with its interchanges on the block's columns alone; Ub: lu_strip_scratch bytes.
template <class T>
int lu_strip_block(m25_ctx* ctx, cx<T>* A, int64_t lda, int n, int b0, int bw, int32_t* ipiv, int* info, int* err,
                   cx<T>* Ub, int cl_min) {
  constexpr int W = strip_w<T>();
  for (int k0 = b0; k0 < b0 + bw; k0 += W) {
    const int w = std::min(W, b0 + bw - k0), m = n - k0;
    // complex64: the smallest cluster that holds the rows (at least cl_min); complex128: the fp64
    // multiply-adds of 16 SMs, unless the rows are few
    int CL = m <= 4 * kStripThreads ? 4 : m <= 8 * kStripThreads ? 8 : 16;
    CL = std::max(CL, cl_min);
    if (sizeof(T) == 8) CL = std::max(CL, m > 256 ? 16 : 8);
    StripArgs<T> a{A, lda, n, k0, w, b0, b0 + bw, (m + CL - 1) / CL, ipiv, Ub, info, err};
    StageTimer tm(ctx, ST_PANEL);
    if (CL == 16) {
      M25_CUDA((launch_rows<T, 16>(a, ctx->stream)));
    } else if (CL == 8) {
      M25_CUDA((launch_rows<T, 8>(a, ctx->stream)));
    } else {
      if constexpr (sizeof(T) == 4) M25_CUDA((launch_strip<T, 4>(a, ctx->stream)));
    }
    const int nc = b0 + bw - k0 - w;
    if (nc > 0) {
      const dim3 grid((nc + StripUpd<T>::CG - 1) / StripUpd<T>::CG, (n - k0 - w + StripUpd<T>::TR - 1) / StripUpd<T>::TR);
      M25_CUDA(launch_chained(strip_update_kernel<T>, grid, 256, 0, ctx->stream, A, lda, n, k0, nc, Ub));
    }
  }
  return M25_OK;
}

template int lu_strip_rows<float>(m25_ctx*);
template int lu_strip_rows<double>(m25_ctx*);
template size_t lu_strip_scratch<float>();
template size_t lu_strip_scratch<double>();
template int lu_strip_block<float>(m25_ctx*, zf*, int64_t, int, int, int, int32_t*, int*, int*, zf*, int);
template int lu_strip_block<double>(m25_ctx*, zd*, int64_t, int, int, int, int32_t*, int*, int*, zd*, int);

}  // namespace m25
