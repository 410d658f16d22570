// The panel of the dense LU (lu.cu): one block of columns is factored strip by
// strip (32 columns of complex64, 16 of complex128), each strip by
//   strip_panel_kernel   one cluster of up to 16 CTAs, the strip's rows in registers
//   strip_update_kernel  U12 of the block's columns right of the strip and their
//                        rank-W update, on the whole GPU
// The panel is a chain of column steps (pivot search, exchange, rank-1
// update), so what bounds it is the latency of a step and, in complex128, the
// rate of fp64 multiply-adds of the SMs that hold the rows (two per clock and
// SM). Hence:
//  - one row per thread, its W columns in registers: a step reads only the
//    pivot row from shared memory, and has one CTA barrier and one wait for the
//    cluster's exchange;
//  - rows are not moved while the strip is factored: a thread follows the
//    position of its row through the interchanges and writes it there at the
//    end, so the row at position k0 + j need not be sent around;
//  - narrow strips: the rank-1 updates of a step cost W / 2 columns on
//    average, and the products between strips go to the whole GPU.
// Measured on GB300 (one factorisation alone, sum over its panels):
//   complex128, N = 546 / 1085 / 2434 / 5943: 2.2 / 4.4 / 10.4 / 32 ms (7.95 / 20.0 / 53.0 / 96.6 ms for
//   64-column panels in shared memory, with the row k0 + j sent around and both divisions on the chain)
//   complex64, N = 1085 / 5943: 2.0 / 11.9 ms (2.5 / 21.1 ms, and 0.2 / 2.1 ms for the products between
//   the two panels of a block)
// A column step of complex64 takes 1.25 us, of which 0.45 us are the exchange's flight.
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
  return v >= 0.0 ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
}
template <class T>
using KeyOf = decltype(val_key(T(0)));

template <class T, int CL>
__host__ __device__ constexpr size_t strip_smem(int R, int nother) {
  constexpr int W = strip_w<T>();
  // the rows (padded to an even count of elements), candidate rows of both parities, the moved rows' other columns
  return sizeof(cx<T>) * (((size_t)R * (W + 1) + 1) / 2 * 2 + 2 * CL * W + (size_t)2 * W * nother);
}

template <class T, int CL>
__global__ void __launch_bounds__(kStripThreads, 1) strip_panel_kernel(StripArgs<T> a) {
  constexpr int W = strip_w<T>(), LD = W + 1;
  constexpr int kVec = 16 / (int)sizeof(cx<T>);  // elements of a 16-byte store
  using Key = KeyOf<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int q = (int)cl_rank(), R = a.rows_per_cta, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarp = blockDim.x >> 5;
  const int w = a.w, k0 = a.k0, r0 = k0 + q * R;
  const int Rq = max(0, min(a.n, r0 + R) - r0);
  const int nother = a.blk1 - a.blk0 - w, nleft = k0 - a.blk0;
  cx<T>* S = reinterpret_cast<cx<T>*>(smem_raw);              // (R, LD): the strip's rows
  cx<T>* crow = S + ((size_t)R * LD + 1) / 2 * 2;              // (2, CL, W) candidate rows
  cx<T>* mv = crow + 2 * CL * W;                               // (<= 2 W, nother) moved rows
  __shared__ StripCand<T> cand[2][CL];
  __shared__ Key wkey[2][kStripThreads / 32];
  __shared__ unsigned wpos[2][kStripThreads / 32];
  __shared__ int fpos[kStripThreads];
  __shared__ int mlist[2 * W];
  __shared__ int nmoved, fail_s;
  __shared__ __align__(8) uint64_t colbar[2];
  volatile int* fail = &fail_s;
  if (tid == 0) {
    bar_init(&colbar[0], 1);
    bar_init(&colbar[1], 1);
    nmoved = 0;
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  for (int e0 = tid; e0 < Rq * W; e0 += 8 * blockDim.x) {  // eight loads in flight per thread
    cx<T> v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + i * blockDim.x, r = e / W, c = e % W;
      v[i] = r < Rq && c < w ? a.A[(int64_t)(r0 + r) * a.lda + k0 + c] : cx<T>();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + i * blockDim.x, r = e / W, c = e % W;
      if (r < Rq) S[r * LD + c] = v[i];
    }
  }
  __syncthreads();
  cx<T> x[W];  // x[i]: column jb + i of this thread's row
  if (tid < Rq)
#pragma unroll
    for (int c = 0; c < W; ++c) x[c] = S[tid * LD + c];
  unsigned pos = (unsigned)(r0 + tid);
  bool live = tid < Rq;  // not yet a pivot row
  cl_sync();             // every CTA runs, with its barriers set up, before the first push
#pragma unroll 1
  for (int jb = 0; jb < w; jb += kGrp) {
#pragma unroll
    for (int jj = 0; jj < kGrp; ++jj) {
      const int j = jb + jj;
      if (j >= w) break;
      const int row_j = k0 + j, par = j & 1;
      // this CTA's candidate: over the warp, then over the warps
      Key key = live ? val_key(cabs1(x[jj])) : Key(0);
      unsigned p = key ? pos : ~0u;
      key = warp_best(key, p);
      if (lane == 0) {
        wkey[par][warp] = key;
        wpos[par][warp] = p;
      }
      if (tid == 0)
        bar_expect(&colbar[par],
                   CL * (uint32_t)(sizeof(StripCand<T>) + (W - j / kVec * kVec) * sizeof(cx<T>)));
      __syncthreads();
      key = lane < nwarp ? wkey[par][lane] : Key(0);
      p = key ? wpos[par][lane] : ~0u;
      key = warp_best(key, p);
      // its owner puts the row's remaining columns into shared memory, and the
      // owner's warp sends them with the candidate to all CTAs
      const bool own = live && key != 0 && pos == p;
      const unsigned ob = __ballot_sync(~0u, own);
      if (key ? ob != 0 : warp == 0) {
        const int ro = key ? (warp * 32 + __ffs(ob) - 1) : 0;
        if (own)
#pragma unroll
          for (int i = 0; i < W; ++i)
            if (i >= jj && jb + i < W) S[ro * LD + jb + i] = x[i];
        __syncwarp();
        constexpr int kCh = W / kVec;
        for (int e = lane; e < CL * kCh; e += 32) {
          const int dst = e / kCh, c = (e % kCh) * kVec;
          if (c + kVec > j) {
            union {
              uint4 v;
              cx<T> z[kVec];
            } u = {make_uint4(0, 0, 0, 0)};
#pragma unroll
            for (int i = 0; i < kVec; ++i) u.z[i] = S[ro * LD + c + i];
            cl_put(cl_map(&crow[(par * CL + q) * W + c], dst), u.v, cl_map(&colbar[par], dst));
          }
        }
        const cx<T> pv = S[ro * LD + j];
        const T m2 = pv.re * pv.re + pv.im * pv.im;
        union {
          uint4 v[sizeof(StripCand<T>) / 16];
          StripCand<T> c;
        } u;
        u.c.key = key;
        u.c.pos = (int)p;
        // both parts of the reciprocal in one division: the even lanes the real, the odd ones the imaginary part
        const T half = ((lane & 1) ? -pv.im : pv.re) / m2;
        u.c.rre = __shfl_sync(~0u, half, 0);
        u.c.rim = __shfl_sync(~0u, half, 1);
        if (lane < CL) {
          const uint32_t b = cl_map(&colbar[par], lane), d = cl_map(&cand[par][q], lane);
#pragma unroll
          for (int i = 0; i < (int)sizeof(StripCand<T>) / 16; ++i) cl_put(d + 16 * i, u.v[i], b);
        }
      }
      bar_wait(&colbar[par], (j >> 1) & 1, fail);
      // the pivot among the CTAs' candidates (each warp for itself)
      key = lane < CL ? cand[par][lane < CL ? lane : 0].key : Key(0);
      p = key ? (unsigned)cand[par][lane < CL ? lane : 0].pos : ~0u;
      const unsigned mine = p;
      key = warp_best(key, p);
      if (key <= 1) {  // zero (or not a number) column: no interchange, no scaling
        if (q == 0 && tid == 0) {
          if (*a.info == 0) *a.info = row_j + 1;
          a.ipiv[row_j] = row_j;
        }
        if (live) {
          if (pos == (unsigned)row_j) {
#pragma unroll
            for (int i = 0; i < W; ++i)
              if (i >= jj && jb + i < W) S[tid * LD + jb + i] = x[i];
            live = false;
          } else {
            S[tid * LD + j] = x[jj];
          }
        }
        continue;
      }
      const int src = __ffs(__ballot_sync(~0u, mine == p)) - 1;  // positions are distinct: one CTA
      if (q == 0 && tid == 0) a.ipiv[row_j] = p < (unsigned)a.n ? (int)p : row_j;
      if (live) {
        if (pos == p) {
          pos = (unsigned)row_j;
          live = false;
        } else {
          if (pos == (unsigned)row_j) pos = p;
          const cx<T> rp(cand[par][src].rre, cand[par][src].rim);
          const cx<T> l = x[jj] * rp;
          S[tid * LD + j] = l;
          const cx<T>* u = crow + (par * CL + src) * W + jb;
#pragma unroll
          for (int i = jj + 1; i < kGrp; ++i) x[i] = fnma(x[i], l, u[i]);
#pragma unroll
          for (int g = 1; g < W / kGrp; ++g)
            if (jb + g * kGrp < W)
#pragma unroll
              for (int i = 0; i < kGrp; ++i) x[g * kGrp + i] = fnma(x[g * kGrp + i], l, u[g * kGrp + i]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i + kGrp < W; ++i) x[i] = x[i + kGrp];
  }
  // rows to their positions; rows that moved or became pivot rows take the
  // block's other columns along
  if (tid < Rq) {
    fpos[tid] = (int)pos;
    if (nother > 0 && (pos != (unsigned)(r0 + tid) || pos < (unsigned)(k0 + w))) {
      const int i = atomicAdd(&nmoved, 1);
      if (i < 2 * W) mlist[i] = tid;
    }
  }
  __syncthreads();
  const int nm = min(nmoved, 2 * W);
  auto other = [&](int c) { return c < nleft ? a.blk0 + c : a.blk0 + w + c; };
  if (nother > 0)
    for (int i = warp; i < nm; i += nwarp) {
      const cx<T>* row = a.A + (int64_t)(r0 + mlist[i]) * a.lda;
#pragma unroll 4
      for (int c = lane; c < nother; c += 32) mv[i * nother + c] = row[other(c)];
    }
  if (!*fail)
    for (int e = tid; e < Rq * W; e += blockDim.x) {
      const int r = e / W, c = e % W, fp = fpos[r];
      if (c < w && fp >= k0 && fp < a.n) a.A[(int64_t)fp * a.lda + k0 + c] = S[r * LD + c];
    }
  // every moved row has been read, and no CTA leaves while a peer may still store into its shared memory
  cl_sync();
  if (*fail) {
    if (tid == 0) atomicExch(a.err, 1);
    return;
  }
  for (int i = warp; i < nm; i += nwarp) {
    const int fp = fpos[mlist[i]];
    if (fp < k0 || fp >= a.n) continue;
    for (int c = lane; c < nother; c += 32) {
      const cx<T> v = mv[i * nother + c];
      a.A[(int64_t)fp * a.lda + other(c)] = v;
      if (fp < k0 + w && c >= nleft) a.Ub[(int64_t)(fp - k0) * (nother - nleft) + c - nleft] = v;
    }
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
  __shared__ cx<T> Lt[W][W + 1];   // Lt[t][r] = L11[r][t] below the diagonal
  __shared__ cx<T> V[W][CG + 1];
  __shared__ cx<T> L[TR][W + 1];
  const int tid = threadIdx.x, c0 = k0 + W;
  const int cb = blockIdx.x * CG, rb = c0 + blockIdx.y * TR;
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
          if (k > kb || l8 > j) x[k] = fnma(x[k], Lt[t][l8 + 8 * k], xt);
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
    const cx<T> u = V[t][tc];
#pragma unroll
    for (int i = 0; i < kOut; ++i) c[i] = fnma(c[i], L[tr + i * kRs][t], u);
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
               cudaFuncSetAttribute(strip_panel_kernel<T, 16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(strip_panel_kernel<T, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(strip_panel_kernel<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(strip_panel_kernel<T, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
                   cudaSuccess;
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
      yes = cudaOccupancyMaxActiveClusters(&nclusters, strip_panel_kernel<T, 16>, &cfg) == cudaSuccess && nclusters > 0;
    }
    cudaGetLastError();  // a refused attribute only means: no cluster panel
    return yes;
  }();
  return ok;
}

template <class T, int CL>
cudaError_t launch_strip(const StripArgs<T>& a, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(CL);
  cfg.blockDim = dim3(std::max(64, (a.rows_per_cta + 31) / 32 * 32));
  cfg.dynamicSmemBytes = strip_smem<T, CL>(a.rows_per_cta, a.blk1 - a.blk0 - a.w);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, strip_panel_kernel<T, CL>, a);
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
    if (CL == 4) M25_CUDA((launch_strip<T, 4>(a, ctx->stream)));
    else if (CL == 8) M25_CUDA((launch_strip<T, 8>(a, ctx->stream)));
    else M25_CUDA((launch_strip<T, 16>(a, ctx->stream)));
    const int nc = b0 + bw - k0 - w;
    if (nc > 0) {
      const dim3 grid((nc + StripUpd<T>::CG - 1) / StripUpd<T>::CG, (n - k0 - w + StripUpd<T>::TR - 1) / StripUpd<T>::TR);
      strip_update_kernel<T><<<grid, 256, 0, ctx->stream>>>(A, lda, n, k0, nc, Ub);
      M25_CHECK_LAUNCH();
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
