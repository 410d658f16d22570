// What the translation units of the dense LU share (lu.cu, lu_panel.cu, lu_oz.cu).
#pragma once

#include "m25_internal.h"

namespace m25 {

// Programmatic dependent launch: a kernel launched by launch_chained starts when
// every CTA of the one before it on the stream has triggered (or ended), and
// waits in grid_wait for that one's end; what comes before the wait overlaps it.
// Every CTA of a chained kernel waits, so that the end of a kernel means the end
// of all before it.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

template <class... K, class... A>
cudaError_t launch_chained(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}

// lu_panel.cu: a block of at most 128 columns factored by one cluster (up to lu_strip_rows rows)
template <class T> int lu_strip_rows(m25_ctx* ctx);
template <class T> size_t lu_strip_scratch();
template <class T>
int lu_strip_block(m25_ctx* ctx, cx<T>* A, int64_t lda, int n, int b0, int bw, int32_t* ipiv, int* info, int* err,
                   cx<T>* Ub, int cl_min);

// lu_oz.cu: the complex128 trailing update of a block of 64 columns on the tensor cores
int lu_oz_prepare(m25_ctx* ctx, int n);
int lu_oz_update(m25_ctx* ctx, zd* A, int64_t lda, int n, int k0);
// the same on the CUDA cores, bit for bit (work: 1.5 KB on the device)
int lu_oz_update_simt(m25_ctx* ctx, zd* A, int64_t lda, int n, int k0, void* work);

}  // namespace m25
