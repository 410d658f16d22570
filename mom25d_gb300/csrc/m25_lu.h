// What the translation units of the dense LU share (lu.cu, lu_panel.cu, lu_oz.cu).
#pragma once

#include "m25_internal.h"

namespace m25 {

// lu_panel.cu: a block of at most 128 columns factored by one cluster (up to lu_strip_rows rows)
template <class T> int lu_strip_rows(m25_ctx* ctx);
template <class T> size_t lu_strip_scratch();
template <class T>
int lu_strip_block(m25_ctx* ctx, cx<T>* A, int64_t lda, int n, int b0, int bw, int32_t* ipiv, int* info, int* err,
                   cx<T>* Ub, int cl_min);

// lu_oz.cu: the complex128 trailing update of a block of 64 columns on the tensor cores
int lu_oz_prepare(m25_ctx* ctx, int n);
int lu_oz_update(m25_ctx* ctx, zd* A, int64_t lda, int n, int k0);
// the same on the CUDA cores, bit for bit (work: 1 KB on the device)
int lu_oz_update_simt(m25_ctx* ctx, zd* A, int64_t lda, int n, int k0, void* work);

}  // namespace m25
