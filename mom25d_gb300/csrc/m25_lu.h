// What the translation units of the dense LU share (lu.cu, lu_panel.cu).
#pragma once

#include "m25_internal.h"

namespace m25 {

// lu_panel.cu: a block of at most 128 columns factored by one cluster (up to lu_strip_rows rows)
template <class T> int lu_strip_rows(m25_ctx* ctx);
template <class T> size_t lu_strip_scratch();
template <class T>
int lu_strip_block(m25_ctx* ctx, cx<T>* A, int64_t lda, int n, int b0, int bw, int32_t* ipiv, int* info, int* err,
                   cx<T>* Ub, int cl_min);

}  // namespace m25
