// rowsplit.cuh -- block rows dealt to several lane groups (rowsplit.cu).
#pragma once

#include "internal.cuh"

namespace mg {

// y = alpha A x + beta yin, and the damped block-Jacobi sweep, for square
// blocks whose rows are long and few; false: not a level for this form
template <class T>
bool split_spmv(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, T alpha, const T* x, T beta, const T* yin, T* y,
                int kclass);
template <class T>
bool split_jacobi(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b, const T* xin, T* xout,
                  T omega, bool xzero);

}  // namespace mg
