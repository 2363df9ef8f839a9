// repeat.cuh -- level operators with few distinct blocks (repeat.cu).
#pragma once

#include "internal.cuh"

namespace mg {

// Table form of a square block-sparse operator whose blocks repeat (grids
// with constant coefficients: 17 distinct blocks on every uniform level).
// Rows with the same sequence of
// table entries form a class, and the slots list the rows class by class, gs
// to a group, so that a warp applies one block to many rows at once.
//
// Images: the value tables as the kernels hold them in shared memory, first
// the nuniq blocks (by columns, or by rows where fewer rows than columns hold
// nonzeros), then the ndiag distinct inverse diagonal blocks (by rows); a
// block is b lines of ld values, for b = 16 with 16 bytes between lines 7 and
// 8 (the two column halves of a line pair then lie in different banks).
struct RepView {
    int b = 0, ld = 0, nbr = 0, nuniq = 0, ndiag = 0, ncls = 0;
    int gs = 16, gu = 16;          // slots per group, every group one class; slots per gcls entry
    int nslots = 0;
    unsigned* mask = nullptr;      // [nuniq] nonzero rows | nonzero columns << 16
    int* cls = nullptr;            // [ncls][kRepCls]: blocks per row, inverse diagonal block, -, -, entries, their masks
    int* gcls = nullptr;           // [nslots / gu] class of gu consecutive slots
    int* rows = nullptr;           // [nslots] row, -1: padding
    int* cols = nullptr;           // [most blocks per row][nslots] block columns
    double* i64 = nullptr;         // FP64 image
    float *i32 = nullptr, *ilo = nullptr;   // FP32 image and the blocks' low halves (val = i32 + ilo)
    float *i16 = nullptr, *s16 = nullptr;   // block-scaled FP16 values (all by rows), their scales
    // the nuniq blocks by columns (b lines of ld values, no gap between the
    // halves), for the multi-vector kernels
    double* c64 = nullptr;
    float *c32 = nullptr, *clo = nullptr;
};
struct RepTable : RepView {
    void* pool = nullptr;          // owns the value tables and mask
    void* slots = nullptr;         // owns cls, gcls, rows, cols
    RepTable() = default;
    RepTable(const RepTable&) = delete;
    RepTable& operator=(const RepTable&) = delete;
    ~RepTable();
};
constexpr int kRepMaxNb = 12;            // longest row
constexpr int kRepCls = 2 * kRepMaxNb + 4;   // ints per class

// Looks for repeated blocks in a level operator (square blocks of 4, 9 or 16).
// rep_sample queues a count of the distinct blocks in a sample, so that its
// result travels with a synchronisation of the caller; false: no form that the
// hierarchy's precision runs on this level would use a table.  rep_build, given
// that count, looks at all blocks, checks each against its table entry and
// attaches the table to A where one of the forms is faster with it.  Dinv: A's
// inverse diagonal blocks.
bool rep_sample(mgldg_ctx* ctx, const mgldg_bsr* A, int precision, bool finest, int* distinct);
void rep_build(mgldg_ctx* ctx, mgldg_bsr* A, const double* Dinv, int precision, bool finest, int distinct);

// the table for multi-vector products (levels from kRepMmRows rows on, also
// those too small for the single-vector kernels) where they are faster with it:
// FP64 sweeps and products, or (df64) the double-float outer product
void rep_ensure_batch(mgldg_ctx* ctx, mgldg_bsr* A, const double* Dinv, bool df64);
constexpr int kRepMmRows = 2048;
bool rep_mm_pays(int b, int64_t rows, int64_t nuniq);
bool rep_mm_df64_pays(int b, int64_t rows);

// FP64 Y = alpha A X + beta Yin, or (Jacobi) Y = X + omega Dinv (B - A X), on
// row-major multi-vectors of k columns (spmm_rep.cu); false: no table
struct RepMM {
    int k;
    const double *X, *Yin, *B;
    double* Y;
    double alpha, beta, omega;
    int jacobi, xzero;
};
bool rep_spmm(mgldg_ctx* ctx, const mgldg_bsr* A, const RepMM& m, int kclass);
// Q = A D in double-float arithmetic, D as float pairs
bool rep_spmm_df64(mgldg_ctx* ctx, const mgldg_bsr* A, int k, const float* Dhi, const float* Dlo, double* Q);

// y = alpha A x + beta yin with the dot epilogue of spmv; false: no table
template <class T>
bool rep_spmv(mgldg_ctx* ctx, const mgldg_bsr* A, T alpha, const T* x, T beta, const T* yin, T* y, const T* dotv,
              double* partials, int* npart, int kclass, bool f16 = false);
// damped block-Jacobi sweep (xzero: x = 0, not read); false: no table
template <class T>
bool rep_jacobi(mgldg_ctx* ctx, const mgldg_bsr* A, const T* b, const T* xin, T* xout, T omega, bool xzero,
                bool f16 = false);
// q = A d in double-float arithmetic and the partial sums of d.q
bool rep_df64(mgldg_ctx* ctx, const mgldg_bsr* A, const float* dhi, const float* dlo, const double* d, double* q,
              double* partials, int* npart);

}  // namespace mg
