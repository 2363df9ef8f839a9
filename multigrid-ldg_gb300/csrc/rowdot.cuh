// rowdot.cuh -- one warp computes (A x)_i for a block row i of a BSR matrix.
//
// Lane layout: S = 32 / br lanes per block row, each owning a contiguous
// chunk of CH columns.  For up to MAXB blocks at a time the warp first issues
// every load of the row -- the block values (128-bit loads where the row is
// 16-byte aligned; their addresses need no index), then the column indices
// (one lane each, broadcast by shuffle) and the x chunks -- and only then
// does the arithmetic, one fused multiply-add per product, so a warp keeps
// MAXB blocks in flight instead of one.
#pragma once

#include "convert.cuh"
#include "internal.cuh"

namespace mg {

template <class T>
struct V16;
template <>
struct V16<double> { typedef double2 type; static constexpr int n = 2; };
template <>
struct V16<float> { typedef float4 type; static constexpr int n = 4; };

// acc += a . b as a chain of fused multiply-adds (one FMA per product)
__device__ __forceinline__ void vfma(double& acc, const double2& a, const double2& b) {
    acc = fma(a.x, b.x, acc);
    acc = fma(a.y, b.y, acc);
}
__device__ __forceinline__ void vfma(float& acc, const float4& a, const float4& b) {
    acc = fmaf(a.x, b.x, acc);
    acc = fmaf(a.y, b.y, acc);
    acc = fmaf(a.z, b.z, acc);
    acc = fmaf(a.w, b.w, acc);
}

// One product a*d of float pairs added to the float pair (sh, sl): the exact
// FP32 product of the high parts (its error recovered with an FMA) plus the
// two cross terms, added with a two-sum (Dekker's and Knuth's error-free
// transformations; explicitly rounded operations, a contraction would break
// them).
__device__ __forceinline__ void df_fma(float& sh, float& sl, float ah, float al, float dh, float dl) {
    const float p = __fmul_rn(ah, dh);
    const float pe = fmaf(ah, dh, -p);
    const float t = fmaf(ah, dl, fmaf(al, dh, pe));
    const float s = __fadd_rn(sh, p);
    const float bb = __fsub_rn(s, sh);
    const float e = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bb)), __fsub_rn(p, bb));
    sh = s;
    sl = __fadd_rn(sl, __fadd_rn(e, t));
}

// The same for two products at once (packed FP32 operations, each half
// rounded as the scalar one): half the instructions.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    return (unsigned long long)__float_as_uint(b) << 32 | __float_as_uint(a);
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    return make_float2(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// (ndh = -dh: the product enters the two-sum with its sign turned, so nothing
// is negated per product)
__device__ __forceinline__ void df_fma2(unsigned long long& sh, unsigned long long& sl, unsigned long long ah,
                                        unsigned long long al, unsigned long long dh, unsigned long long ndh,
                                        unsigned long long dl) {
    const unsigned long long np = mul2(ah, ndh);
    const unsigned long long t = fma2(ah, dl, fma2(al, dh, fma2(ah, dh, np)));
    const unsigned long long s = sub2(sh, np);
    const unsigned long long bb = sub2(s, sh);
    const unsigned long long e = sub2(sub2(sh, sub2(s, bb)), add2(np, bb));
    sh = s;
    sl = add2(sl, add2(e, t));
}

// One row of the dense coarsest solve, sum_c Cinv(row, c) b_c, by one warp
// (valid in every lane): four 16-byte loads per lane in flight, four partial
// sums per lane added in a fixed order.  Rows of an odd n start on an odd
// entry every second time; the entry before the first 16-byte word and one
// after the last are added apart.  b in shared memory.
//
// The plain loop (up to four 8-byte loads in flight) is the shorter one where a
// lane has eight entries at most: 256 unknowns 2.4 us against 3.2 with Cinv in
// L2, 3.0 / 3.5 from HBM.  Between, the wide loads win when Cinv comes from HBM
// (1,053 unknowns 8.6 / 7.7 us, 1,944 14.3 / 13.0) by more than they lose from L2
// (5.5 / 6.1, 11.1 / 11.6).  Beyond, a CTA's eight warps have rows enough to
// cover the latency, and the plain loop has the fewer instructions: 2,304 16.1 /
// 16.6 (L2 13.6 / 15.2), 4,096 in FP64 V-cycles 40.7 / 43.1.
constexpr int kCoarseWideMin = 257, kCoarseWideMax = 2048;
__device__ __forceinline__ double coarse_row(const double* __restrict__ Cinv, const double* b, int n, int row,
                                             int lane) {
    const double* cr = Cinv + (size_t)row * n;
    if (n < kCoarseWideMin || n > kCoarseWideMax) {
        double s = 0;
        for (int c = lane; c < n; c += 32) s += __ldg(cr + c) * b[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    }
    double a[4] = {0, 0, 0, 0};
    const int head = (int)(((size_t)row * n) & 1);
    if (head && lane == 0) a[0] = __ldg(cr) * b[0];
    const int n2 = (n - head) / 2;
    const double2* c2 = reinterpret_cast<const double2*>(cr + head);
    int c = lane;
    for (; c + 96 < n2; c += 128) {
        double2 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = __ldg(c2 + c + 32 * q);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = head + 2 * (c + 32 * q);
            a[q] = fma(v[q].x, b[e], a[q]);
            a[q] = fma(v[q].y, b[e + 1], a[q]);
        }
    }
    // at most three words are left, loaded together
    double2 v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (c + 32 * q < n2) v[q] = __ldg(c2 + c + 32 * q);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (c + 32 * q < n2) {
            const int e = head + 2 * (c + 32 * q);
            a[0] = fma(v[q].x, b[e], a[0]);
            a[0] = fma(v[q].y, b[e + 1], a[0]);
        }
    if (lane == 0 && head + 2 * n2 < n) a[1] = fma(__ldg(cr + n - 1), b[n - 1], a[1]);
    double s = (a[0] + a[1]) + (a[2] + a[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// can this block shape use 128-bit loads for every lane chunk?
template <class T, int BR, int BC>
struct RowVec {
    using L = WL<BR, BC>;
    static constexpr bool ok = ((BC * sizeof(T)) % 16 == 0) && ((L::CH * sizeof(T)) % 16 == 0) &&
                               (L::CH * L::S == BC) && ((BR * BC * sizeof(T)) % 16 == 0);
    static constexpr int NV = ok ? (int)(L::CH * sizeof(T) / 16) : 1;
};

// Partial (A x)_i over this lane's chunk; reduce with seg_sum<S> afterwards.
// XL: load x through the read-only path (true) or through L2 (false, when x
// changes during the kernel).
template <class T, int BR, int BC, int MAXB, bool XL = true>
__device__ __forceinline__ T row_dot(const int* __restrict__ col_idx, const T* __restrict__ val,
                                     const int* __restrict__ blk, const T* x, int k0, int k1, int r, int c0,
                                     bool active, int lane) {
    using L = WL<BR, BC>;
    using RV = RowVec<T, BR, BC>;
    T acc = 0;
    for (int kb = k0; kb < k1; kb += MAXB) {
        const int nb = min(MAXB, k1 - kb);
        // block values first: their addresses need no loaded index (unless
        // the matrix stores a block table), so they go out immediately
        if constexpr (RV::ok) {
            typedef typename V16<T>::type V;
            V av[MAXB][RV::NV], xv[MAXB][RV::NV];
#pragma unroll
            for (int q = 0; q < MAXB; ++q)
                if (q < nb && active) {
                    const int bq = blk ? __ldg(blk + kb + q) : kb + q;
                    const V* ap = reinterpret_cast<const V*>(val + (size_t)bq * (BR * BC) + r * BC + c0);
#pragma unroll
                    for (int v = 0; v < RV::NV; ++v) av[q][v] = __ldg(ap + v);
                }
            const int jl = (lane < nb) ? __ldg(col_idx + kb + lane) : 0;
#pragma unroll
            for (int q = 0; q < MAXB; ++q) {
                const int j = __shfl_sync(0xffffffffu, jl, q);
                if (q < nb && active) {
                    const V* xp = reinterpret_cast<const V*>(x + (size_t)j * BC + c0);
#pragma unroll
                    for (int v = 0; v < RV::NV; ++v) xv[q][v] = XL ? __ldg(xp + v) : __ldcg(xp + v);
                }
            }
#pragma unroll
            for (int q = 0; q < MAXB; ++q)
                if (q < nb && active) {
#pragma unroll
                    for (int v = 0; v < RV::NV; ++v) vfma(acc, av[q][v], xv[q][v]);
                }
        } else {
            T av[MAXB][L::CH], xv[MAXB][L::CH];
#pragma unroll
            for (int q = 0; q < MAXB; ++q)
                if (q < nb && active) {
                    const int bq = blk ? __ldg(blk + kb + q) : kb + q;
                    const T* ap = val + (size_t)bq * (BR * BC) + r * BC + c0;
#pragma unroll
                    for (int c = 0; c < L::CH; ++c) av[q][c] = (c0 + c < BC) ? __ldg(ap + c) : T(0);
                }
            const int jl = (lane < nb) ? __ldg(col_idx + kb + lane) : 0;
#pragma unroll
            for (int q = 0; q < MAXB; ++q) {
                const int j = __shfl_sync(0xffffffffu, jl, q);
                if (q < nb && active) {
                    const T* xp = x + (size_t)j * BC + c0;
#pragma unroll
                    for (int c = 0; c < L::CH; ++c)
                        xv[q][c] = (c0 + c < BC) ? (XL ? __ldg(xp + c) : __ldcg(xp + c)) : T(0);
                }
            }
#pragma unroll
            for (int q = 0; q < MAXB; ++q)
                if (q < nb && active) {
#pragma unroll
                    for (int c = 0; c < L::CH; ++c) acc = fma(av[q][c], xv[q][c], acc);
                }
        }
    }
    return acc;
}

// One block at a time with 128-bit loads: the lean form for FP64, whose
// block products are bound by GB300's FP64 pipes rather than by HBM, so
// registers are better spent on occupancy than on loads in flight.
template <class T, int BR, int BC>
__device__ __forceinline__ T row_dot_lean(const int* __restrict__ col_idx, const T* __restrict__ val,
                                          const int* __restrict__ blk, const T* x, int k0, int k1, int r, int c0,
                                          bool active) {
    using L = WL<BR, BC>;
    using RV = RowVec<T, BR, BC>;
    T acc = 0;
#pragma unroll 2
    for (int k = k0; k < k1; ++k) {
        const int j = __ldg(col_idx + k);
        const T* a = val + (size_t)(blk ? __ldg(blk + k) : k) * (BR * BC) + r * BC + c0;
        const T* xj = x + (size_t)j * BC + c0;
        if (!active) continue;
        if constexpr (RV::ok) {
            typedef typename V16<T>::type V;
#pragma unroll
            for (int v = 0; v < RV::NV; ++v) vfma(acc, __ldg(reinterpret_cast<const V*>(a) + v), __ldg(reinterpret_cast<const V*>(xj) + v));
        } else {
#pragma unroll
            for (int c = 0; c < L::CH; ++c)
                if (c0 + c < BC) acc = fma(__ldg(a + c), __ldg(xj + c), acc);
        }
    }
    return acc;
}

// (A x)_i partial for this lane: prefetching form for FP32 (HBM-bound, five
// blocks -- a full 5-point block row -- in flight), lean form for FP64
template <class T, int BR, int BC>
__device__ __forceinline__ T row_product(const int* __restrict__ col_idx, const T* __restrict__ val,
                                         const int* __restrict__ blk, const T* x, int k0, int k1, int r, int c0,
                                         bool active, int lane) {
    if constexpr (sizeof(T) == 4) return row_dot<T, BR, BC, 5>(col_idx, val, blk, x, k0, k1, r, c0, active, lane);
    else return row_dot_lean<T, BR, BC>(col_idx, val, blk, x, k0, k1, r, c0, active);
}

// ---------------------------------------------------------- small blocks --
// Blocks of BR x BC with max(BR, BC) <= 32 (used for square 3..10): lane
// groups of S = max(BR, BC) lanes, 32 / S block rows per warp, lane (g, c) owning
// column c (< BC) of the warp's g-th block row.  For every block the lane
// reads column c of each block row r -- a[r][c], the group's lanes together
// one contiguous BC-value row per load -- and its single entry x_j[c], and
// keeps BR partial sums acc[r].  The warp's block rows are consecutive, so
// their blocks are one contiguous run of the value array.  rows_reduce then
// sums acc[r] over the group's lanes through shared memory, in column
// order, and leaves row r's total on lane (g, r) (r < BR).
template <int BR, int BC = BR>
struct Rows {
    static constexpr int S = BR > BC ? BR : BC;   // lanes per block row
    static constexpr int G = 32 / S;              // block rows per warp
    static constexpr int LD = BC + 1;             // padded shared-memory row
    static constexpr int SM = G * BR * LD;        // values per warp
};

// value readers: T from the stored type (FP64, FP32 or block-scaled FP16)
__device__ __forceinline__ double ld_val(const double* p) { return __ldg(p); }
__device__ __forceinline__ float ld_val(const float* p) { return __ldg(p); }
__device__ __forceinline__ float ld_val(const __half* p) { return __half2float(__ldg(p)); }

// scl: per-block scales of a block-scaled FP16 matrix (null otherwise); a
// block's scale is folded into the lane's x entry
template <class T, class VT, int BR, int BC, int MAXB>
__device__ __forceinline__ void cols_accumulate(const int* __restrict__ col_idx, const VT* __restrict__ val,
                                                const float* __restrict__ scl, const int* __restrict__ blk,
                                                const T* __restrict__ x, int k0, int k1, int c, T (&acc)[BR]) {
    for (int kb = k0; kb < k1; kb += MAXB) {
        const int nb = min(MAXB, k1 - kb);
        T a[MAXB][BR], xv[MAXB], sc[MAXB];
        int j[MAXB];
#pragma unroll
        for (int q = 0; q < MAXB; ++q) j[q] = (q < nb) ? __ldg(col_idx + kb + q) : 0;
#pragma unroll
        for (int q = 0; q < MAXB; ++q)
            if (q < nb) {
                const int bq = blk ? __ldg(blk + kb + q) : kb + q;
                const VT* ap = val + (size_t)bq * (BR * BC) + c;
#pragma unroll
                for (int r = 0; r < BR; ++r) a[q][r] = ld_val(ap + r * BC);
                sc[q] = scl ? (T)__ldg(scl + bq) : T(1);
            }
#pragma unroll
        for (int q = 0; q < MAXB; ++q) xv[q] = (q < nb) ? __ldg(x + (size_t)j[q] * BC + c) * sc[q] : T(0);
#pragma unroll
        for (int q = 0; q < MAXB; ++q)
            if (q < nb) {
#pragma unroll
                for (int r = 0; r < BR; ++r) acc[r] = fma(a[q][r], xv[q], acc[r]);
            }
    }
}

// Sum of acc[r] over the group's lanes c < BC, returned on lane (g, r) for
// r < BR (0 elsewhere); `s` is the warp's Rows<BR, BC>::SM values of shared
// memory.  All lanes must call it.
template <class T, int BR, int BC>
__device__ __forceinline__ T rows_reduce(const T (&acc)[BR], T* s, int g, int c, bool in_group) {
    using R = Rows<BR, BC>;
    if (in_group && c < BC) {
#pragma unroll
        for (int r = 0; r < BR; ++r) s[(g * BR + r) * R::LD + c] = acc[r];
    }
    __syncwarp();
    T y = 0;
    if (in_group && c < BR) {
#pragma unroll
        for (int cc = 0; cc < BC; ++cc) y += s[(g * BR + c) * R::LD + cc];
    }
    __syncwarp();
    return y;
}

}  // namespace mg
