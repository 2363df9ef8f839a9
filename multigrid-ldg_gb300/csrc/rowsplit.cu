// rowsplit.cu -- products and Jacobi sweeps of levels with few, long block
// rows (agglomerated levels: 9 x 9 blocks on triangles, 27 x 27 on
// tetrahedra, 9 to 18 blocks per row).
//
// Lanes as in the small-block kernels (a group of B lanes, lane c owning
// block column c, so every block row is one coalesced load and each lane
// keeps B partial sums), but the blocks of one row are dealt to SPL groups of
// the CTA, whose partial rows are added through shared memory in a fixed
// order.  Without the split a level of 2,000 rows has four warps per SM, each
// reading its row's blocks one after another.
//
// The sweep's inverse diagonal block is dealt out the same way: group p
// applies rows p * RCH .. of it, loaded before the product so that their
// latency hides behind it.
#include <algorithm>
#include <type_traits>

#include "api.cuh"
#include "rowdot.cuh"
#include "rowsplit.cuh"

using namespace mg;

namespace mg {

namespace {

template <class T>
struct SplitArgs {
    int n;
    const int *row_ptr, *col_idx;
    const T *val, *Dinv, *x, *b;
    T* y;
    T alpha, beta, omega;
    int xzero;
};

// warps per CTA (static shared memory stays below 48 KB)
template <class T, int B>
constexpr int split_warps() {
    return sizeof(T) == 8 && B > 16 ? 4 : 8;
}

// JACOBI: y = x + omega Dinv (b - A x); else y = alpha A x + beta b (b may be y)
template <class T, int B, int SPL, int MAXB, bool JACOBI>
__global__ void __launch_bounds__(split_warps<T, B>() * 32) k_rows_split(const SplitArgs<T> a) {
    using R = Rows<B>;
    constexpr int NW = split_warps<T, B>(), G = R::G, NG = NW * G, RPC = NG / SPL;   // groups, rows per CTA
    constexpr int RCH = (B + SPL - 1) / SPL;
    static_assert(NG % SPL == 0, "whole rows per CTA");
    __shared__ T red[NW * R::SM];
    __shared__ T part[NG][B];
    __shared__ T ts[RPC][B];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / B, c = lane - g * B;
    const bool in = g < G;
    const int gid = warp * G + (in ? g : 0), rl = gid / SPL, p = gid - rl * SPL;
    T* s = red + warp * R::SM;
    for (int base = blockIdx.x * RPC; base < a.n; base += gridDim.x * RPC) {
        const int row = base + rl;
        const bool valid = in && row < a.n;
        const size_t o = (size_t)row * B + c;
        T dv[RCH];
        if (JACOBI) {
#pragma unroll
            for (int q = 0; q < RCH; ++q)
                dv[q] = (valid && p * RCH + q < B) ? __ldg(a.Dinv + ((size_t)row * B + p * RCH + q) * B + c) : T(0);
        }
        T bi = 0;
        if (valid && p == 0 && (JACOBI || a.beta != T(0))) bi = a.b[o];
        T acc[B];
#pragma unroll
        for (int r = 0; r < B; ++r) acc[r] = T(0);
        if (valid && !(JACOBI && a.xzero)) {
            const int k1 = __ldg(a.row_ptr + row + 1);
            for (int kb = __ldg(a.row_ptr + row) + p; kb < k1; kb += SPL * MAXB) {
                T av[MAXB][B], xv[MAXB];
                int j[MAXB];
#pragma unroll
                for (int q = 0; q < MAXB; ++q) j[q] = kb + q * SPL < k1 ? __ldg(a.col_idx + kb + q * SPL) : -1;
#pragma unroll
                for (int q = 0; q < MAXB; ++q)
                    if (j[q] >= 0) {
                        const T* ap = a.val + (size_t)(kb + q * SPL) * (B * B) + c;
#pragma unroll
                        for (int r = 0; r < B; ++r) av[q][r] = __ldg(ap + r * B);
                        xv[q] = __ldg(a.x + (size_t)j[q] * B + c);
                    }
#pragma unroll
                for (int q = 0; q < MAXB; ++q)
                    if (j[q] >= 0) {
#pragma unroll
                        for (int r = 0; r < B; ++r) acc[r] = fma(av[q][r], xv[q], acc[r]);
                    }
            }
        }
        T sum = rows_reduce<T, B, B>(acc, s, g, c, in);
        if (in) part[gid][c] = sum;
        __syncthreads();
        if (p == 0 && in) {
#pragma unroll
            for (int q = 1; q < SPL; ++q) sum += part[gid + q][c];
            if (JACOBI) ts[rl][c] = bi - sum;
            else if (valid) {
                T v = a.alpha * sum;
                if (a.beta != T(0)) v += a.beta * bi;
                a.y[o] = v;
            }
        }
        if (JACOBI) {
            __syncthreads();
            const T t = in ? ts[rl][c] : T(0);
            // products d[q][c] t[c] of the group's rows, each summed by one lane
            if (in) {
#pragma unroll
                for (int q = 0; q < RCH; ++q) s[(g * B + q) * R::LD + c] = dv[q] * t;
            }
            __syncwarp();
            if (valid && c < RCH && p * RCH + c < B) {
                T y = 0;
#pragma unroll
                for (int cc = 0; cc < B; ++cc) y += s[(g * B + c) * R::LD + cc];
                const size_t oo = (size_t)row * B + p * RCH + c;
                const T xi = a.xzero ? T(0) : __ldg(a.x + oo);
                a.y[oo] = xi + a.omega * y;
            }
            __syncwarp();
        } else {
            __syncthreads();   // part is rewritten by the next rows
        }
    }
}

template <class T, int B, int SPL, int MAXB, bool JACOBI>
void launch_split(mgldg_ctx* ctx, const SplitArgs<T>& a, int kclass) {
    constexpr int NW = split_warps<T, B>(), RPC = NW * Rows<B>::G / SPL;
    const int grid = std::max(1, std::min((a.n + RPC - 1) / RPC, ctx->sm_count * 16));
    {
        Launch L(ctx, kclass);
        k_rows_split<T, B, SPL, MAXB, JACOBI><<<grid, NW * 32, 0, ctx->stream>>>(a);
    }
    check_launch();
}

// Where the split pays (event times of a Jacobi sweep, us).  27 x 27
// (agglomerated tetrahedra) and 25 x 25 (Q4), FP32: the general kernel gives
// each lane a block row (strided loads, 1.1 TB/s).  General / 1 / 2 / 4 / 8
// groups per row on a 5-level ball: 5,143 rows (11.7 blocks each) 161 / 39.8 /
// 32.8 / 34.3 / 40.4, 605 rows (14.2) 60.4 / 14.5 / 10.8 / 9.3 / 10.9; 25 x 25,
// 20,000 rows of 5.5 blocks 270 / - / 65.5, 300 rows 24.6 / - / - / 6.5.
//
// FP64 is bound by its pipes, which the row sums of this form load further: it
// pays while the SMs are nearly empty, and the longer for longer rows.  One
// V-cycle of eight sweeps, general / 4 groups, 27 x 27: 1 block per row 150 rows
// 79 / 79, 200 rows 79 / 95, 2,000 rows 128 / 349; 4 blocks 300 rows 129 / 96,
// 450 rows 128 / 127, 800 rows 129 / 226; 9 blocks 600 rows 210 / 183, 800 rows
// 210 / 303; 16 blocks 600 rows 302 / 227, 800 rows 309 / 349.  25 x 25 has the
// same lines (4 blocks 450 rows 128 / 116, 600 rows 128 / 144).
//
// 9 x 9 (agglomerated triangles), general / 1 / 3 / 6 / 12 groups: FP32 8,859
// rows (13.1) 13.7 / 13.9 / 15.2 / 16.5 / 19.5, 1,995 rows (16.5) 10.9 / 12.3 /
// 8.8 / 8.7 / 9.6; FP64 1,995 rows 21.0 / 16.7 (3), 4,000 rows 34.9 / 26.9 (3).
// In FP64 the split has the time of two CTAs (16 rows) on an SM up to 16 rows
// per SM, the general kernel that of one CTA (24 rows) up to 24: eight sweeps of
// rows of 13 blocks 2,000 rows 144 / 128, 3,000 rows 145 / 161, 4,000 rows 225 /
// 196.  Uniform grids have five blocks per row, too few to deal out.
template <class T, bool JACOBI>
bool split_dispatch(mgldg_ctx* ctx, const mgldg_bsr* A, SplitArgs<T>& a, int kclass) {
    if (A->br != A->bc || A->blk || A->nbr == 0) return false;
    constexpr bool f64 = sizeof(T) == 8;
    a.n = A->nbr;
    a.row_ptr = A->row_ptr;
    a.col_idx = A->col_idx;
    const int64_t n = A->nbr, nnzb = A->nnzb;
    if (A->br == 27 || A->br == 25) {
        if constexpr (f64) {
            if (!(n <= 150 || (n < 400 && nnzb >= 3 * n) || (n < 640 && nnzb >= 8 * n))) return false;
        } else if (n >= 2048) {
            if (A->br == 27) launch_split<T, 27, 2, 1, JACOBI>(ctx, a, kclass);
            else launch_split<T, 25, 2, 1, JACOBI>(ctx, a, kclass);
            return true;
        }
        if (A->br == 27) launch_split<T, 27, 4, 1, JACOBI>(ctx, a, kclass);
        else launch_split<T, 25, 4, 1, JACOBI>(ctx, a, kclass);
        return true;
    }
    if (A->br == 9 && n < 4096 && nnzb >= 8 * n && (!f64 || n <= 16 * ctx->sm_count || n > 24 * ctx->sm_count)) {
        launch_split<T, 9, 3, 2, JACOBI>(ctx, a, kclass);
        return true;
    }
    return false;
}

}  // namespace

template <class T>
bool split_spmv(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, T alpha, const T* x, T beta, const T* yin, T* y,
                int kclass) {
    SplitArgs<T> a{};
    a.val = vals;
    a.x = x;
    a.b = yin;
    a.y = y;
    a.alpha = alpha;
    a.beta = beta;
    return split_dispatch<T, false>(ctx, A, a, kclass);
}
template bool split_spmv<float>(mgldg_ctx*, const mgldg_bsr*, const float*, float, const float*, float, const float*,
                                float*, int);
template bool split_spmv<double>(mgldg_ctx*, const mgldg_bsr*, const double*, double, const double*, double,
                                 const double*, double*, int);

template <class T>
bool split_jacobi(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b, const T* xin, T* xout,
                  T omega, bool xzero) {
    SplitArgs<T> a{};
    a.val = vals;
    a.Dinv = Dinv;
    a.x = xin;
    a.b = b;
    a.y = xout;
    a.omega = omega;
    a.xzero = xzero ? 1 : 0;
    return split_dispatch<T, true>(ctx, A, a, MGLDG_K_JACOBI);
}
template bool split_jacobi<float>(mgldg_ctx*, const mgldg_bsr*, const float*, const float*, const float*, const float*,
                                  float*, float, bool);
template bool split_jacobi<double>(mgldg_ctx*, const mgldg_bsr*, const double*, const double*, const double*,
                                   const double*, double*, double, bool);

}  // namespace mg
