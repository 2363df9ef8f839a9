// spmm_rep.cu -- multi-vector products of level operators with few distinct
// blocks (repeat.cuh).
//
// For the products bound by arithmetic: FP64 (its pipes) and the double-float
// outer product (11 FP32 operations per product).  Block columns that are
// zero are skipped with their part of X -- half of the products on quadtree
// operators -- and the distinct blocks are read from L1.  A warp takes E rows
// of one class, so a block value is read once for E rows and 32 V columns.
// The sums run in the general kernels' order.  44,197 rows of 9 x 9: FP64 sweep
// with 24 columns 954 -> 764 us, double-float product with 64 columns 706 ->
// 566 us (rows in pairs, packed operations).  FP32 products are bound by their
// vectors and keep the general kernel (batched.cu level_spmm).
#include <algorithm>
#include <type_traits>

#include "api.cuh"
#include "repeat.cuh"
#include "rowdot.cuh"

using namespace mg;

namespace mg {

namespace {

template <class T>
struct MMArgs {
    int ngroups, nslots, nuniq, gu, k;
    const int *gcls, *rows, *cols, *cls;
    const T *c, *img;     // blocks by columns; the image (for the inverse diagonal blocks, by rows)
    const T *X, *Yin, *B;
    T* Y;
    T alpha, beta, omega;
    int xzero;
};

template <int V>
__device__ __forceinline__ void ldv(const float* p, float (&v)[V]) {
    if constexpr (V == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = p[0];
    }
}
template <int V>
__device__ __forceinline__ void ldv(const double* p, double (&v)[V]) {
    if constexpr (V == 2) {
        const double2 t = *reinterpret_cast<const double2*>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = p[0];
    }
}
template <int V>
__device__ __forceinline__ void stv(double* p, const double (&v)[V]) {
    if constexpr (V == 2) *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    else p[0] = v[0];
}
// one table line (B values and padding)
template <int LD>
__device__ __forceinline__ void line(const float* p, float (&v)[LD]) {
#pragma unroll
    for (int q = 0; q < LD / 4; ++q) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p) + q);
        v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
}
template <int LD>
__device__ __forceinline__ void line(const double* p, double (&v)[LD]) {
#pragma unroll
    for (int q = 0; q < LD / 2; ++q) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p) + q);
        v[2 * q] = t.x; v[2 * q + 1] = t.y;
    }
}
template <class T, int B>
struct MMImg {
    static constexpr int LD = (B + 3) / 4 * 4;
    static constexpr int PAD = B == 16 ? 16 / (int)sizeof(T) : 0;   // as in repeat.cu
    static constexpr int SIZE = B * LD + PAD;
    static __device__ constexpr int at(int l) { return l * LD + (B == 16 && l >= 8 ? PAD : 0); }
};

// a warp: E rows of one class, 32 V columns
template <class T, int B, int V, int E, bool JACOBI>
__global__ void __launch_bounds__(128) k_spmm_rep(const MMArgs<T> a) {
    using I = MMImg<T, B>;
    constexpr int LD = I::LD, CB = B == 9 ? 3 : 4;   // columns whose parts of X are in flight together
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.y * 32 + lane) * V, k = a.k;
    const bool cok = c < k;
    for (int g = blockIdx.x * 4 + (threadIdx.x >> 5); g < a.ngroups; g += gridDim.x * 4) {
        const int slot = g * E;
        int row[E];
#pragma unroll
        for (int e = 0; e < E; ++e) row[e] = __ldg(a.rows + slot + e);
        if (row[0] < 0) continue;   // a class's rows come before its padding
        const int* cls = a.cls + (size_t)__ldg(a.gcls + slot / a.gu) * kRepCls;
        T acc[E][B][V];
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
            for (int r = 0; r < B; ++r)
#pragma unroll
                for (int v = 0; v < V; ++v) acc[e][r][v] = T(0);
        if (cok && !(JACOBI && a.xzero)) {
            const int nb = __ldg(cls);
#pragma unroll 1
            for (int q = 0; q < nb; ++q) {
                const int id = __ldg(cls + 4 + q);
                const unsigned cm = (unsigned)__ldg(cls + 4 + kRepMaxNb + q) >> 16;
                const T* tab = a.c + (size_t)id * (B * LD);
                const T* xp[E];
#pragma unroll
                for (int e = 0; e < E; ++e)
                    xp[e] = a.X + (size_t)__ldg(a.cols + (size_t)q * a.nslots + slot + e) * B * k + c;
#pragma unroll
                for (int cb = 0; cb < B; cb += CB) {
                    if (!((cm >> cb) & ((1u << CB) - 1u))) continue;
                    T xv[CB][E][V];
#pragma unroll
                    for (int d = 0; d < CB; ++d)
                        if ((cm >> (cb + d)) & 1u) {
#pragma unroll
                            for (int e = 0; e < E; ++e) ldv<V>(xp[e] + (size_t)(cb + d) * k, xv[d][e]);
                        }
#pragma unroll
                    for (int d = 0; d < CB; ++d)
                        if ((cm >> (cb + d)) & 1u) {
                            T av[LD];
                            line<LD>(tab + (cb + d) * LD, av);
#pragma unroll
                            for (int e = 0; e < E; ++e)
#pragma unroll
                                for (int r = 0; r < B; ++r)
#pragma unroll
                                    for (int v = 0; v < V; ++v) acc[e][r][v] = fma(av[r], xv[d][e][v], acc[e][r][v]);
                        }
                }
            }
        }
        if (!cok) continue;
        if constexpr (JACOBI) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const T* bp = a.B + (size_t)max(row[e], 0) * B * k + c;
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    T bv[V];
                    ldv<V>(bp + (size_t)r * k, bv);
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[e][r][v] = bv[v] - acc[e][r][v];
                }
            }
            const T* D = a.img + (size_t)(a.nuniq + __ldg(cls + 1)) * I::SIZE;
#pragma unroll
            for (int r = 0; r < B; ++r) {
                T dv[LD];
                line<LD>(D + I::at(r), dv);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if (row[e] < 0) continue;
                    const size_t o = ((size_t)row[e] * B + r) * k + c;
                    T y[V], xv[V];
                    if (a.xzero) {
#pragma unroll
                        for (int v = 0; v < V; ++v) xv[v] = T(0);
                    } else {
                        ldv<V>(a.X + o, xv);
                    }
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        y[v] = T(0);
#pragma unroll
                        for (int cc = 0; cc < B; ++cc) y[v] = fma(dv[cc], acc[e][cc][v], y[v]);
                        xv[v] = xv[v] + a.omega * y[v];
                    }
                    stv<V>(a.Y + o, xv);
                }
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                if (row[e] < 0) continue;
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    const size_t o = ((size_t)row[e] * B + r) * k + c;
                    T out[V];
                    if (a.beta != T(0)) {
                        T yv[V];
                        ldv<V>(a.Yin + o, yv);
#pragma unroll
                        for (int v = 0; v < V; ++v) out[v] = a.alpha * acc[e][r][v] + a.beta * yv[v];
                    } else {
#pragma unroll
                        for (int v = 0; v < V; ++v) out[v] = a.alpha * acc[e][r][v];
                    }
                    stv<V>(a.Y + o, out);
                }
            }
        }
    }
}

// Q = A D in double-float arithmetic: one row per warp, 32 V columns; the
// rows of a block column are taken in pairs (packed FP32 operations), which
// halves the instructions of the compute-bound product
template <int B, int V>
__global__ void __launch_bounds__(128) k_spmm_rep_df64(MMArgs<float> a, const float* __restrict__ clo,
                                                       const float* __restrict__ Dlo, double* __restrict__ Q) {
    constexpr int LD = (B + 3) / 4 * 4, NP = (B + 1) / 2, CB = B == 9 ? 3 : 4;
    typedef unsigned long long u64;
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.y * 32 + lane) * V, k = a.k;
    if (c >= k) return;
    for (int slot = blockIdx.x * 4 + (threadIdx.x >> 5); slot < a.ngroups; slot += gridDim.x * 4) {
        const int row = __ldg(a.rows + slot);
        if (row < 0) continue;
        const int* cls = a.cls + (size_t)__ldg(a.gcls + slot / a.gu) * kRepCls;
        u64 sh[NP][V], sl[NP][V];
#pragma unroll
        for (int r = 0; r < NP; ++r)
#pragma unroll
            for (int v = 0; v < V; ++v) sh[r][v] = sl[r][v] = 0ULL;
        const int nb = __ldg(cls);
#pragma unroll 1
        for (int q = 0; q < nb; ++q) {
            const int id = __ldg(cls + 4 + q);
            const unsigned cm = (unsigned)__ldg(cls + 4 + kRepMaxNb + q) >> 16;
            const size_t xo = (size_t)__ldg(a.cols + (size_t)q * a.nslots + slot) * B * k + c;
#pragma unroll
            for (int cb = 0; cb < B; cb += CB) {
                if (!((cm >> cb) & ((1u << CB) - 1u))) continue;
                float xh[CB][V], xl[CB][V];
#pragma unroll
                for (int d = 0; d < CB; ++d)
                    if ((cm >> (cb + d)) & 1u) {
                        ldv<V>(a.X + xo + (size_t)(cb + d) * k, xh[d]);
                        ldv<V>(Dlo + xo + (size_t)(cb + d) * k, xl[d]);
                    }
#pragma unroll
                for (int d = 0; d < CB; ++d)
                    if ((cm >> (cb + d)) & 1u) {
                        const size_t to = (size_t)id * (B * LD) + (cb + d) * LD;
                        float ah[LD], al[LD];
                        line<LD>(a.c + to, ah);
                        line<LD>(clo + to, al);
#pragma unroll
                        for (int r = 0; r < NP; ++r) {
                            const u64 a2 = pack2(ah[2 * r], ah[2 * r + 1]), b2 = pack2(al[2 * r], al[2 * r + 1]);
#pragma unroll
                            for (int v = 0; v < V; ++v)
                                df_fma2(sh[r][v], sl[r][v], a2, b2, pack2(xh[d][v], xh[d][v]),
                                        pack2(-xh[d][v], -xh[d][v]), pack2(xl[d][v], xl[d][v]));
                        }
                    }
            }
        }
        double* qp = Q + (size_t)row * B * k + c;
#pragma unroll
        for (int r = 0; r < B; ++r) {
            double out[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const float2 h = unpack2(sh[r / 2][v]), l = unpack2(sl[r / 2][v]);
                out[v] = (r & 1) ? widen(h.y) + widen(l.y) : widen(h.x) + widen(l.x);
            }
            stv<V>(qp + (size_t)r * k, out);
        }
    }
}

bool aligned_to(const void* p, size_t a) { return (uintptr_t)p % a == 0; }

template <class T>
MMArgs<T> mm_args(const RepTable* t, int k) {
    MMArgs<T> a{};
    a.nslots = t->nslots;
    a.nuniq = t->nuniq;
    a.gu = t->gu;
    a.k = k;
    a.gcls = t->gcls;
    a.rows = t->rows;
    a.cols = t->cols;
    a.cls = t->cls;
    if constexpr (std::is_same<T, float>::value) {
        a.c = t->c32;
        a.img = t->i32;
    } else {
        a.c = t->c64;
        a.img = t->i64;
    }
    return a;
}

template <class T, int B, int V, int E>
void mm_launch(mgldg_ctx* ctx, MMArgs<T>& a, bool jacobi, int kclass) {
    a.ngroups = a.nslots / E;
    const dim3 grid(std::max(1, std::min((a.ngroups + 3) / 4, ctx->sm_count * 32)), (a.k + 32 * V - 1) / (32 * V));
    {
        Launch L(ctx, kclass);
        if (jacobi) k_spmm_rep<T, B, V, E, true><<<grid, 128, 0, ctx->stream>>>(a);
        else k_spmm_rep<T, B, V, E, false><<<grid, 128, 0, ctx->stream>>>(a);
    }
    check_launch();
}

template <int B>
void mm_dispatch(mgldg_ctx* ctx, MMArgs<double>& a, bool two, bool jacobi, int kclass) {
    // accumulators: 36 at most per lane
    if (two) mm_launch<double, B, 2, (B == 16 ? 1 : 2)>(ctx, a, jacobi, kclass);
    else mm_launch<double, B, 1, 2>(ctx, a, jacobi, kclass);
}

}  // namespace

// Where the tables pay (us per sweep, general / table).  FP64 4 x 4 blocks have
// little to skip, and a warp's rows lose their locality: 49,645 quadtree rows
// 229 / 238 with 1 column, 456 / 473 with 64; 4,096 of a uniform grid 26 / 28, 45
// / 53.  9 x 9: 4,096 uniform rows (17 distinct blocks) 95 / 88, 185 / 174, 3,709
// rows of a quadtree's third coarse level 98 / 89, 176 / 176, but levels with few rows
// per distinct block 2,230 64 / 74, 111 / 141; 4,096 with 744 blocks 97 / 104, 185 /
// 203.  16 x 16: 2,230 rows 184 / 203 up to 32 columns, 336 / 306 with 33; 4,096
// uniform rows 286 / 258.
bool rep_mm_pays(int b, int64_t rows, int64_t nuniq) {
    return b == 16 || (b == 9 && rows >= 10 * nuniq);
}
// double-float products: 4 x 4 4,096 rows 21 / 23, 10,036 38 / 40, 16,384 even,
// 25,597 and more faster; the others from kRepMmRows on
bool rep_mm_df64_pays(int b, int64_t rows) { return b != 4 || rows >= 20000; }

bool rep_spmm(mgldg_ctx* ctx, const mgldg_bsr* A, const RepMM& m, int kclass) {
    const RepTable* t = A->rep;
    if (!t || t->nbr < kRepMmRows || !rep_mm_pays(t->b, t->nbr, t->nuniq)) return false;
    if (t->b == 16 && m.k <= 32 && t->nbr < 3072) return false;
    MMArgs<double> a = mm_args<double>(t, m.k);
    a.X = m.X;
    a.Yin = m.Yin;
    a.B = m.B;
    a.Y = m.Y;
    a.alpha = m.alpha;
    a.beta = m.beta;
    a.omega = m.omega;
    a.xzero = m.xzero;
    const size_t al = 2 * sizeof(double);
    const bool two = m.k % 2 == 0 && m.k > 32 && aligned_to(m.X, al) && aligned_to(m.Yin, al) && aligned_to(m.B, al) &&
                     aligned_to(m.Y, al);
    if (t->b == 9) mm_dispatch<9>(ctx, a, two, m.jacobi != 0, kclass);
    else mm_dispatch<16>(ctx, a, two, m.jacobi != 0, kclass);
    return true;
}

bool rep_spmm_df64(mgldg_ctx* ctx, const mgldg_bsr* A, int k, const float* Dhi, const float* Dlo, double* Q) {
    const RepTable* t = A->rep;
    if (!t || t->nbr < kRepMmRows || !rep_mm_df64_pays(t->b, t->nbr)) return false;
    MMArgs<float> a = mm_args<float>(t, k);
    a.X = Dhi;
    a.ngroups = t->nslots;
    const bool two = k % 2 == 0 && k > 32 && aligned_to(Dhi, 8) && aligned_to(Dlo, 8) && aligned_to(Q, 16);
    const int V = two ? 2 : 1;
    const dim3 grid(std::max(1, std::min((a.ngroups + 3) / 4, ctx->sm_count * 32)), (k + 32 * V - 1) / (32 * V));
    {
        Launch L(ctx, MGLDG_K_SPMV);
        switch (t->b * 10 + V) {
            case 41: k_spmm_rep_df64<4, 1><<<grid, 128, 0, ctx->stream>>>(a, t->clo, Dlo, Q); break;
            case 42: k_spmm_rep_df64<4, 2><<<grid, 128, 0, ctx->stream>>>(a, t->clo, Dlo, Q); break;
            case 91: k_spmm_rep_df64<9, 1><<<grid, 128, 0, ctx->stream>>>(a, t->clo, Dlo, Q); break;
            case 92: k_spmm_rep_df64<9, 2><<<grid, 128, 0, ctx->stream>>>(a, t->clo, Dlo, Q); break;
            case 161: k_spmm_rep_df64<16, 1><<<grid, 128, 0, ctx->stream>>>(a, t->clo, Dlo, Q); break;
            default: k_spmm_rep_df64<16, 2><<<grid, 128, 0, ctx->stream>>>(a, t->clo, Dlo, Q); break;
        }
    }
    check_launch();
    return true;
}

}  // namespace mg
