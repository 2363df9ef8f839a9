// repeat.cu -- level operators with few distinct blocks.
//
// On grids with constant coefficients the LDG operator and every Galerkin
// coarse operator consist of a handful of distinct blocks (17 on every level
// of a uniform grid, tens to hundreds on an adaptive quadtree), and most
// off-diagonal blocks have only P nonzero rows or columns of P^2.  The general
// kernels read all blocks from HBM (1.3 GB per FP32 product of 512 x 512 Q3)
// and are bound by it, or by the FP64 pipes; here the distinct blocks sit in
// shared memory, a product moves its vectors and indices only, and all-zero
// block rows (or columns) are skipped.  Level 0 of 512 x 512 Q3, event times
// before and after: FP32 sweeps (three full, one from x = 0) 213 -> 36 us on
// average, FP32 residual 240 -> 34 us, double-float product 410 -> 110 us;
// 256 x 256 Q3 FP64 sweeps 174 -> 105 us, residual 185 -> 90 us.  What is
// left: vector traffic and shared-memory reads (FP32), the FP64 pipes (FP64
// and the conversions of the double-float product).
//
// Mapping: the rows are sorted by class (same sequence of table entries) and
// a warp's rows belong to one class, so a block value read once from shared
// memory serves all of them.  16 x 16 blocks: two lanes per row, one per
// column half, E = 1 or 2 rows per lane pair; smaller blocks: one lane per
// row.  The sums run in the general kernels' order (16 x 16: the two column
// halves in block order, then their sum; smaller blocks: one sum per column
// over the blocks, then the columns), and a skipped product is one with a
// zero block entry, so for finite vectors the results are the general
// kernels' values.
#include <algorithm>
#include <memory>
#include <type_traits>

#include "api.cuh"
#include "repeat.cuh"
#include "rowdot.cuh"

using namespace mg;

namespace mg {

RepTable::~RepTable() {
    if (pool) cudaFree(pool);
    if (slots) cudaFree(slots);
}

// -------------------------------------------------------------- detection --
namespace {
constexpr int kMaxUniq = 2048;    // most distinct blocks kept
constexpr int kMaxCls = 4096;     // most row classes kept
constexpr int kHash = 8192;       // hash slots
constexpr int kSample = 2560;     // blocks of the sample, more than kMaxUniq
constexpr int kSampleKeys = 4096;
struct HashSlot {
    unsigned long long key;       // hash of a block (a row), 0: empty
    int first;                    // smallest block (row) index with this hash
    int id;                       // table entry (class), second step
};
}  // namespace

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    // finaliser of the SplitMix64 generator (Steele, Lea, Flood 2014)
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

// hash of one block's values by a warp, with -0 taken as +0 (valid in every
// lane, never 0)
__device__ __forceinline__ unsigned long long block_hash(const double* __restrict__ a, int bsz, int lane) {
    unsigned long long h = 0;
    for (int e = lane; e < bsz; e += 32) {
        const unsigned long long bits = (unsigned long long)__double_as_longlong(__ldg(a + e) + 0.0);
        h += mix64(bits + 0x9e3779b97f4a7c15ULL * (unsigned long long)(e + 1));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
    return h ? h : 1ULL;
}

// Number of distinct blocks among m evenly spaced ones, one warp each: more
// than kMaxUniq of them rule a table out.  Most operators without repeated
// blocks end here, with no allocation and no wait of their own (hashing all of
// them, with the table's memory, took mgldg_mg_create 0.4 ms per large level).
__global__ void __launch_bounds__(256) k_rep_sample(int64_t nnzb, int bsz, const double* __restrict__ val, int m,
                                                    unsigned long long* keys, int* count) {
    const int lane = threadIdx.x & 31, t = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (t >= m) return;
    const int64_t k = (int64_t)t * nnzb / m;
    const unsigned long long h = block_hash(val + k * bsz, bsz, lane);
    if (lane) return;
    int s = (int)(h & (kSampleKeys - 1));
    for (int probe = 0; probe < kSampleKeys; ++probe) {   // m < kSampleKeys: ends
        const unsigned long long cur = atomicCAS(keys + s, 0ULL, h);
        if (cur == 0ULL) atomicAdd(count, 1);
        if (cur == 0ULL || cur == h) return;
        s = (s + 1) & (kSampleKeys - 1);
    }
}

__global__ void k_rep_clear(HashSlot* slots, int* head) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 2 * kHash) slots[t] = HashSlot{0ULL, 0x7fffffff, -1};
    if (t < 4) head[t] = 0;
}

// enters hash h of item k; head: distinct hashes, set once there are more
// than `most`.  The slot, or -1 after that.
__device__ __forceinline__ int hash_enter(HashSlot* slots, int* head, int most, unsigned long long h, int k) {
    int s = (int)(h & (kHash - 1));
    for (int probe = 0; probe < kHash; ++probe) {
        unsigned long long cur = *(volatile unsigned long long*)&slots[s].key;
        if (cur == 0) {
            cur = atomicCAS(&slots[s].key, 0ULL, h);
            if (cur == 0) {
                if (atomicAdd(&head[0], 1) >= most) *(volatile int*)&head[1] = 1;
                cur = h;
            }
        }
        if (cur == h) {
            if (*(volatile int*)&slots[s].first > k) atomicMin(&slots[s].first, k);
            return s;
        }
        if (*(volatile int*)&head[1]) break;
        s = (s + 1) & (kHash - 1);
    }
    return -1;
}

// One warp per block: its hash, entered into the hash table with the smallest
// block index.  Once more than kMaxUniq distinct hashes were met the warps
// stop.
__global__ void __launch_bounds__(256) k_rep_hash(int64_t nnzb, int bsz, const double* __restrict__ val,
                                                  HashSlot* slots, int* head, int* __restrict__ slot_of) {
    const int lane = threadIdx.x & 31;
    for (int64_t k = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); k < nnzb; k += (int64_t)gridDim.x * 8) {
        if (*(volatile int*)&head[1]) return;
        const unsigned long long h = block_hash(val + k * bsz, bsz, lane);
        if (lane == 0) {
            const int s = hash_enter(slots, head, kMaxUniq, h, (int)k);
            if (s >= 0) slot_of[k] = s;
        }
    }
}

// table entry of every block, checked value by value against the entry's
// first block (a hash collision sets head[1] and the table is not used)
__global__ void __launch_bounds__(256) k_rep_assign(int64_t nnzb, int bsz, const double* __restrict__ val,
                                                    const HashSlot* __restrict__ slots, int* head,
                                                    int* slot_of) {
    const int lane = threadIdx.x & 31;
    for (int64_t k = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); k < nnzb; k += (int64_t)gridDim.x * 8) {
        const HashSlot s = slots[slot_of[k]];
        bool same = true;
        for (int e = lane; e < bsz; e += 32)
            same = same && __double_as_longlong(__ldg(val + k * bsz + e) + 0.0) ==
                               __double_as_longlong(__ldg(val + (int64_t)s.first * bsz + e) + 0.0);
        same = __all_sync(0xffffffffu, same);
        if (lane == 0) {
            if (!same) head[1] = 1;
            slot_of[k] = s.id;
        }
    }
}

// Row classes (same sequence of table entries and the diagonal one in the same
// place), the same way: hash of every row, then every row against the class's
// first row.  (Made row by row on the host, the tables of a hierarchy with
// 175,006 quadtree rows of 9 x 9 took mgldg_mg_create 15 ms, now 6.)
__global__ void __launch_bounds__(256) k_rep_row_hash(int n, const int* __restrict__ row_ptr,
                                                      const int* __restrict__ diag, const int* __restrict__ id,
                                                      HashSlot* slots, int* head, int* __restrict__ slot_of) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const int k0 = __ldg(row_ptr + i), nb = __ldg(row_ptr + i + 1) - k0, dk = __ldg(diag + i);
        if (nb < 1 || nb > kRepMaxNb || dk < 0) {
            head[1] = 1;
            return;
        }
        unsigned long long h = mix64((unsigned long long)nb * 64 + (unsigned long long)(dk - k0));
        for (int q = 0; q < nb; ++q) h = mix64(h + 0x9e3779b97f4a7c15ULL * (unsigned long long)(id[k0 + q] + 1));
        const int s = hash_enter(slots, head, kMaxCls, h ? h : 1ULL, i);
        if (s < 0) return;
        slot_of[i] = s;
    }
}

__global__ void __launch_bounds__(256) k_rep_classes(int ncls, const int* __restrict__ first,
                                                     const int* __restrict__ row_ptr, const int* __restrict__ diag,
                                                     const int* __restrict__ id, int* __restrict__ cls) {
    for (int t = blockIdx.x * 256 + threadIdx.x; t < ncls * kRepCls; t += gridDim.x * 256) {
        const int c = t / kRepCls, e = t - c * kRepCls, i = first[c];
        const int k0 = __ldg(row_ptr + i), nb = __ldg(row_ptr + i + 1) - k0;
        int v = 0;
        if (e == 0) v = nb;
        else if (e == 1) v = id[__ldg(diag + i)];
        else if (e == 2) v = __ldg(diag + i) - k0;
        else if (e >= 4 && e < 4 + nb) v = id[k0 + e - 4];
        cls[t] = v;
    }
}

__global__ void __launch_bounds__(256) k_rep_row_assign(int n, const int* __restrict__ row_ptr,
                                                        const int* __restrict__ diag, const int* __restrict__ id,
                                                        const HashSlot* __restrict__ slots, const int* __restrict__ cls,
                                                        int* head, int* slot_of) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const int c = slots[slot_of[i]].id;
        const int k0 = __ldg(row_ptr + i), nb = __ldg(row_ptr + i + 1) - k0;
        const int* d = cls + (size_t)c * kRepCls;
        bool same = d[0] == nb && d[2] == __ldg(diag + i) - k0;
        for (int q = 0; q < nb && same; ++q) same = d[4 + q] == id[k0 + q];
        if (!same) head[1] = 1;
        slot_of[i] = c;
    }
}

// block columns of the slots; padding slots read what their group's first row
// reads
__global__ void __launch_bounds__(256) k_rep_cols(int nslots, int gs, int most, const int* __restrict__ rows,
                                                  const int* __restrict__ row_ptr, const int* __restrict__ col_idx,
                                                  int* __restrict__ cols) {
    for (int s = blockIdx.x * 256 + threadIdx.x; s < nslots; s += gridDim.x * 256) {
        const int r = rows[s], i = r >= 0 ? r : rows[s / gs * gs];
        const int k0 = __ldg(row_ptr + i), nb = __ldg(row_ptr + i + 1) - k0;
        for (int q = 0; q < most; ++q) cols[(size_t)q * nslots + s] = __ldg(col_idx + k0 + min(q, nb - 1));
    }
}

// first value of line l of an image block, and the block's size
template <class T, int B>
struct Img {
    static constexpr int LD = (B + 3) / 4 * 4;
    static constexpr int PAD = B == 16 ? 16 / (int)sizeof(T) : 0;
    static constexpr int SIZE = B * LD + PAD;
    static __host__ __device__ constexpr int line(int l) { return l * LD + (B == 16 && l >= 8 ? PAD : 0); }
};

// images of one table entry per CTA (the diagonal entries also fill their
// inverse block): T = double, float
template <class T, int B>
__device__ void fill_image(T* img, const double* a, bool cols, int part) {
    using I = Img<T, B>;
    for (int e = threadIdx.x; e < B * I::LD; e += blockDim.x) {
        const int l = e / I::LD, q = e % I::LD;
        const double v = q < B ? (cols ? a[q * B + l] : a[l * B + q]) + 0.0 : 0.0;
        img[I::line(l) + q] = part == 0 ? (T)v : (T)(v - (double)(float)v);
    }
}

template <int B>
__global__ void __launch_bounds__(256) k_rep_tables(const double* __restrict__ val, const int* __restrict__ first,
                                                    const int* __restrict__ drow, const int* __restrict__ didx,
                                                    const double* __restrict__ Dinv, RepView t) {
    __shared__ unsigned rm, cm;
    __shared__ unsigned long long mx;
    const int u = blockIdx.x;
    const double* a = val + (size_t)first[u] * (B * B);
    if (threadIdx.x == 0) rm = cm = 0u, mx = 0ULL;
    __syncthreads();
    for (int e = threadIdx.x; e < B * B; e += blockDim.x) {
        const double v = fabs(a[e]);
        if (v != 0.0) {
            atomicOr(&rm, 1u << (e / B));
            atomicOr(&cm, 1u << (e % B));
            atomicMax(&mx, (unsigned long long)__double_as_longlong(v));   // nonnegative doubles order as integers
        }
    }
    __syncthreads();
    // small blocks are always read by columns
    const bool cols = B != 16 || __popc(rm) >= __popc(cm);
    using I8 = Img<double, B>;
    using I4 = Img<float, B>;
    fill_image<double, B>(t.i64 + (size_t)u * I8::SIZE, a, cols, 0);
    fill_image<float, B>(t.i32 + (size_t)u * I4::SIZE, a, cols, 0);
    fill_image<float, B>(t.ilo + (size_t)u * I4::SIZE, a, cols, 1);
    const double s = mx ? __longlong_as_double((long long)mx) : 1.0;
    for (int e = threadIdx.x; e < B * B; e += blockDim.x)
        t.i16[(size_t)u * I4::SIZE + I4::line(e / B) + e % B] = __half2float(__float2half_rn((float)(a[e] / s)));
    if (drow[u] >= 0) {
        const double* D = Dinv + (size_t)drow[u] * (B * B);
        const size_t at = t.nuniq + didx[u];
        fill_image<double, B>(t.i64 + at * I8::SIZE, D, false, 0);
        fill_image<float, B>(t.i32 + at * I4::SIZE, D, false, 0);
        fill_image<float, B>(t.i16 + at * I4::SIZE, D, false, 0);
    }
    if constexpr (B == 16) {
        for (int e = threadIdx.x; e < 256; e += blockDim.x) {
            const double v = a[(e % 16) * 16 + e / 16] + 0.0;
            t.c64[(size_t)u * 256 + e] = v;
            t.c32[(size_t)u * 256 + e] = (float)v;
            t.clo[(size_t)u * 256 + e] = (float)(v - (double)(float)v);
        }
    }
    if (threadIdx.x == 0) {
        t.mask[u] = rm | (cm << 16);
        t.s16[u] = (float)s;
    }
}

// Where the table kernels pay (event times in us, general / table; u: 26
// images as on uniform grids, otherwise quadtree levels).  A launch copies the
// images (nuniq blocks, ndiag inverse diagonal ones) to every CTA, their size
// bounds the CTAs of an SM, and a warp's rows of one class lie apart in the
// vectors: many rows and few images pay, the more the wider the block and in
// FP64, whose pipes the general kernels load with the zeros.
//   4 x 4, FP64 sweep: 47,899 rows 124 images 22.2 / 19.5, 65,536 u 28.2 / 20.2,
//     30,916 84 18.2 / 18.2 (residual 20.6 / 21.9), 55,567 472 24.6 / 30.6;
//     FP32: 65,536 u 11.8 / 9.5, 109,825 98 14.5 / 12.7, 47,899 124 9.8 / 9.9,
//     38,218 148 8.1 / 9.9, 77,575 492 12.2 / 13.9; double-float product: 65,536 u
//     25.2 / 21.7, 52,210 with 69 distinct 23.3 / 21.6, 47,899 82 20.8 / 22.6
//   9 x 9, FP64 sweep: 16,384 u 27.4 / 26.0, 50,347 70 67.6 / 54.8, 26,431 84 41.3 /
//     45.1, 16,765 118 28.9 / 36.6; FP32: 65,536 u 30.1 / 14.8, 50,347 70 24.1 /
//     21.2, 16,384 u 10.0 / 11.3 (residual 11.4 / 15.1), 47,899 120 23.1 / 26.1
//     (23.6 / 30.5), 65,593 96 30.3 / 27.2, 143,032 140 55.7 / 41.0; double-float:
//     50,347 47 73.8 / 60.5, 47,899 80 73.7 / 76.5, 26,431 56 44.8 / 55.5, 16,384 17
//     30.0 / 31.0
//   16 x 16, FP64 sweep: 16,384 u 56.2 / 35.2, 4,096 u 20.0 / 27.8; FP32: 16,384 u
//     20.7 / 11.3, 26,431 84 32.2 / 24.8, 15,559 96 22.5 / 22.9 (21.7 / 19.1),
//     11,542 88 17.8 / 22.0; FP16 values: 16,384 u 15.3 / 12.6, 65,593 96 49.5 /
//     32.8, 30,916 98 28.2 / 27.5, 26,431 84 25.2 / 28.5, 15,559 96 17.4 / 25.1
enum class Form { F64, F32, F16, DF };   // DF: the double-float product, which reads both halves of the blocks

// most images of a form with this many rows, -1: none
static int64_t rep_most_images(int b, Form f, int64_t rows) {
    if (b == 4) {
        if (f == Form::F64) return rows < 40000 ? -1 : rows / 160;
        if (f == Form::DF) return rows < 50000 ? -1 : rows / 600;
        return rows < 65536 ? -1 : rows / 400;
    }
    if (b == 9) {
        if (f == Form::F64) return rows < 16384 ? -1 : rows / 500;
        if (f == Form::DF) return rows < 32768 ? -1 : rows / 700;
        return rows < 32768 ? -1 : (rows < 65536 ? rows / 650 : rows / 400);
    }
    if (rows < 8192) return -1;
    return f == Form::F64 || f == Form::DF ? 1 << 30 : (f == Form::F16 ? rows / 400 : rows / 160);
}

constexpr int kRepSmem = 100 * 1024;   // largest shared-memory image (two CTAs per SM)

// bytes of `count` images in shared memory
static size_t rep_image_bytes(int b, Form f, int64_t count) {
    if (f == Form::F64) return 8 * count * (b == 16 ? Img<double, 16>::SIZE : b * ((b + 3) / 4 * 4));
    return (f == Form::DF ? 8 : 4) * count * (b == 16 ? Img<float, 16>::SIZE : b * ((b + 3) / 4 * 4));
}

static bool rep_pays(int b, Form f, int64_t rows, int64_t nuniq, int64_t ndiag) {
    const int64_t count = f == Form::DF ? nuniq : nuniq + ndiag;
    return count <= rep_most_images(b, f, rows) && rep_image_bytes(b, f, count) <= (size_t)kRepSmem;
}

// the forms a hierarchy's level runs in: its V-cycle's, on the finest level
// also the outer product's
static std::vector<Form> rep_forms(int b, int precision, bool finest) {
    if (precision == MGLDG_PREC_FP64) return {Form::F64};
    std::vector<Form> f{precision == MGLDG_PREC_MIXED_F16 && b == 16 ? Form::F16 : Form::F32};
    if (finest) f.push_back(Form::DF);
    return f;
}

static bool rep_shape(const mgldg_bsr* A, int min_rows) {
    return A->br == A->bc && A->nbr == A->nbc && !A->blk && (A->br == 4 || A->br == 9 || A->br == 16) &&
           A->nbr >= min_rows && A->nnzb < (1LL << 31);
}

static bool sample(mgldg_ctx* ctx, const mgldg_bsr* A, int* distinct, int min_rows) {
    if (A->rep || !rep_shape(A, min_rows)) return false;
    // keys and count in the reduction scratch
    unsigned long long* keys = (unsigned long long*)ctx->d_partials;
    int* count = (int*)(keys + kSampleKeys);
    MG_REQUIRE(ctx->n_partials > kSampleKeys, MGLDG_ERR_ARG, "reduction scratch too small");
    MG_CHECK_CUDA(cudaMemsetAsync(keys, 0, (kSampleKeys + 1) * sizeof(*keys), ctx->stream));
    const int m = (int)std::min<int64_t>(A->nnzb, kSample);
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_sample<<<(m + 7) / 8, 256, 0, ctx->stream>>>(A->nnzb, (int)A->bsz(), A->val, m, keys, count);
    }
    check_launch();
    download(ctx, distinct, count, 1);
    return true;
}

bool rep_sample(mgldg_ctx* ctx, const mgldg_bsr* A, int precision, bool finest, int* distinct) {
    bool any = false;
    for (Form f : rep_forms(A->br, precision, finest)) any = any || rep_most_images(A->br, f, A->nbr) >= 2;
    return any && sample(ctx, A, distinct, 1);
}

// pays(nuniq, ndiag): whether a table of that size is wanted
template <class F>
static void build(mgldg_ctx* ctx, mgldg_bsr* A, const double* Dinv, int distinct, int gs_want, F&& pays) {
    // (what rules the sample out rules all blocks out)
    if (distinct > kMaxUniq || (int64_t)distinct * 4 > A->nnzb || !pays(distinct, 1)) return;
    const int b = A->br, n = A->nbr, ld = (b + 3) / 4 * 4;
    const int* rp = A->h_row_ptr.data();
    if (A->nnzb > (int64_t)kRepMaxNb * n) return;
    for (int i = 0; i < n; ++i)
        if (rp[i + 1] - rp[i] > kRepMaxNb) return;
    struct Mem {
        char* p = nullptr;
        ~Mem() { dfree(p); }
    } mem;
    mem.p = dalloc<char>(16 + 2 * kHash * sizeof(HashSlot) +
                         ((size_t)A->nnzb + n + (size_t)kMaxCls * (kRepCls + 1)) * sizeof(int));
    int* head = (int*)mem.p;   // distinct blocks, not for a table; the same of the row classes
    HashSlot *slots = (HashSlot*)(mem.p + 16), *cslots = slots + kHash;
    int *slot_of = (int*)(cslots + kHash), *cls_of_d = slot_of + A->nnzb, *cfirst = cls_of_d + n, *cls_d = cfirst + kMaxCls;
    const int g = (int)std::min<int64_t>((A->nnzb + 7) / 8, ctx->sm_count * 8), gr = std::min((n + 255) / 256, ctx->sm_count * 8);
    // slots in the order of their first blocks or rows (independent of the
    // order in which the hashing threads arrived)
    std::vector<HashSlot> hs(kHash);
    auto number = [&](HashSlot* dev, std::vector<int>& first) {
        std::vector<int> order;
        for (int s = 0; s < kHash; ++s)
            if (hs[s].key) order.push_back(s);
        std::sort(order.begin(), order.end(), [&](int x, int y) { return hs[x].first < hs[y].first; });
        for (size_t u = 0; u < order.size(); ++u) {
            hs[order[u]].id = (int)u;
            first.push_back(hs[order[u]].first);
        }
        upload(ctx, dev, hs.data(), hs.size());
    };
    int hd[4] = {0, 0, 0, 0};
    k_rep_clear<<<2 * kHash / 256, 256, 0, ctx->stream>>>(slots, head);
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_hash<<<g, 256, 0, ctx->stream>>>(A->nnzb, (int)A->bsz(), A->val, slots, head, slot_of);
    }
    check_launch();
    download(ctx, hd, head, 4);
    download(ctx, hs.data(), slots, hs.size());
    sync(ctx);
    // a table pays when a block is used several times
    const int nu = hd[0];
    if (hd[1] || nu < 1 || (int64_t)nu * 4 > A->nnzb || !pays(nu, 1)) return;
    std::vector<int> first, cls_first;
    number(slots, first);
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_assign<<<g, 256, 0, ctx->stream>>>(A->nnzb, (int)A->bsz(), A->val, slots, head, slot_of);
    }
    // ---- row classes ----
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_row_hash<<<gr, 256, 0, ctx->stream>>>(n, A->row_ptr, A->diag, slot_of, cslots, head + 2, cls_of_d);
    }
    check_launch();
    download(ctx, hd, head, 4);
    download(ctx, hs.data(), cslots, hs.size());
    sync(ctx);
    if (hd[1] || hd[3]) return;   // two different blocks with one hash; too many classes
    number(cslots, cls_first);
    const int ncls = (int)cls_first.size();
    upload(ctx, cfirst, cls_first.data(), ncls);
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_classes<<<std::min((ncls * kRepCls + 255) / 256, ctx->sm_count), 256, 0, ctx->stream>>>(
            ncls, cfirst, A->row_ptr, A->diag, slot_of, cls_d);
    }
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_row_assign<<<gr, 256, 0, ctx->stream>>>(n, A->row_ptr, A->diag, slot_of, cslots, cls_d, head, cls_of_d);
    }
    check_launch();
    std::vector<int> cls_of(n), cls((size_t)ncls * kRepCls);   // cls: kRepCls ints per class
    download(ctx, hd, head, 4);
    download(ctx, cls.data(), cls_d, cls.size());
    download(ctx, cls_of.data(), cls_of_d, n);
    sync(ctx);
    if (hd[1]) return;
    std::vector<int> drow(nu, -1);   // a row with this diagonal block
    for (int c = 0; c < ncls; ++c) {
        int& d = drow[cls[(size_t)c * kRepCls + 1]];
        if (d < 0) d = cls_first[c];
    }
    if (!pays(nu, nu - (int)std::count(drow.begin(), drow.end(), -1))) return;
    // ---- slots: the rows of a chunk sorted by class, each class padded to
    // whole groups.  Chunks of 4,096 consecutive rows keep a warp's gathers
    // within one stretch of the vectors; with many classes one chunk wastes
    // fewer slots. ----
    const int gs = gs_want ? gs_want : (b != 16 || n >= 32768 ? 32 : 16), gu = std::min(gs, 16);
    const int chunk = ncls <= 32 ? 4096 : n;
    std::vector<int> rows, gcls;
    {
        std::vector<int> cnt(ncls + 1), pos(ncls);
        for (int s = 0; s < n; s += chunk) {
            const int e = std::min(n, s + chunk);
            std::fill(cnt.begin(), cnt.end(), 0);
            for (int i = s; i < e; ++i) cnt[cls_of[i]]++;
            size_t at = rows.size();
            for (int c = 0; c < ncls; ++c) {
                pos[c] = (int)at;
                const size_t w = ((size_t)cnt[c] + gs - 1) / gs * gs;
                gcls.insert(gcls.end(), w / gu, c);
                at += w;
            }
            rows.resize(at, -1);
            for (int i = s; i < e; ++i) rows[pos[cls_of[i]]++] = i;
        }
    }
    // more than twice as many slots as rows: rare classes, mostly idle lanes
    if (rows.size() > 2 * (size_t)n) return;
    const int nslots = (int)rows.size();
    std::unique_ptr<RepTable> t(new RepTable());
    t->b = b;
    t->ld = ld;
    t->nbr = n;
    t->nuniq = nu;
    t->ncls = ncls;
    t->gs = gs;
    t->gu = gu;
    t->nslots = nslots;
    // the classes name their inverse diagonal block by its place in the image
    std::vector<int> didx(nu, -1);
    for (int u = 0; u < nu; ++u)
        if (drow[u] >= 0) didx[u] = t->ndiag++;
    for (int c = 0; c < ncls; ++c) cls[(size_t)c * kRepCls + 1] = didx[cls[(size_t)c * kRepCls + 1]];
    // ---- device tables ----
    const size_t nimg = (size_t)nu + t->ndiag;
    const size_t v8 = (size_t)(b == 16 ? Img<double, 16>::SIZE : b * ld) * nimg;
    const size_t v4 = (size_t)(b == 16 ? Img<float, 16>::SIZE : b * ld) * nimg;
    const size_t vc = b == 16 ? (size_t)nu * 256 : 0;   // smaller blocks' images are by columns
    t->pool = dalloc<char>((v8 + vc) * 8 + (3 * v4 + 2 * vc) * 4 + (size_t)nu * 8);
    MG_CHECK_CUDA(cudaMemsetAsync(t->pool, 0, (v8 + vc) * 8 + (3 * v4 + 2 * vc) * 4, ctx->stream));
    t->i64 = (double*)t->pool;
    t->c64 = vc ? t->i64 + v8 : t->i64;
    t->i32 = (float*)(t->i64 + v8 + vc);
    t->ilo = t->i32 + v4;
    t->i16 = t->ilo + v4;
    t->c32 = vc ? t->i16 + v4 : t->i32;
    t->clo = vc ? t->c32 + vc : t->ilo;
    t->s16 = t->i16 + v4 + 2 * vc;
    t->mask = (unsigned*)(t->s16 + nu);
    int* dint = (int*)slots;   // the hash slots are done with: three index lists go there
    upload(ctx, dint, first.data(), first.size());
    upload(ctx, dint + nu, drow.data(), drow.size());
    upload(ctx, dint + 2 * nu, didx.data(), didx.size());
    {
        Launch L(ctx, MGLDG_K_SETUP);
        const RepView& v = *t;
        if (b == 4) k_rep_tables<4><<<nu, 256, 0, ctx->stream>>>(A->val, dint, dint + nu, dint + 2 * nu, Dinv, v);
        else if (b == 9) k_rep_tables<9><<<nu, 256, 0, ctx->stream>>>(A->val, dint, dint + nu, dint + 2 * nu, Dinv, v);
        else k_rep_tables<16><<<nu, 256, 0, ctx->stream>>>(A->val, dint, dint + nu, dint + 2 * nu, Dinv, v);
    }
    check_launch();
    std::vector<unsigned> mask(nu);
    download(ctx, mask.data(), t->mask, nu);
    sync(ctx);
    for (int c = 0; c < ncls; ++c) {
        int* d = &cls[(size_t)c * kRepCls];
        for (int q = 0; q < d[0]; ++q) d[4 + kRepMaxNb + q] = (int)mask[d[4 + q]];
    }
    int most = 0;
    for (int c = 0; c < ncls; ++c) most = std::max(most, cls[(size_t)c * kRepCls]);
    const size_t nc = cls.size(), ng = gcls.size();
    t->slots = dalloc<int>(nc + ng + nslots + (size_t)most * nslots + 16);
    t->cls = (int*)t->slots;
    t->cols = t->cls + nc;
    t->rows = t->cols + (size_t)most * nslots;
    t->gcls = t->rows + nslots;
    upload(ctx, t->cls, cls.data(), nc);
    upload(ctx, t->rows, rows.data(), nslots);
    upload(ctx, t->gcls, gcls.data(), ng);
    {
        Launch L(ctx, MGLDG_K_SETUP);
        k_rep_cols<<<std::min((nslots + 255) / 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(
            nslots, gs, most, t->rows, A->row_ptr, A->col_idx, t->cols);
    }
    check_launch();
    sync(ctx);   // the host arrays go out of scope
    A->rep = t.release();
}

void rep_build(mgldg_ctx* ctx, mgldg_bsr* A, const double* Dinv, int precision, bool finest, int distinct) {
    build(ctx, A, Dinv, distinct, 0, [&](int nuniq, int ndiag) {
        bool any = false;
        for (Form f : rep_forms(A->br, precision, finest))
            any = any || rep_pays(A->br, f, A->nbr, nuniq, ndiag);
        return any;
    });
}

void rep_ensure_batch(mgldg_ctx* ctx, mgldg_bsr* A, const double* Dinv, bool df64) {
    int distinct = 0;
    auto pays = [&](int nuniq, int) {
        return df64 ? rep_mm_df64_pays(A->br, A->nbr) : rep_mm_pays(A->br, A->nbr, nuniq);
    };
    if (!pays(1, 1) || !sample(ctx, A, &distinct, kRepMmRows)) return;
    sync(ctx);
    build(ctx, A, Dinv, distinct, 4, pays);
}

// ---------------------------------------------------------------- kernels --
namespace {

template <class T>
struct RepArgs {
    int nwarps, nslots, nimg, nuniq;
    const int *gcls, *rows, *cols, *cls;
    const unsigned* mask;
    const T* img;
    const float* scale;   // FP16 form: block scales
    const T *x, *b;
    T* y;
    T alpha, beta, omega;
    int xzero;
    const T* dotv;
    int self_dot;
    double* partials;
};

__device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }

// N values (N * sizeof(T) a multiple of 16) with 16-byte accesses; ldc: plain
// loads, for a line that the same lane may write later
template <int N>
__device__ __forceinline__ void lds(const float* p, float (&v)[N]) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const float4 t = reinterpret_cast<const float4*>(p)[q];
        v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
}
template <int N>
__device__ __forceinline__ void lds(const double* p, double (&v)[N]) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
        const double2 t = reinterpret_cast<const double2*>(p)[q];
        v[2 * q] = t.x; v[2 * q + 1] = t.y;
    }
}
template <int N>
__device__ __forceinline__ void ldg(const float* p, float (&v)[N]) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p) + q);
        v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
}
template <int N>
__device__ __forceinline__ void ldg(const double* p, double (&v)[N]) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p) + q);
        v[2 * q] = t.x; v[2 * q + 1] = t.y;
    }
}
__device__ __forceinline__ void st8(float* p, const float (&v)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void st8(double* p, const double (&v)[8]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) reinterpret_cast<double2*>(p)[q] = make_double2(v[2 * q], v[2 * q + 1]);
}

// copies the image (nvec 16-byte words) to shared memory
__device__ __forceinline__ void load_image(const void* g, void* s, int nvec) {
    const float4* gp = reinterpret_cast<const float4*>(g);
    float4* sp = reinterpret_cast<float4*>(s);
#pragma unroll 8
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) sp[i] = __ldg(gp + i);
    __syncthreads();
}

// CTA sum of dacc into partials[blockIdx.x] (fixed order)
__device__ __forceinline__ void rep_partial(double dacc, double* partials) {
    __shared__ double sm[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dacc += __shfl_xor_sync(0xffffffffu, dacc, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = dacc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sm[w];
        partials[blockIdx.x] = t;
    }
}

// the lane pair (column halves) holds two partial sums of 16 rows each; the
// lane gets the sums of the 8 rows of its half
template <class T>
__device__ __forceinline__ void pair_sum(const T (&p)[16], int half, T (&s)[8]) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const T other = __shfl_xor_sync(0xffffffffu, half ? p[r] : p[r + 8], 1);
        s[r] = (half ? p[r + 8] : p[r]) + other;
    }
}

// p[e] += the lane's column half of (A x)_i for its E rows (slots slot + 16 e).
// The gathers of block k + 1 and the column indices of block k + 2 are in
// flight while block k is applied (their latency, three loads in a row,
// otherwise bounds the kernel: 65,536 rows, E = 2, 19.6 us at 73 % of the
// warps' time in it).
template <class T, int E, bool F16>
__device__ __forceinline__ void acc16(const RepArgs<T>& a, const T* simg, const int* cls, int slot, int half,
                                      T (&p)[E][16]) {
    using I = Img<T, 16>;
    const int nb = __ldg(cls);
    const int* cp = a.cols + slot;
    const T* xh = a.x + 8 * half;
    int col[E];
    T xn[E][8];
#pragma unroll
    for (int e = 0; e < E; ++e) ldg<8>(xh + (size_t)__ldg(cp + 16 * e) * 16, xn[e]);
#pragma unroll
    for (int e = 0; e < E; ++e) col[e] = nb > 1 ? __ldg(cp + a.nslots + 16 * e) : 0;
    int id = __ldg(cls + 4);
    unsigned m = (unsigned)__ldg(cls + 4 + kRepMaxNb);
#pragma unroll 1
    for (int k = 0; k < nb; ++k) {
        T xv[E][8];
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
            for (int c = 0; c < 8; ++c) xv[e][c] = xn[e][c];
        const int idk = id;
        const unsigned rm = m & 0xffffu, cm = m >> 16;
        if (k + 1 < nb) {
#pragma unroll
            for (int e = 0; e < E; ++e) ldg<8>(xh + (size_t)col[e] * 16, xn[e]);
            id = __ldg(cls + 5 + k);
            m = (unsigned)__ldg(cls + 5 + kRepMaxNb + k);
        }
        if (k + 2 < nb) {
            const int* cq = cp + (size_t)(k + 2) * a.nslots;
#pragma unroll
            for (int e = 0; e < E; ++e) col[e] = __ldg(cq + 16 * e);
        }
        const T* ab = simg + idk * I::SIZE;
        if (F16 || __popc(rm) < __popc(cm)) {
            const T sc = F16 ? (T)__ldg(a.scale + idk) : T(0);
#pragma unroll
            for (int r = 0; r < 16; ++r)
                if ((rm >> r) & 1u) {
                    T av[8];
                    lds<8>(ab + I::line(r) + 8 * half, av);
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        if (F16) {
                            T t = av[0] * xv[e][0];
#pragma unroll
                            for (int c = 1; c < 8; ++c) t = fma_(av[c], xv[e][c], t);
                            p[e][r] = fma_(sc, t, p[e][r]);
                        } else {
#pragma unroll
                            for (int c = 0; c < 8; ++c) p[e][r] = fma_(av[c], xv[e][c], p[e][r]);
                        }
                    }
                }
        } else {
            const unsigned any = cm | (cm >> 8);
            const T* ac = ab + (half ? I::line(8) : 0);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if ((any >> c) & 1u) {
                    T av[16];
                    lds<16>(ac + c * 16, av);
#pragma unroll
                    for (int e = 0; e < E; ++e)
#pragma unroll
                        for (int r = 0; r < 16; ++r) p[e][r] = fma_(av[r], xv[e][c], p[e][r]);
                }
        }
    }
}

// 16 x 16 blocks.  JACOBI: y = x + omega Dinv (b - A x); else y = alpha A x + beta b
template <class T, int E, bool JACOBI, bool F16>
__global__ void __launch_bounds__(128) k_rep16(const RepArgs<T> a) {
    using I = Img<T, 16>;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* simg = reinterpret_cast<T*>(smraw);
    const bool zero = JACOBI && a.xzero;
    // the sweep from x = 0 reads the inverse diagonal blocks only
    const int first = zero ? a.nuniq : 0;
    load_image(a.img + (size_t)first * I::SIZE, simg + first * I::SIZE,
               (a.nimg - first) * (I::SIZE * (int)sizeof(T) / 16));
    const int lane = threadIdx.x & 31, half = lane & 1;
    double dacc = 0;
    for (int w = blockIdx.x * 4 + (threadIdx.x >> 5); w < a.nwarps; w += gridDim.x * 4) {
        const int slot = w * 16 * E + (lane >> 1);
        const int* cls = a.cls + (size_t)__ldg(a.gcls + w * E) * kRepCls;
        T p[E][16];
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
            for (int r = 0; r < 16; ++r) p[e][r] = T(0);
        if (!zero) acc16<T, E, F16>(a, simg, cls, slot, half, p);
        if constexpr (JACOBI) {
            T t[E][8];
            size_t o[E];
            bool live[E];
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int row = __ldg(a.rows + slot + 16 * e);
                live[e] = row >= 0;
                o[e] = (size_t)max(row, 0) * 16 + 8 * half;
                T bv[8];
                ldg<8>(a.b + o[e], bv);
                if (zero) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) t[e][r] = bv[r];
                } else {
                    pair_sum(p[e], half, t[e]);
#pragma unroll
                    for (int r = 0; r < 8; ++r) t[e][r] = bv[r] - t[e][r];
                }
            }
            const T* D = simg + (size_t)(a.nuniq + __ldg(cls + 1)) * I::SIZE;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                T dv[8];
                lds<8>(D + I::line(r) + 8 * half, dv);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    T y = dv[0] * t[e][0];
#pragma unroll
                    for (int c = 1; c < 8; ++c) y = fma_(dv[c], t[e][c], y);
                    p[e][r] = y;
                }
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                T yv[8], xi[8];
                pair_sum(p[e], half, yv);
                if (zero) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) xi[r] = T(0);
                } else {
                    ldg<8>(a.x + o[e], xi);
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) xi[r] = xi[r] + a.omega * yv[r];
                if (live[e]) st8(a.y + o[e], xi);
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                T s[8];
                pair_sum(p[e], half, s);
                const int row = __ldg(a.rows + slot + 16 * e);
                if (row < 0) continue;
                const size_t o = (size_t)row * 16 + 8 * half;
                T v[8], bv[8];
                if (a.beta != T(0)) lds<8>(a.b + o, bv);   // yin may be y: plain loads, this lane's entries only
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    v[r] = a.alpha * s[r];
                    if (a.beta != T(0)) v[r] += a.beta * bv[r];
                }
                st8(a.y + o, v);
                if (a.self_dot) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) dacc += (double)v[r] * (double)v[r];
                } else if (a.dotv) {
                    ldg<8>(a.dotv + o, bv);
#pragma unroll
                    for (int r = 0; r < 8; ++r) dacc += (double)v[r] * (double)bv[r];
                }
            }
        }
    }
    if (!JACOBI && a.partials) rep_partial(dacc, a.partials);
}

// Blocks of 4 and 9, one row per lane: CB columns at a time, one sum per
// (row, column) over the row's blocks, then the columns in order.
template <class T, int B, bool JACOBI>
__global__ void __launch_bounds__(128) k_repc(const RepArgs<T> a) {
    using I = Img<T, B>;
    constexpr int CB = B == 9 ? 3 : 4, LD = I::LD;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* simg = reinterpret_cast<T*>(smraw);
    const bool zero = JACOBI && a.xzero;
    const int first = zero ? a.nuniq : 0;
    load_image(a.img + (size_t)first * I::SIZE, simg + first * I::SIZE,
               (a.nimg - first) * (I::SIZE * (int)sizeof(T) / 16));
    const int lane = threadIdx.x & 31;
    double dacc = 0;
    for (int w = blockIdx.x * 4 + (threadIdx.x >> 5); w < a.nwarps; w += gridDim.x * 4) {
        const int slot = w * 32 + lane;
        const int* cls = a.cls + (size_t)__ldg(a.gcls + 2 * w) * kRepCls;
        T s[B];
#pragma unroll
        for (int r = 0; r < B; ++r) s[r] = T(0);
        if (!zero) {
            const int nb = __ldg(cls);
#pragma unroll 1
            for (int cb = 0; cb < B; cb += CB) {
                T acc[CB][B];
#pragma unroll
                for (int q = 0; q < CB; ++q)
#pragma unroll
                    for (int r = 0; r < B; ++r) acc[q][r] = T(0);
#pragma unroll 2
                for (int k = 0; k < nb; ++k) {
                    const int id = __ldg(cls + 4 + k);
                    const unsigned cm = __ldg(a.mask + id) >> (16 + cb);
                    if (!(cm & ((1u << CB) - 1u))) continue;
                    const T* ac = simg + id * I::SIZE + cb * LD;
                    const T* xp = a.x + (size_t)__ldg(a.cols + (size_t)k * a.nslots + slot) * B + cb;
                    T xv[CB];
#pragma unroll
                    for (int q = 0; q < CB; ++q) xv[q] = __ldg(xp + q);
#pragma unroll
                    for (int q = 0; q < CB; ++q) {
                        if (!((cm >> q) & 1u)) continue;
                        T av[LD];
                        lds<LD>(ac + q * LD, av);
#pragma unroll
                        for (int r = 0; r < B; ++r) acc[q][r] = fma_(av[r], xv[q], acc[q][r]);
                    }
                }
#pragma unroll
                for (int q = 0; q < CB; ++q)
#pragma unroll
                    for (int r = 0; r < B; ++r) s[r] += acc[q][r];
            }
        }
        const int row = __ldg(a.rows + slot);
        const size_t o = (size_t)max(row, 0) * B;
        if constexpr (JACOBI) {
            const T* D = simg + (size_t)(a.nuniq + __ldg(cls + 1)) * I::SIZE;
#pragma unroll
            for (int r = 0; r < B; ++r) s[r] = __ldg(a.b + o + r) - s[r];
#pragma unroll
            for (int r = 0; r < B; ++r) {
                T dv[LD];
                lds<LD>(D + r * LD, dv);
                T y = T(0);
#pragma unroll
                for (int c = 0; c < B; ++c) y = fma_(dv[c], s[c], y);
                const T xi = zero ? T(0) : __ldg(a.x + o + r);
                if (row >= 0) a.y[o + r] = xi + a.omega * y;
            }
        } else if (row >= 0) {
#pragma unroll
            for (int r = 0; r < B; ++r) {
                T v = a.alpha * s[r];
                if (a.beta != T(0)) v += a.beta * a.b[o + r];
                a.y[o + r] = v;
                if (a.self_dot) dacc += (double)v * (double)v;
                else if (a.dotv) dacc += (double)v * (double)__ldg(a.dotv + o + r);
            }
        }
    }
    if (!JACOBI && a.partials) rep_partial(dacc, a.partials);
}

struct RepDfArgs {
    int nwarps, nslots, nuniq;
    const int *gcls, *rows, *cols, *cls;
    const unsigned* mask;
    const float *img, *imglo;
    const float *xh, *xl;
    const double* d;
    double* q;
    double* partials;
};

// q = A d in double-float arithmetic, 16 x 16 blocks, two lanes per row: a
// float-pair sum per row and column half, the two pairs added as in FP64
// (PairSum), q and the partial d.q in FP64.  Blocks read by columns take two
// rows at a time (packed FP32 operations).  The work is on the FP32 pipes (11
// operations per product, zero block rows and columns skipped; 34 % of the
// cycles at 65,536 rows, one wave of CTAs) and the FP64 ones (three operations
// per entry; adding the halves as float pairs and widening without conversions
// took away five more; 21 %).  262,144 rows: 122 us with four CTAs an SM and x
// loaded a block ahead, 110 us with five and without.
__global__ void __launch_bounds__(128, 5) k_rep16_df64(const RepDfArgs a) {
    using I = Img<float, 16>;
    extern __shared__ __align__(16) unsigned char smraw[];
    float* sh_ = reinterpret_cast<float*>(smraw);
    float* sl_ = sh_ + a.nuniq * I::SIZE;
    load_image(a.img, sh_, a.nuniq * (I::SIZE / 4));
    load_image(a.imglo, sl_, a.nuniq * (I::SIZE / 4));
    const int lane = threadIdx.x & 31, half = lane & 1;
    double dacc = 0;
    for (int w = blockIdx.x * 4 + (threadIdx.x >> 5); w < a.nwarps; w += gridDim.x * 4) {
        const int slot = w * 16 + (lane >> 1);
        const int* cls = a.cls + (size_t)__ldg(a.gcls + w) * kRepCls;
        const int nb = __ldg(cls);
        const int* cp = a.cols + slot;
        unsigned long long sh[8], sl[8];   // rows 2 r, 2 r + 1
#pragma unroll
        for (int r = 0; r < 8; ++r) sh[r] = sl[r] = 0ULL;
        int col = __ldg(cp);
        int id = __ldg(cls + 4);
        unsigned m = (unsigned)__ldg(cls + 4 + kRepMaxNb);
#pragma unroll 1
        for (int k = 0; k < nb; ++k) {
            float xh[8], xl[8];
            const size_t xo = (size_t)col * 16 + 8 * half;
            ldg<8>(a.xh + xo, xh);
            ldg<8>(a.xl + xo, xl);
            const unsigned rm = m & 0xffffu, cm = m >> 16;
            const int bo = id * I::SIZE;
            if (k + 1 < nb) {
                col = __ldg(cp + (size_t)(k + 1) * a.nslots);
                id = __ldg(cls + 5 + k);
                m = (unsigned)__ldg(cls + 5 + kRepMaxNb + k);
            }
            if (__popc(rm) < __popc(cm)) {
#pragma unroll
                for (int r = 0; r < 16; ++r)
                    if ((rm >> r) & 1u) {
                        float ah[8], al[8];
                        lds<8>(sh_ + bo + I::line(r) + 8 * half, ah);
                        lds<8>(sl_ + bo + I::line(r) + 8 * half, al);
                        float2 h = unpack2(sh[r / 2]), l = unpack2(sl[r / 2]);
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            df_fma(r & 1 ? h.y : h.x, r & 1 ? l.y : l.x, ah[c], al[c], xh[c], xl[c]);
                        sh[r / 2] = pack2(h.x, h.y);
                        sl[r / 2] = pack2(l.x, l.y);
                    }
            } else {
                const unsigned any = cm | (cm >> 8);
                const int co = bo + (half ? I::line(8) : 0);
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if ((any >> c) & 1u) {
                        float ah[16], al[16];
                        lds<16>(sh_ + co + c * 16, ah);
                        lds<16>(sl_ + co + c * 16, al);
                        const unsigned long long d2 = pack2(xh[c], xh[c]), n2 = pack2(-xh[c], -xh[c]),
                                                 e2 = pack2(xl[c], xl[c]);
#pragma unroll
                        for (int r = 0; r < 8; ++r)
                            df_fma2(sh[r], sl[r], pack2(ah[2 * r], ah[2 * r + 1]), pack2(al[2 * r], al[2 * r + 1]), d2,
                                    n2, e2);
                    }
            }
        }
        const int row = __ldg(a.rows + slot);
        const size_t o = (size_t)max(row, 0) * 16 + 8 * half;
        double dv[8], qv[8];
        ldg<8>(a.d + o, dv);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float2 h0 = unpack2(sh[r / 2]), h1 = unpack2(sh[r / 2 + 4]);
            const float2 l0 = unpack2(sl[r / 2]), l1 = unpack2(sl[r / 2 + 4]);
            const float ha = r & 1 ? h0.y : h0.x, hb = r & 1 ? h1.y : h1.x;
            const float la = r & 1 ? l0.y : l0.x, lb = r & 1 ? l1.y : l1.x;
            const float oh = __shfl_xor_sync(0xffffffffu, half ? ha : hb, 1);
            const float ol = __shfl_xor_sync(0xffffffffu, half ? la : lb, 1);
            const float mh = half ? hb : ha, ml = half ? lb : la;
            PairSum v{mh, ml};
            v.add(oh, ol);
            qv[r] = v.value();
            if (row >= 0) dacc += qv[r] * dv[r];
        }
        if (row >= 0) st8(a.q + o, qv);
    }
    rep_partial(dacc, a.partials);
}

// the same for blocks of 4 and 9, one lane per row: one float-pair sum per
// (row, column) over the row's blocks, summed over the columns in FP64
template <int B>
__global__ void __launch_bounds__(128) k_repc_df64(const RepDfArgs a) {
    using I = Img<float, B>;
    constexpr int LD = I::LD;
    extern __shared__ __align__(16) unsigned char smraw[];
    float* sh_ = reinterpret_cast<float*>(smraw);
    float* sl_ = sh_ + a.nuniq * I::SIZE;
    load_image(a.img, sh_, a.nuniq * (I::SIZE / 4));
    load_image(a.imglo, sl_, a.nuniq * (I::SIZE / 4));
    const int lane = threadIdx.x & 31;
    double dacc = 0;
    for (int w = blockIdx.x * 4 + (threadIdx.x >> 5); w < a.nwarps; w += gridDim.x * 4) {
        const int slot = w * 32 + lane;
        const int* cls = a.cls + (size_t)__ldg(a.gcls + 2 * w) * kRepCls;
        const int nb = __ldg(cls);
        double v[B];
#pragma unroll
        for (int r = 0; r < B; ++r) v[r] = 0.0;
#pragma unroll 1
        for (int c = 0; c < B; ++c) {
            float sh[B], sl[B];
#pragma unroll
            for (int r = 0; r < B; ++r) sh[r] = sl[r] = 0.f;
#pragma unroll 2
            for (int k = 0; k < nb; ++k) {
                const int id = __ldg(cls + 4 + k);
                if (!((__ldg(a.mask + id) >> (16 + c)) & 1u)) continue;
                const size_t xo = (size_t)__ldg(a.cols + (size_t)k * a.nslots + slot) * B + c;
                const float xh = __ldg(a.xh + xo), xl = __ldg(a.xl + xo);
                float ah[LD], al[LD];
                lds<LD>(sh_ + id * I::SIZE + c * LD, ah);
                lds<LD>(sl_ + id * I::SIZE + c * LD, al);
#pragma unroll
                for (int r = 0; r < B; ++r) df_fma(sh[r], sl[r], ah[r], al[r], xh, xl);
            }
#pragma unroll
            for (int r = 0; r < B; ++r) v[r] += (double)sh[r] + (double)sl[r];
        }
        const int row = __ldg(a.rows + slot);
        if (row >= 0) {
            const size_t o = (size_t)row * B;
#pragma unroll
            for (int r = 0; r < B; ++r) {
                a.q[o + r] = v[r];
                dacc += v[r] * __ldg(a.d + o + r);
            }
        }
    }
    rep_partial(dacc, a.partials);
}

template <class T>
RepArgs<T> rep_args(const RepTable* t, bool f16) {
    RepArgs<T> a{};
    a.nslots = t->nslots;
    a.nuniq = t->nuniq;
    a.nimg = t->nuniq + t->ndiag;
    a.gcls = t->gcls;
    a.rows = t->rows;
    a.cols = t->cols;
    a.cls = t->cls;
    a.mask = t->mask;
    if constexpr (std::is_same<T, float>::value) {
        a.img = f16 ? t->i16 : t->i32;
        a.scale = t->s16;
    } else {
        a.img = t->i64;
    }
    return a;
}

// one launch of a slot kernel (128 threads, `smem` bytes of images): as many
// CTAs as fit at once, so that each copies the images once
template <class K, class A>
void rep_launch_k(mgldg_ctx* ctx, K kern, const A& a, size_t smem, int kclass, int* npart) {
    if (smem > 48 * 1024)
        MG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRepSmem));
    int per_sm = 0;
    MG_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, smem));
    int grid = std::max(1, std::min((a.nwarps + 3) / 4, std::max(1, per_sm) * ctx->sm_count));
    if (npart) grid = std::min(grid, ctx->n_partials);
    {
        Launch L(ctx, kclass);
        kern<<<grid, 128, smem, ctx->stream>>>(a);
    }
    check_launch();
    if (npart) *npart = grid;
}

template <class T, bool JACOBI>
void rep_launch(mgldg_ctx* ctx, const RepTable* t, RepArgs<T>& a, Form form, int kclass, int* npart) {
    const int E = std::is_same<T, float>::value ? t->gs / 16 : 1;
    a.nwarps = t->b == 16 ? t->nslots / (16 * E) : t->nslots / 32;
    const size_t smem = rep_image_bytes(t->b, form, a.nimg);
    if (t->b == 4) {
        rep_launch_k(ctx, k_repc<T, 4, JACOBI>, a, smem, kclass, npart);
    } else if (t->b == 9) {
        rep_launch_k(ctx, k_repc<T, 9, JACOBI>, a, smem, kclass, npart);
    } else if constexpr (std::is_same<T, float>::value) {
        // two rows per lane pair from 32,768 rows on (four measured no better:
        // 35.7 against 32.5 us per sweep of 262,144 rows)
        if (form == Form::F16) {
            if (E == 2) rep_launch_k(ctx, k_rep16<float, 2, JACOBI, true>, a, smem, kclass, npart);
            else rep_launch_k(ctx, k_rep16<float, 1, JACOBI, true>, a, smem, kclass, npart);
        } else {
            if (E == 2) rep_launch_k(ctx, k_rep16<float, 2, JACOBI, false>, a, smem, kclass, npart);
            else rep_launch_k(ctx, k_rep16<float, 1, JACOBI, false>, a, smem, kclass, npart);
        }
    } else {
        rep_launch_k(ctx, k_rep16<double, 1, JACOBI, false>, a, smem, kclass, npart);
    }
}

}  // namespace

// (groups of 4 slots, made for multi-vectors, are no whole warps)
static bool rep_used(const RepTable* t, Form f) {
    return t && t->gs >= 16 && rep_pays(t->b, f, t->nbr, t->nuniq, t->ndiag);
}
template <class T>
static Form form_of(const RepTable* t, bool f16) {
    if (std::is_same<T, double>::value) return Form::F64;
    return f16 && t && t->b == 16 ? Form::F16 : Form::F32;   // smaller blocks keep FP32 in the F16 form
}

template <class T>
bool rep_spmv(mgldg_ctx* ctx, const mgldg_bsr* A, T alpha, const T* x, T beta, const T* yin, T* y, const T* dotv,
              double* partials, int* npart, int kclass, bool f16) {
    const RepTable* t = A->rep;
    const Form form = form_of<T>(t, f16);
    if (!rep_used(t, form)) return false;
    // 16 x 16: whole 16-byte words of every vector (the general kernels read
    // only x that way)
    if (t->b == 16 && ((uintptr_t)x | (uintptr_t)(beta != T(0) ? yin : nullptr) | (uintptr_t)y | (uintptr_t)dotv) % 16)
        return false;
    RepArgs<T> a = rep_args<T>(t, form == Form::F16);
    a.x = x;
    a.b = yin;
    a.y = y;
    a.alpha = alpha;
    a.beta = beta;
    a.self_dot = (dotv != nullptr && dotv == y) ? 1 : 0;
    a.dotv = a.self_dot ? nullptr : dotv;
    a.partials = partials;
    rep_launch<T, false>(ctx, t, a, form, kclass, npart);
    return true;
}
template bool rep_spmv<float>(mgldg_ctx*, const mgldg_bsr*, float, const float*, float, const float*, float*,
                              const float*, double*, int*, int, bool);
template bool rep_spmv<double>(mgldg_ctx*, const mgldg_bsr*, double, const double*, double, const double*, double*,
                               const double*, double*, int*, int, bool);

template <class T>
bool rep_jacobi(mgldg_ctx* ctx, const mgldg_bsr* A, const T* b, const T* xin, T* xout, T omega, bool xzero, bool f16) {
    const RepTable* t = A->rep;
    const Form form = form_of<T>(t, f16);
    if (!rep_used(t, form)) return false;
    RepArgs<T> a = rep_args<T>(t, form == Form::F16);
    a.x = xin;
    a.b = b;
    a.y = xout;
    a.omega = omega;
    a.xzero = xzero ? 1 : 0;
    rep_launch<T, true>(ctx, t, a, form, MGLDG_K_JACOBI, nullptr);
    return true;
}
template bool rep_jacobi<float>(mgldg_ctx*, const mgldg_bsr*, const float*, const float*, float*, float, bool, bool);
template bool rep_jacobi<double>(mgldg_ctx*, const mgldg_bsr*, const double*, const double*, double*, double, bool,
                                 bool);

bool rep_df64(mgldg_ctx* ctx, const mgldg_bsr* A, const float* dhi, const float* dlo, const double* d, double* q,
              double* partials, int* npart) {
    const RepTable* t = A->rep;
    if (!rep_used(t, Form::DF)) return false;
    RepDfArgs a{};
    a.nwarps = t->nslots / (t->b == 16 ? 16 : 32);
    a.nslots = t->nslots;
    a.nuniq = t->nuniq;
    a.gcls = t->gcls;
    a.rows = t->rows;
    a.cols = t->cols;
    a.cls = t->cls;
    a.mask = t->mask;
    a.img = t->i32;
    a.imglo = t->ilo;
    a.xh = dhi;
    a.xl = dlo;
    a.d = d;
    a.q = q;
    a.partials = partials;
    const size_t smem = rep_image_bytes(t->b, Form::DF, t->nuniq);
    if (t->b == 4) rep_launch_k(ctx, k_repc_df64<4>, a, smem, MGLDG_K_SPMV, npart);
    else if (t->b == 9) rep_launch_k(ctx, k_repc_df64<9>, a, smem, MGLDG_K_SPMV, npart);
    else rep_launch_k(ctx, k_rep16_df64, a, smem, MGLDG_K_SPMV, npart);
    return true;
}

}  // namespace mg
