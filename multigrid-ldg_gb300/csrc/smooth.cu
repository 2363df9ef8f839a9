// smooth.cu -- block smoothers: fused damped block-Jacobi and block
// Gauss-Seidel run as a level-scheduled dataflow sweep that reproduces the
// reference's sequential order exactly.
//
// Reference: Level::jacobi and Level::gauss_seidel
// (src/cartesian/multigrid/multigrid.h:223-262).  The diagonal blocks are
// pre-inverted (Dinv) instead of LDL^T-solved.
//
// Gauss-Seidel.  A forward sweep updates block rows i = 0..n-1 in order,
// using new values of the neighbours j < i and old values of j > i.  Row i
// therefore depends only on its earlier neighbours; rows are grouped into
// level sets (level(i) = 1 + max level of its earlier neighbours) and the
// rows of one level are independent.  One persistent cooperative launch
// covers a pass of consecutive sweeps: warps take rows in level order, read
// the later neighbours (their old values are stable until row i publishes,
// because each of them waits for row i), wait for the earlier neighbours'
// published values, finish the row and publish it; blocks of up to 16 in tiles
// of rows per CTA (k_gs_tiles), 25 and 27 row by row (k_gs_pass).  Every wait
// is bounded (about one second of %globaltimer);
// on expiry the kernel records an error word, every other waiter gives up,
// and the host returns MGLDG_ERR_TIMEOUT with the context still usable.
// The sweep counter lives in device memory and is advanced by the last CTA
// to finish, so consecutive sweeps need no host involvement.
#include <algorithm>
#include <type_traits>

#include "api.cuh"
#include "rowdot.cuh"
#include "rowsplit.cuh"
#include "smooth.cuh"

using namespace mg;

namespace mg {

// ---------------------------------------------------------------- helpers --
template <class T, int BR, int BC>
__device__ __forceinline__ T chunk_dot_coherent(const T* __restrict__ a, const T* xj, int r, int c0) {
    // block values through the read-only path, x through L2 (it changes
    // during the sweep)
    using L = WL<BR, BC>;
    T acc = 0;
#pragma unroll
    for (int c = 0; c < L::CH; ++c)
        if (c0 + c < BC) acc += __ldg(a + r * BC + c0 + c) * __ldcg(xj + c0 + c);
    return acc;
}

// y_r = sum_c D(r,c) t_c where t_c is held by lane c*S (rows' first lanes)
template <class T, int B>
__device__ __forceinline__ T apply_block(const T* __restrict__ D, T t_mine, int r, int c0) {
    using L = WL<B, B>;
    T acc = 0;
#pragma unroll
    for (int c = 0; c < L::CH; ++c) {
        const int cc = c0 + c;
        T tc = __shfl_sync(0xffffffffu, t_mine, (cc * L::S) & 31);
        if (cc < B && r < B) acc += __ldg(D + r * B + cc) * tc;
    }
    return seg_sum<L::S>(acc);
}

__device__ __forceinline__ bool wait_flag(const unsigned* f, unsigned target, GsSync* sync, int64_t timeout_ns) {
    const uint64_t t0 = globaltimer_ns();
    unsigned it = 0;
    while (true) {
        const unsigned v = ld_acquire_u32(f);
        if ((int)(v - target) >= 0) return true;
        if ((++it & 63u) == 0) {
            if (*(volatile unsigned*)&sync->err) return false;
            if ((int64_t)(globaltimer_ns() - t0) > timeout_ns) {
                atomicOr(&sync->err, 1u);
                return false;
            }
            __nanosleep(32);
        }
    }
}

// ------------------------------------------------------------ GS pass --
// One launch runs a smoothing pass: nsw consecutive sweeps in one direction
// (the npre forward or npost reverse sweeps of multigrid.h:202-216).  Its
// work items are (sweep s, row i), ordered by the level sets of the combined
// dependency graph: (s, i) needs sweep s's new values of its earlier
// neighbours and sweep s-1's values of its later neighbours and of itself, so
// sweep s+1 trails sweep s by a few levels instead of starting after it
// (2 n_side + 1 dependent steps for two sweeps of an n_side^2 grid, not
// 2 (2 n_side - 1)).  Every row reads exactly the values the sequential
// sweeps of the reference read.
//
// Rows publish their values as packed 64-bit words, (epoch << 32) | 32 value
// bits: one word per FP32 entry, two (high and low halves) per FP64 entry,
// written and read with relaxed gpu-scope 64-bit accesses (single-copy
// atomic), so a reader that finds every word of a row at the epoch it needs
// holds that version of the row -- no separate flag, fence or second read on
// the dependency's critical path.  Epoch base + s + 1 marks sweep s of the
// launch whose device-side counter reads base; the last CTA to finish adds
// nsw.  Values a row reads before its launch's first sweep touches them come
// from the plain vector x, which only the last sweep of the pass writes.
// Every wait is bounded (about one second of %globaltimer); on expiry the
// kernel records an error word, every other waiter gives up and the host
// returns MGLDG_ERR_TIMEOUT with the context still usable.
template <class T>
struct Packed {
    static constexpr int WPV = sizeof(T) / 4;   // 64-bit words per entry
};

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Reads the packed row j (W words, word w in lane w % 32, register w / 32)
// until every word carries an epoch at or after tgt.  Warp-uniform result:
// false if the wait ran out or another waiter gave up.
template <int W>
__device__ __forceinline__ bool read_row(const unsigned long long* xp, int j, unsigned tgt, unsigned (&v)[(W + 31) / 32],
                                         GsSync* sync, int64_t timeout_ns, int lane) {
    constexpr int NW = (W + 31) / 32;
    const unsigned long long* row = xp + (size_t)j * W;
    uint64_t t0 = 0;
    unsigned it = 0;
    while (true) {
        bool ok = true;
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const int w = lane + 32 * q;
            if (w < W) {
                const unsigned long long u = ld_relaxed_u64(row + w);
                v[q] = (unsigned)u;
                ok = ok && (int)((unsigned)(u >> 32) - tgt) >= 0;
            }
        }
        if (__all_sync(0xffffffffu, ok)) return true;
        if ((++it & 15u) == 0) {
            if (it == 16) t0 = globaltimer_ns();
            bool stop = *(volatile unsigned*)&sync->err != 0;
            if (!stop && (int64_t)(globaltimer_ns() - t0) > timeout_ns) {
                atomicOr(&sync->err, 1u);
                stop = true;
            }
            if (__any_sync(0xffffffffu, stop)) return false;
        }
    }
}

// Polls several packed rows at once: the rows of the slots in `sel` (a
// warp-uniform bit mask) are loaded together, one L2 round trip per polling
// round, until every word of each carries an epoch at or after its target.
// Warp-uniform result: false if the wait ran out or another waiter gave up.
template <int W, int MAXE>
__device__ __forceinline__ bool poll_rows(const unsigned long long* xp, const int (&rows)[MAXE],
                                          const unsigned (&tgt)[MAXE], unsigned sel,
                                          unsigned (&v)[MAXE][(W + 31) / 32], GsSync* sync, int64_t timeout_ns,
                                          int lane) {
    constexpr int NW = (W + 31) / 32;
    uint64_t t0 = 0;
    unsigned it = 0;
    unsigned pending = sel;
    while (pending) {
        unsigned long long u[MAXE][NW];
        // issue every load of the round before checking any of them
#pragma unroll
        for (int q = 0; q < MAXE; ++q)
            if ((pending >> q) & 1u) {
                const unsigned long long* row = xp + (size_t)rows[q] * W;
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    const int w = lane + 32 * k;
                    u[q][k] = w < W ? ld_relaxed_u64(row + w) : ((unsigned long long)tgt[q] << 32);
                }
            }
        unsigned still = 0;
#pragma unroll
        for (int q = 0; q < MAXE; ++q)
            if ((pending >> q) & 1u) {
                bool ok = true;
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    v[q][k] = (unsigned)u[q][k];
                    ok = ok && (int)((unsigned)(u[q][k] >> 32) - tgt[q]) >= 0;
                }
                if (!__all_sync(0xffffffffu, ok)) still |= 1u << q;
            }
        pending = still;
        if (!pending) return true;
        if ((++it & 15u) == 0) {
            if (it == 16) t0 = globaltimer_ns();
            bool stop = *(volatile unsigned*)&sync->err != 0;
            if (!stop && (int64_t)(globaltimer_ns() - t0) > timeout_ns) {
                atomicOr(&sync->err, 1u);
                stop = true;
            }
            if (__any_sync(0xffffffffu, stop)) return false;
        }
    }
    return true;
}

// entry cc of a row read by read_row (every lane of the warp takes part)
template <class T, int W>
__device__ __forceinline__ T row_entry(const unsigned (&v)[(W + 31) / 32], int cc) {
    constexpr int NW = (W + 31) / 32;
    if constexpr (sizeof(T) == 4) {
        unsigned u = __shfl_sync(0xffffffffu, v[0], cc & 31);
        if constexpr (NW > 1) {
            const unsigned u1 = __shfl_sync(0xffffffffu, v[1], cc & 31);
            if (cc >= 32) u = u1;
        }
        return __uint_as_float(u);
    } else {
        const int wh = 2 * cc, wl = 2 * cc + 1;
        unsigned h = __shfl_sync(0xffffffffu, v[0], wh & 31);
        unsigned l = __shfl_sync(0xffffffffu, v[0], wl & 31);
        if constexpr (NW > 1) {
            const unsigned h1 = __shfl_sync(0xffffffffu, v[1], wh & 31);
            const unsigned l1 = __shfl_sync(0xffffffffu, v[1], wl & 31);
            if (wh >= 32) h = h1;
            if (wl >= 32) l = l1;
        }
        return __hiloint2double((int)h, (int)l);
    }
}

template <class T>
__device__ __forceinline__ void publish(unsigned long long* xp, size_t e, T val, unsigned tag) {
    const unsigned long long hi = (unsigned long long)tag << 32;
    if constexpr (sizeof(T) == 4) {
        st_relaxed_u64(xp + e, hi | __float_as_uint(val));
    } else {
        st_relaxed_u64(xp + 2 * e, hi | (unsigned)__double2hiint(val));
        st_relaxed_u64(xp + 2 * e + 1, hi | (unsigned)__double2loint(val));
    }
}

// Up to MAXE neighbour blocks per row (every neighbour whose value the row
// waits for) are loaded into registers, with the row's Dinv chunk and b_i,
// before the row waits; the later neighbours of the pass's first sweep are
// multiplied at once (their values predate the launch).
template <class T, int B, int WPB, int MAXE>
__global__ void __launch_bounds__(WPB * 32)
    k_gs_pass(int nitems, const int* __restrict__ items, int nsw, const int* __restrict__ row_ptr,
              const int* __restrict__ col_idx, const T* __restrict__ val, const T* __restrict__ Dinv,
              const T* __restrict__ b, T* x, unsigned long long* xp, const int* __restrict__ xptr,
              const int* __restrict__ xidx, GsSync* sync, T omega, int reverse, int64_t timeout_ns) {
    using L = WL<B, B>;
    constexpr int W = B * Packed<T>::WPV;
    constexpr int NW = (W + 31) / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = lane / L::S, sl = lane - r * L::S;
    const bool active = r < B;
    const int c0 = sl * L::CH;
    const unsigned base = __ldcg(&sync->epoch);
    bool failed = false;
    for (int w = blockIdx.x * WPB + warp; w < nitems && !failed; w += gridDim.x * WPB) {
        const int item = __ldg(items + w);
        const int i = item >> 3, s = item & 7;
        const unsigned tgt_new = base + (unsigned)s + 1u;   // this sweep's values
        const unsigned tgt_old = base + (unsigned)s;        // the previous sweep's values
        const int k0 = __ldg(row_ptr + i), k1 = __ldg(row_ptr + i + 1);
        // ---- work that does not depend on the pass's progress ----
        T bi = 0, xi = 0;
        if (active && sl == 0) {
            bi = __ldg(b + (size_t)i * B + r);
            if (s == 0) xi = __ldcg(x + (size_t)i * B + r);
        }
        T dch[L::CH];
        const T* Di = Dinv + (size_t)i * B * B;
#pragma unroll
        for (int c = 0; c < L::CH; ++c) dch[c] = (active && c0 + c < B) ? __ldg(Di + r * B + c0 + c) : T(0);
        T ech[MAXE][L::CH];
        int ej[MAXE];
#pragma unroll
        for (int q = 0; q < MAXE; ++q) ej[q] = -1;
        int ne = 0;
        T acc = 0;
        for (int k = k0; k < k1; ++k) {
            const int j = __ldg(col_idx + k);
            if (j == i) continue;
            const bool earlier = reverse ? (j > i) : (j < i);
            const T* a = val + (size_t)k * B * B;
            if (!earlier && s == 0) {
                if (active) acc += chunk_dot_coherent<T, B, B>(a, x + (size_t)j * B, r, c0);
            } else {
#pragma unroll
                for (int q = 0; q < MAXE; ++q)
                    if (q == ne) {
                        ej[q] = j;
#pragma unroll
                        for (int c = 0; c < L::CH; ++c)
                            ech[q][c] = (active && c0 + c < B) ? __ldg(a + r * B + c0 + c) : T(0);
                    }
                ++ne;
            }
        }
        // ---- neighbours of the symmetrised pattern outside the row's own
        // pattern: wait for them without reading ----
        const int e0 = __ldg(xptr + i), e1 = __ldg(xptr + i + 1);
        for (int q = e0; q < e1 && !failed; ++q) {
            const int j = __ldg(xidx + q);
            const bool earlier = reverse ? (j > i) : (j < i);
            if (!earlier && s == 0) continue;
            unsigned v[NW];
            if (!read_row<W>(xp, j, earlier ? tgt_new : tgt_old, v, sync, timeout_ns, lane)) failed = true;
        }
        if (failed) break;
        // ---- neighbours' values at the versions this sweep reads: first the
        // later neighbours and the row itself (the previous sweep's values,
        // usually published long before), then the earlier neighbours (this
        // sweep's values, the dependency chain); each group is polled as a
        // batch and summed in column order ----
        unsigned tg[MAXE + 1];
        int rw[MAXE + 1];
        unsigned later_sel = 0, earlier_sel = 0;
#pragma unroll
        for (int q = 0; q < MAXE; ++q) {
            rw[q] = ej[q] < 0 ? i : ej[q];
            const bool earlier = reverse ? (ej[q] > i) : (ej[q] < i);
            tg[q] = earlier ? tgt_new : tgt_old;
            if (ej[q] >= 0) {
                if (earlier) earlier_sel |= 1u << q;
                else later_sel |= 1u << q;
            }
        }
        rw[MAXE] = i;
        tg[MAXE] = tgt_old;
        if (s > 0) later_sel |= 1u << MAXE;
        unsigned v[MAXE + 1][NW];
        if (later_sel && !poll_rows<W, MAXE + 1>(xp, rw, tg, later_sel, v, sync, timeout_ns, lane)) failed = true;
        if (failed) break;
#pragma unroll
        for (int q = 0; q < MAXE; ++q) {
            if (!((later_sel >> q) & 1u)) continue;
#pragma unroll
            for (int c = 0; c < L::CH; ++c) {
                const int cc = c0 + c;
                const T xv = row_entry<T, W>(v[q], cc < B ? cc : 0);
                if (cc < B && active) acc += ech[q][c] * xv;
            }
        }
        if (s > 0) {
            const T xv = row_entry<T, W>(v[MAXE], active ? r : 0);
            if (active && sl == 0) xi = xv;
        }
        if (earlier_sel && !poll_rows<W, MAXE + 1>(xp, rw, tg, earlier_sel, v, sync, timeout_ns, lane)) failed = true;
        if (failed) break;
#pragma unroll
        for (int q = 0; q < MAXE; ++q) {
            if (!((earlier_sel >> q) & 1u)) continue;
#pragma unroll
            for (int c = 0; c < L::CH; ++c) {
                const int cc = c0 + c;
                const T xv = row_entry<T, W>(v[q], cc < B ? cc : 0);
                if (cc < B && active) acc += ech[q][c] * xv;
            }
        }
        if (ne > MAXE) {
            // rows with more waited-for neighbours than registers: the rest,
            // one at a time
            int seen = 0;
            for (int k = k0; k < k1 && !failed; ++k) {
                const int j = __ldg(col_idx + k);
                const bool earlier = reverse ? (j > i) : (j < i);
                if (j == i || (!earlier && s == 0)) continue;
                if (seen++ < MAXE) continue;
                unsigned v1[NW];
                if (!read_row<W>(xp, j, earlier ? tgt_new : tgt_old, v1, sync, timeout_ns, lane)) {
                    failed = true;
                    break;
                }
                const T* a = val + (size_t)k * B * B;
#pragma unroll
                for (int c = 0; c < L::CH; ++c) {
                    const int cc = c0 + c;
                    const T xv = row_entry<T, W>(v1, cc < B ? cc : 0);
                    if (cc < B && active) acc += __ldg(a + r * B + cc) * xv;
                }
            }
        }
        if (failed) break;
        acc = seg_sum<L::S>(acc);
        // t = b_i - sum_{j != i} A_ij x_j ;  x_i += omega (Dinv_i t - x_i)
        const T t = (active && sl == 0) ? bi - acc : T(0);
        T y = 0;
#pragma unroll
        for (int c = 0; c < L::CH; ++c) {
            const int cc = c0 + c;
            const T tc = __shfl_sync(0xffffffffu, t, (cc * L::S) & 31);
            if (cc < B && active) y += dch[c] * tc;
        }
        y = seg_sum<L::S>(y);
        if (active && sl == 0) {
            const T xn = xi + omega * (y - xi);
            if (s == nsw - 1) x[(size_t)i * B + r] = xn;
            publish<T>(xp, (size_t)i * B + r, xn, tgt_new);
        }
    }
    // the last CTA to finish advances the epoch past this pass
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned prev = atomicAdd(&sync->done, 1u);
        if (prev == gridDim.x - 1) {
            sync->done = 0;
            __threadfence();
            atomicExch(&sync->epoch, base + (unsigned)nsw);
        }
    }
}

// ------------------------------------------------- GS pass, tiles of rows --
// The same pass for blocks of up to 16 with most of its dependency chain
// inside SMs.  A pass is a chain of level sets (511 for one sweep of a
// 256 x 256 grid); through L2 each of its steps costs a store's way there and
// a poll's way back, about 1,900 cycles with the arithmetic.  Here kGsTile
// consecutive rows of one sweep -- a compact patch in the space-filling orders
// of the meshes -- go to one CTA, which also publishes its rows in a ring in
// shared memory; a row waits there for its own CTA's rows and only for the
// others in L2.  A step inside a CTA takes 770 cycles in FP32 (16 x 16
// blocks), 1,400 in FP64 (9 x 9; ten dependent FP64 operations).
//
// A CTA's items are dealt to its warps in level order, so every wait is for
// an item that an earlier or concurrent warp holds.  What a row needs besides
// its neighbours' values is copied to shared memory while the warp's previous
// row waits (item records three items ahead, columns two, blocks one): loading
// it row by row held a warp for 5,000 cycles, longer than the steps it has to
// spare.  Keeping the blocks in registers instead made the code long straight
// lines per neighbour slot (26.6 ms for the 256 x 256 mixed solve below).
//
// 256 x 256, 16 x 16 blocks FP32, two sweeps: 514 -> 344 us; 64 x 64, 9 x 9
// FP64: 223 -> 153 us; 15.7k triangles, 6 x 6 FP32: 447 -> 223 us.  Solve of
// the 256 x 256 grid 33.0 -> 23.5 ms.
//
// Two consecutive rows may be of different tiles and a tile's rows of
// different levels: the ring's slots carry the item's number in the CTA, and a
// reader that finds its slot taken by a later item reads the row from L2.  The
// ring's length is a multiple of the warp count, so that all items of a slot
// belong to one warp and are written in order: an older item's tag put over a
// newer one would leave the newer one's readers waiting.
constexpr int kGsRing = 64;   // most slots

// Rows that go to one CTA: 4 x 4 patches, whose diagonals have a row for each
// of the SM's warp schedulers (8 x 8: 858 us instead of 449 for the 256 x 256
// pass, both before the copies to shared memory; 2 x 2: 382 against 344 with
// them).  FP64 blocks of 16 are bound by the SM's FP64
// pipes, which a patch's rows share: 2 x 2 (219 us against 233 for 64 x 64).
template <class T, int B>
constexpr int kGsTile = sizeof(T) == 8 && B == 16 ? 4 : 16;

__device__ __forceinline__ void lds_pair(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.cta.shared.v2.b64 {%0, %1}, [%2];"
                 : "=l"(a), "=l"(b)
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ unsigned long long lds_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.cta.shared.b64 %0, [%1];" : "=l"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
__device__ __forceinline__ void sts_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.cta.shared.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "l"(v) : "memory");
}

// The lane's CH entries, starting at c0, of a row published in shared memory
// with `tag`; polls until they carry it.  Warp-uniform result: 0 read, 1 the
// slot has passed to a later row (the value is in global memory), 2 gave up.
template <class T, int B, int CH>
__device__ __forceinline__ int poll_local(const unsigned long long* row, int c0, unsigned tag, T (&xv)[CH],
                                          GsSync* sync, int64_t timeout_ns) {
    constexpr int WPV = Packed<T>::WPV, NW = CH * WPV;
    constexpr bool FULL = WL<B, B>::S * CH == B;
    const unsigned long long* p = row + c0 * WPV;
    uint64_t t0 = 0;
    unsigned it = 0;
    while (true) {
        unsigned long long u[NW];
        if constexpr (NW % 2 == 0) {
#pragma unroll
            for (int w = 0; w < NW; w += 2) lds_pair(p + w, u[w], u[w + 1]);
        } else {
#pragma unroll
            for (int w = 0; w < NW; ++w) u[w] = lds_word(p + w);
        }
        unsigned diff[2] = {0u, 0u};
#pragma unroll
        for (int w = 0; w < NW; ++w)
            if (FULL || c0 + w / WPV < B) diff[w & 1] |= (unsigned)(u[w] >> 32) ^ tag;
        if (__all_sync(0xffffffffu, (diff[0] | diff[1]) == 0)) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                if constexpr (sizeof(T) == 4) xv[c] = __uint_as_float((unsigned)u[c]);
                else xv[c] = __hiloint2double((int)(unsigned)u[2 * c], (int)(unsigned)u[2 * c + 1]);
            }
            return 0;
        }
        const bool later = (FULL || c0 < B) && (int)((unsigned)(u[0] >> 32) - tag) > 0;
        if (__any_sync(0xffffffffu, later)) return 1;
        if ((++it & 255u) == 0) {
            if (it == 256u) t0 = globaltimer_ns();
            bool stop = *(volatile unsigned*)&sync->err != 0;
            if (!stop && (int64_t)(globaltimer_ns() - t0) > timeout_ns) {
                atomicOr(&sync->err, 1u);
                stop = true;
            }
            if (__any_sync(0xffffffffu, stop)) return 2;
        }
    }
}

// Copies nbytes from global to shared memory by one warp (asynchronous, CP
// bytes per lane and step; both sides CP-aligned).
template <int CP>
__device__ __forceinline__ void warp_copy(void* dst, const void* src, int nbytes, int lane) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const char* g = reinterpret_cast<const char*>(src);
    for (int o = lane * CP; o < nbytes; o += 32 * CP) {
        if constexpr (CP == 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + o), "l"(g + o) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + o), "l"(g + o), "n"(CP) : "memory");
    }
}

// Sizes of the tile kernel: blocks of a row kept in shared memory (two rows
// per warp, the one in work and the next), warps per CTA.
template <class T, int B>
struct GsTile {
    using L = WL<B, B>;
    static constexpr int BB = B * B;
    static constexpr int WPV = Packed<T>::WPV, W = B * WPV;
    static constexpr int XL = L::S * L::CH;                        // entries of a staged row
    static constexpr int LDW = (XL * WPV + 1) / 2 * 2;             // words of a ring row
    static constexpr int MAXB = B == 16 ? 5 : 8;
    static constexpr int NR = 4;                                   // rows gathered at a time
    static constexpr int KW = (NR * W + 31) / 32;
    static constexpr int BUF = ((MAXB + 1) * BB * (int)sizeof(T) + 15) / 16 * 16;
    static constexpr int STAGE = (NR * XL * (int)sizeof(T) + 15) / 16 * 16;
    static constexpr int PER_WARP = 2 * BUF + STAGE;
    static constexpr int RMAX = kGsRing * LDW * 8;
    static constexpr int WPB = RMAX + 16 * PER_WARP <= 220 * 1024 ? 16 : (RMAX + 12 * PER_WARP <= 220 * 1024 ? 12 : 8);
    static constexpr unsigned SLOTS = kGsRing / WPB * WPB;
    static_assert(SLOTS > 0 && SLOTS % WPB == 0, "one warp per ring slot");
    static constexpr int RING = (int)SLOTS * LDW * 8;
    static constexpr int SMEM = RING + WPB * PER_WARP;
    static constexpr int CP = BB * (int)sizeof(T) % 16 == 0 ? 16 : (BB * (int)sizeof(T) % 8 == 0 ? 8 : 4);
};

// Gathers nr <= NR rows into the warp's stage: row q is jl's lane t_q (byte q
// of tp; 0xff: row i itself).  plain: from the vector x; else from the packed
// rows, once every word carries an epoch at or after tgt.  Warp-uniform
// result: false if the wait ran out or another waiter gave up.
template <class T, int B>
__device__ __forceinline__ bool gather_rows(const unsigned long long* xp, const T* x, bool plain, unsigned tgt,
                                            unsigned tp, int nr, int i, int jl, T* stage, GsSync* sync,
                                            int64_t timeout_ns, int lane) {
    using G = GsTile<T, B>;
    constexpr int KW = G::KW, W = G::W, WPV = G::WPV;
    size_t at[KW];
    unsigned v[KW];
#pragma unroll
    for (int k = 0; k < KW; ++k) {
        const int w = lane + 32 * k, q = w / W;
        const int t = (int)((tp >> (8 * (q & 3))) & 0xffu);
        const int j = __shfl_sync(0xffffffffu, jl, t & 31);
        at[k] = (size_t)(t == 0xff ? i : j) * W + (w - q * W);
        v[k] = 0;
    }
    const int n = nr * W;
    if (plain) {
        // hi and lo halves of an FP64 entry are in the packed order
#pragma unroll
        for (int k = 0; k < KW; ++k)
            if (lane + 32 * k < n) v[k] = __ldcg(reinterpret_cast<const unsigned*>(x) + (WPV == 2 ? at[k] ^ 1u : at[k]));
    } else {
        uint64_t t0 = 0;
        unsigned it = 0;
        while (true) {
            bool ok = true;
            unsigned long long u[KW];
#pragma unroll
            for (int k = 0; k < KW; ++k) u[k] = lane + 32 * k < n ? ld_relaxed_u64(xp + at[k]) : (unsigned long long)tgt << 32;
#pragma unroll
            for (int k = 0; k < KW; ++k) {
                v[k] = (unsigned)u[k];
                ok = ok && (int)((unsigned)(u[k] >> 32) - tgt) >= 0;
            }
            if (__all_sync(0xffffffffu, ok)) break;
            if ((++it & 15u) == 0) {
                if (it == 16u) t0 = globaltimer_ns();
                bool stop = *(volatile unsigned*)&sync->err != 0;
                if (!stop && (int64_t)(globaltimer_ns() - t0) > timeout_ns) {
                    atomicOr(&sync->err, 1u);
                    stop = true;
                }
                if (__any_sync(0xffffffffu, stop)) return false;
            }
        }
    }
    __syncwarp();
    unsigned* st = reinterpret_cast<unsigned*>(stage);
#pragma unroll
    for (int k = 0; k < KW; ++k) {
        const int w = lane + 32 * k, q = w / W, e = w - q * W;
        if (w < n) st[q * (G::XL * WPV) + (WPV == 2 ? e ^ 1 : e)] = v[k];
    }
    __syncwarp();
    return true;
}

// the lane's part of a block: columns c0 .. of row rr (zero past the last)
template <class T, int B>
__device__ __forceinline__ void block_part(const T* a, int rr, int c0, T (&v)[WL<B, B>::CH]) {
    constexpr int CH = WL<B, B>::CH;
    constexpr bool FULL = WL<B, B>::S * CH == B;
#pragma unroll
    for (int c = 0; c < CH; ++c) v[c] = FULL || c0 + c < B ? a[rr * B + c0 + c] : T(0);
}

template <class T, int B>
__global__ void __launch_bounds__(GsTile<T, B>::WPB * 32, 1)
    k_gs_tiles(const int* __restrict__ cta_ptr, const int4* __restrict__ items, const signed char* __restrict__ ltag,
               int64_t nnzb, int nsw, const int* __restrict__ col_idx, const T* __restrict__ val,
               const T* __restrict__ Dinv, const T* __restrict__ b, T* x, unsigned long long* xp,
               const int* __restrict__ xptr, const int* __restrict__ xidx, GsSync* sync, T omega, int reverse,
               int64_t timeout_ns) {
    using G = GsTile<T, B>;
    using L = WL<B, B>;
    constexpr int CH = L::CH, BB = G::BB, WPV = G::WPV, WPB = G::WPB;
    constexpr bool FULL = L::S * CH == B;
    constexpr unsigned ALL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned long long* ring = reinterpret_cast<unsigned long long*>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* mine = smem + G::RING + warp * G::PER_WARP;
    T* stage = reinterpret_cast<T*>(mine + 2 * G::BUF);
    const int r = lane / L::S, sl = lane - r * L::S;
    const bool active = B * L::S == 32 || r < B;
    const bool first = active && sl == 0;
    const int rr = active ? r : 0;
    const int c0 = sl * CH;
    for (int q = threadIdx.x; q < (int)G::SLOTS * G::LDW; q += WPB * 32) ring[q] = 0;
    for (int q = lane; q < G::NR * G::XL; q += 32) stage[q] = T(0);
    const unsigned base = __ldcg(&sync->epoch);
    __syncthreads();
    const int w0 = __ldg(cta_ptr + blockIdx.x), w1 = __ldg(cta_ptr + blockIdx.x + 1);
    // records are loaded three items ahead, columns two, blocks one
    const int4 none = make_int4(-1, 0, 0, 0);
    auto record = [&](int w) { return w < w1 ? __ldg(items + w) : none; };
    auto columns = [&](const int4& it, int& jl, int& tl) {
        jl = lane < it.z ? __ldg(col_idx + it.y + lane) : -1;
        tl = lane < it.z ? (int)__ldg(ltag + (it.x & 7) * nnzb + it.y + lane) : 0;
    };
    T bn = 0, xn0 = 0;
    auto blocks = [&](const int4& it, int buf) {
        if (it.x < 0) return;
        T* d = reinterpret_cast<T*>(mine + buf * G::BUF);
        const int i = it.x >> 3;
        warp_copy<G::CP>(d, Dinv + (size_t)i * BB, BB * (int)sizeof(T), lane);
        warp_copy<G::CP>(d + BB, val + (size_t)it.y * BB, min(it.z, G::MAXB) * BB * (int)sizeof(T), lane);
    };
    auto vectors = [&](const int4& it) {
        bn = xn0 = 0;
        if (first && it.x >= 0) {
            const size_t o = (size_t)(it.x >> 3) * B + r;
            bn = __ldg(b + o);
            if ((it.x & 7) == 0) xn0 = __ldcg(x + o);
        }
    };
    int4 it = record(w0 + warp), it1 = record(w0 + warp + WPB), it2 = record(w0 + warp + 2 * WPB);
    int jl, tl, jl1, tl1;
    columns(it, jl, tl);
    columns(it1, jl1, tl1);
    blocks(it, 0);
    vectors(it);
    asm volatile("cp.async.commit_group;" ::: "memory");
    int pb = 0;
    for (int w = w0 + warp; w < w1; w += WPB, pb ^= 1) {
        const int i = it.x >> 3, s = it.x & 7, k0 = it.y, nk = it.z;
        const unsigned tgt_new = base + (unsigned)s + 1u;   // this sweep's values
        const unsigned tgt_old = base + (unsigned)s;        // the previous sweep's values
        T acc = bn, xi = xn0;
        __syncwarp();
        blocks(it1, pb ^ 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        vectors(it1);
        int jl2, tl2;
        columns(it2, jl2, tl2);
        const int4 it3 = record(w + 3 * WPB);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const T* buf = reinterpret_cast<const T*>(mine + pb * G::BUF);
        // ---- work that does not depend on the pass's progress ----
        T dch[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) dch[c] = active && (FULL || c0 + c < B) ? buf[rr * B + c0 + c] : T(0);
        const unsigned nb = __ballot_sync(ALL, lane < nk && jl != i);
        const unsigned early = __ballot_sync(ALL, reverse ? jl > i : jl < i) & nb;
        unsigned own = __ballot_sync(ALL, tl != 0) & early;
        bool failed = false;
        // the blocks of the rows in sel times their values at version tgt,
        // up to NR rows per L2 round trip, in column order
        auto others = [&](unsigned sel, bool self, bool plain, unsigned tgt) {
            while ((sel || self) && !failed) {
                unsigned tp = 0;
                int nr = 0;
                if (self) {
                    tp = 0xffu;
                    nr = 1;
                }
                while (nr < G::NR && sel) {
                    tp |= (unsigned)(__ffs(sel) - 1) << (8 * nr++);
                    sel &= sel - 1;
                }
                if (!gather_rows<T, B>(xp, x, plain, tgt, tp, nr, i, jl, stage, sync, timeout_ns, lane)) {
                    failed = true;
                    return;
                }
#pragma unroll 1
                for (int q = 0; q < nr; ++q) {
                    const int t = (int)((tp >> (8 * q)) & 0xffu);
                    if (t == 0xff) {
                        if (first) xi = stage[r];
                        continue;
                    }
                    T av[CH];
                    if (t < G::MAXB) block_part<T, B>(buf + (t + 1) * BB, rr, c0, av);
                    else block_part<T, B>(val + (size_t)(k0 + t) * BB, rr, c0, av);
#pragma unroll
                    for (int c = 0; c < CH; ++c) acc = fma(-av[c], stage[q * G::XL + c0 + c], acc);
                }
                self = false;
            }
        };
        // neighbours of the symmetrised pattern outside the row's own
        // pattern: waited for without reading
        if (it.w) {
            const int e0 = __ldg(xptr + i), e1 = __ldg(xptr + i + 1);
            for (int q = e0; q < e1 && !failed; ++q) {
                const int j = __ldg(xidx + q);
                const bool earlier = reverse ? (j > i) : (j < i);
                if (!earlier && s == 0) continue;
                if (!gather_rows<T, B>(xp, x, false, earlier ? tgt_new : tgt_old, 0u, 1, i, j, stage, sync, timeout_ns,
                                       lane))
                    failed = true;
            }
        }
        // blocks past the 32 columns held by the lanes, one at a time
        for (int t = 32; t < nk && !failed; ++t) {
            const int j = __ldg(col_idx + k0 + t);
            if (j == i) continue;
            const bool earlier = reverse ? (j > i) : (j < i);
            if (!gather_rows<T, B>(xp, x, !earlier && s == 0, earlier ? tgt_new : tgt_old, 0u, 1, i, j, stage, sync,
                                   timeout_ns, lane)) {
                failed = true;
                break;
            }
            T av[CH];
            block_part<T, B>(val + (size_t)(k0 + t) * BB, rr, c0, av);
#pragma unroll
            for (int c = 0; c < CH; ++c) acc = fma(-av[c], stage[c0 + c], acc);
        }
        // later neighbours and the row itself (the previous sweep's values),
        // then the earlier neighbours of other CTAs, then this CTA's
        others(nb & ~early, s > 0, s == 0, tgt_old);
        const T xs = (T(1) - omega) * xi;
        others(early & ~own, false, false, tgt_new);
#pragma unroll 1
        while (own && !failed) {
            const int t = __ffs(own) - 1;
            own &= own - 1;
            const unsigned tag = (unsigned)(w - w0 + 1 - __shfl_sync(ALL, tl, t));
            T av[CH], xv[CH];
            if (t < G::MAXB) block_part<T, B>(buf + (t + 1) * BB, rr, c0, av);
            else block_part<T, B>(val + (size_t)(k0 + t) * BB, rr, c0, av);
            const int st = poll_local<T, B, CH>(ring + ((tag - 1u) % G::SLOTS) * G::LDW, c0, tag, xv, sync,
                                                timeout_ns);
            if (st == 0) {
#pragma unroll
                for (int c = 0; c < CH; ++c) acc = fma(-av[c], xv[c], acc);
            } else if (st == 1) {
                others(1u << t, false, false, tgt_new);
            } else {
                failed = true;
            }
        }
        if (failed) break;
        // x_i + omega (Dinv_i t - x_i), t = b_i - sum_{j != i} A_ij x_j
        const T tt = seg_sum<L::S>(acc);
        T y = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const T tc = __shfl_sync(ALL, tt, ((c0 + c) * L::S) & 31);
            y = fma(dch[c], FULL || c0 + c < B ? tc : T(0), y);
        }
        const T xn = fma(omega, seg_sum<L::S>(y), xs);
        if (first) {
            const unsigned seq = (unsigned)(w - w0);
            unsigned long long* so = ring + (seq % G::SLOTS) * G::LDW + r * WPV;
            const unsigned long long hi = (unsigned long long)(seq + 1u) << 32;
            if constexpr (sizeof(T) == 4) {
                sts_word(so, hi | __float_as_uint(xn));
            } else {
                sts_word(so, hi | (unsigned)__double2hiint(xn));
                sts_word(so + 1, hi | (unsigned)__double2loint(xn));
            }
            publish<T>(xp, (size_t)i * B + r, xn, tgt_new);
            if (s == nsw - 1) x[(size_t)i * B + r] = xn;
        }
        it = it1; it1 = it2; it2 = it3;
        jl = jl1; tl = tl1; jl1 = jl2; tl1 = tl2;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // the last CTA to finish advances the epoch past this pass
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned prev = atomicAdd(&sync->done, 1u);
        if (prev == gridDim.x - 1) {
            sync->done = 0;
            __threadfence();
            atomicExch(&sync->epoch, base + (unsigned)nsw);
        }
    }
}

// ------------------------------------------------------------ Jacobi sweep --
// x_out_i = x_in_i + omega * Dinv_i (b_i - sum_j A_ij x_in_j)
//
// xzero: x_in is the zero vector (the first sweep of a V-cycle level), so
// the kernels neither read A nor x_in.  The product of A with zeros is +0 in
// every lane and b_i - (+0) = b_i, so the sweep still gives the full
// sweep's values bit for bit.
template <class T, int B, int WPB>
__global__ void __launch_bounds__(WPB * 32, 2)
    k_jacobi(int n, const int* __restrict__ row_ptr, const int* __restrict__ col_idx, const T* __restrict__ val,
             const T* __restrict__ Dinv, const T* __restrict__ b, const T* __restrict__ xin, T* __restrict__ xout,
             T omega, bool xzero) {
    using L = WL<B, B>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = lane / L::S, s = lane - r * L::S;
    const bool active = r < B;
    const int c0 = s * L::CH;
    for (int i = blockIdx.x * WPB + warp; i < n; i += gridDim.x * WPB) {
        // the row's own data is independent of the product: issue it first
        T bi = 0, xi = 0;
        if (active && s == 0) {
            bi = __ldg(b + (size_t)i * B + r);
            if (!xzero) xi = __ldg(xin + (size_t)i * B + r);
        }
        T dch[L::CH];
        const T* Di = Dinv + (size_t)i * B * B;
#pragma unroll
        for (int c = 0; c < L::CH; ++c) dch[c] = (active && c0 + c < B) ? __ldg(Di + r * B + c0 + c) : T(0);
        T acc = 0;
        if (!xzero) {
            const int k0 = __ldg(row_ptr + i), k1 = __ldg(row_ptr + i + 1);
            acc = row_product<T, B, B>(col_idx, val, nullptr, xin, k0, k1, r, c0, active, lane);
            acc = seg_sum<L::S>(acc);
        }
        const T t = (active && s == 0) ? bi - acc : T(0);
        T y = 0;
#pragma unroll
        for (int c = 0; c < L::CH; ++c) {
            const int cc = c0 + c;
            const T tc = __shfl_sync(0xffffffffu, t, (cc * L::S) & 31);
            if (cc < B && active) y += dch[c] * tc;
        }
        y = seg_sum<L::S>(y);
        if (active && s == 0) xout[(size_t)i * B + r] = xi + omega * y;
    }
}

// Small blocks (B <= 10): 32 / B block rows per warp, one lane per block
// column for the product (cols_accumulate, rows_reduce), then lane (g, r)
// holds t_r = b_r - (A x_in)_r and applies row r of Dinv with t's entries
// shuffled within the group.  The row loop is warp-uniform so every lane
// takes part in the shuffles and the shared-memory reduction.
template <class T, class VT, int B, int MAXB, int MINB>
__global__ void __launch_bounds__(256, MINB)
    k_jacobi_rows(int n, const int* __restrict__ row_ptr, const int* __restrict__ col_idx, const VT* __restrict__ val,
                  const float* __restrict__ scl, const T* __restrict__ Dinv, const T* __restrict__ b,
                  const T* __restrict__ xin, T* __restrict__ xout, T omega, bool xzero) {
    using R = Rows<B>;
    __shared__ T sr[8 * R::SM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / R::S, c = lane - g * R::S;
    T* s = sr + warp * R::SM;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int base = (blockIdx.x * (blockDim.x >> 5) + warp) * R::G; base < n; base += nw * R::G) {
        const int row = base + g;
        const bool valid = g < R::G && row < n;
        const size_t o = (size_t)row * B + c;
        T acc[B];
#pragma unroll
        for (int r = 0; r < B; ++r) acc[r] = 0;
        T bi = 0, xi = 0;
        if (valid) {
            bi = __ldg(b + o);
            if (!xzero) {
                xi = __ldg(xin + o);
                cols_accumulate<T, VT, B, B, MAXB>(col_idx, val, scl, nullptr, xin, __ldg(row_ptr + row),
                                                   __ldg(row_ptr + row + 1), c, acc);
            }
        }
        const T t = bi - rows_reduce<T, B, B>(acc, s, g, c, g < R::G);
        // lane (g, c) now holds t_c; y_c = sum_k Dinv(c, k) t_k
        const T* Di = Dinv + ((size_t)row * B + c) * B;
        const int src = (g < R::G ? g : 0) * B;
        T y = 0;
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const T tk = __shfl_sync(0xffffffffu, t, src + k);
            if (valid) y = fma(__ldg(Di + k), tk, y);
        }
        if (valid) xout[o] = xi + omega * y;
    }
}

template <class T, int B, class VT = T>
static void launch_jacobi_rows(mgldg_ctx* ctx, const mgldg_bsr* A, const VT* vals, const T* Dinv, const T* b,
                               const T* xin, T* xout, T omega, bool xzero, const float* scl = nullptr) {
    // FP32 blocks of 6, 9 and 10: blocks in flight given up for four CTAs an SM:
    // 39.9 -> 33.1 us at 6 x 6, 175k rows; 28.5 -> 27.4 at 9 x 9, 40.0k rows;
    // 35.5 -> 29.6 at 10 x 10, 43.5k rows.  FP64 stays with the registers the
    // compiler takes (9 x 9: 93 us against 97, 10 x 10: 94 against 103).
    constexpr bool F4 = sizeof(T) == 4 && (B == 6 || B == 9 || B == 10);
    constexpr int MINB = F4 ? 4 : 0;
    constexpr int MAXB = F4 ? (B == 10 ? 2 : 3) : ((sizeof(T) == 4 || B <= 4) ? 4 : 2);
    const int rows_per_cta = 8 * Rows<B>::G;
    const int grid = std::max(1, std::min((A->nbr + rows_per_cta - 1) / rows_per_cta, ctx->sm_count * 8));
    {
        Launch L(ctx, MGLDG_K_JACOBI);
        k_jacobi_rows<T, VT, B, MAXB, MINB><<<grid, 256, 0, ctx->stream>>>(A->nbr, A->row_ptr, A->col_idx, vals, scl,
                                                                           Dinv, b, xin, xout, omega, xzero);
    }
    check_launch();
}

// -------------------------------------------------------------- scheduling --
// Level sets of one sweep direction (dir 0: rows ascending, 1: descending).
// A row depends on its earlier neighbours in the symmetrised pattern (an
// entry A_ij or A_ji); level(i) = 1 + max level of those, 0 if none.
// Outputs the level of every row, the wait lists and the rows in level order.
void gs_levels_host(int n, const int* row_ptr, const int* col_idx, int dir, std::vector<int>& lev,
                    std::vector<int>& wp, std::vector<int>& wi, std::vector<int>& order, int& nlev) {
    std::vector<std::vector<int>> nb(n);
    for (int i = 0; i < n; ++i)
        for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
            int j = col_idx[k];
            if (j == i || j < 0 || j >= n) continue;
            nb[i].push_back(j);
            nb[j].push_back(i);
        }
    for (auto& v : nb) {
        std::sort(v.begin(), v.end());
        v.erase(std::unique(v.begin(), v.end()), v.end());
    }
    lev.assign(n, 0);
    wp.assign(n + 1, 0);
    wi.clear();
    int maxlev = 0;
    for (int t = 0; t < n; ++t) {
        const int i = dir == 0 ? t : n - 1 - t;
        int l = 0;
        for (int j : nb[i]) {
            const bool earlier = dir == 0 ? (j < i) : (j > i);
            if (earlier) l = std::max(l, lev[j] + 1);
        }
        lev[i] = l;
        maxlev = std::max(maxlev, l);
    }
    for (int i = 0; i < n; ++i) {
        for (int j : nb[i]) {
            const bool earlier = dir == 0 ? (j < i) : (j > i);
            if (earlier) wi.push_back(j);
        }
        wp[i + 1] = (int)wi.size();
    }
    // counting sort by level; ascending rows inside a level for the forward
    // sweep, descending for the reverse sweep
    std::vector<int> cnt(maxlev + 2, 0);
    order.assign(n, 0);
    for (int i = 0; i < n; ++i) cnt[lev[i] + 1]++;
    for (int l = 0; l <= maxlev; ++l) cnt[l + 1] += cnt[l];
    for (int t = 0; t < n; ++t) {
        const int i = dir == 0 ? t : n - 1 - t;
        order[cnt[lev[i]]++] = i;
    }
    nlev = n ? maxlev + 1 : 0;
}

// neighbours of every row in the symmetrised pattern, row i's at idx[ptr[i]] ..
// idx[ptr[i + 1] - 1] in ascending order: its own columns merged with the rows
// that have it as a column (one pass over the pattern each)
static void symmetrised_neighbours(int n, const int* row_ptr, const int* col_idx, std::vector<int>& ptr,
                                   std::vector<int>& idx) {
    std::vector<int> tp(n + 1, 0);
    auto other = [&](int i, int j) { return j != i && j >= 0 && j < n; };
    int64_t nnz = 0;
    for (int i = 0; i < n; ++i)
        for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k)
            if (other(i, col_idx[k])) tp[col_idx[k] + 1]++, ++nnz;
    for (int i = 0; i < n; ++i) tp[i + 1] += tp[i];
    std::vector<int> ti(nnz), at(tp.begin(), tp.end() - 1);
    for (int i = 0; i < n; ++i)
        for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k)
            if (other(i, col_idx[k])) ti[at[col_idx[k]]++] = i;
    ptr.assign(n + 1, 0);
    idx.clear();
    idx.reserve(nnz + nnz / 8);
    std::vector<int> own;
    for (int i = 0; i < n; ++i) {
        own.clear();
        for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k)
            if (other(i, col_idx[k])) own.push_back(col_idx[k]);
        if (!std::is_sorted(own.begin(), own.end())) std::sort(own.begin(), own.end());
        const int *p = own.data(), *pe = p + own.size(), *q = ti.data() + tp[i], *qe = ti.data() + tp[i + 1];
        int last = -1;
        while (p < pe || q < qe) {
            const int j = q == qe || (p < pe && *p <= *q) ? *p++ : *q++;
            if (j != last) idx.push_back(j);
            last = j;
        }
        ptr[i + 1] = (int)idx.size();
    }
}

void sched_build(mgldg_ctx* ctx, const mgldg_bsr* A, Sched& S) {
    const int n = A->nbr;
    S.n = n;
    S.A = A;
    symmetrised_neighbours(n, A->h_row_ptr.data(), A->h_col_idx.data(), S.nbp, S.nbi);
    // neighbours j of i with A_ji stored but not A_ij: waited for, not read
    std::vector<int> xp_(n + 1, 0), xi;
    for (int i = 0; i < n; ++i) {
        const int* c0 = A->h_col_idx.data() + A->h_row_ptr[i];
        const int* c1 = A->h_col_idx.data() + A->h_row_ptr[i + 1];
        for (int q = S.nbp[i]; q < S.nbp[i + 1]; ++q)
            if (std::find(c0, c1, S.nbi[q]) == c1) xi.push_back(S.nbi[q]);
        xp_[i + 1] = (int)xi.size();
    }
    S.xptr = dalloc<int>(n + 1);
    S.xidx = dalloc<int>(std::max<size_t>(1, xi.size()));
    upload(ctx, S.xptr, xp_.data(), xp_.size());
    if (!xi.empty()) upload(ctx, S.xidx, xi.data(), xi.size());
    S.sync = dalloc<GsSync>(1);
    MG_CHECK_CUDA(cudaMemsetAsync(S.sync, 0, sizeof(GsSync), ctx->stream));
    sync(ctx);
}

// Level sets of nsw consecutive sweeps: (s, i) follows (s, j) for earlier
// neighbours j, (s - 1, j) for later neighbours j and (s - 1, i).
// lev[s * n + i] is the level of (s, i); returns the number of levels.
static int gs_pass_levels_host(int n, const std::vector<int>& nbp, const std::vector<int>& nbi, int dir, int nsw,
                               std::vector<int>& lev) {
    lev.assign((size_t)nsw * n, 0);
    int maxlev = -1;
    for (int s = 0; s < nsw; ++s) {
        int* cur = lev.data() + (size_t)s * n;
        const int* old = s > 0 ? cur - n : nullptr;
        for (int t = 0; t < n; ++t) {
            const int i = dir == 0 ? t : n - 1 - t;
            int l = old ? old[i] + 1 : 0;
            for (int q = nbp[i]; q < nbp[i + 1]; ++q) {
                const int j = nbi[q];
                const bool earlier = dir == 0 ? (j < i) : (j > i);
                if (earlier) l = std::max(l, cur[j] + 1);
                else if (old) l = std::max(l, old[j] + 1);
            }
            cur[i] = l;
            maxlev = std::max(maxlev, l);
        }
    }
    return maxlev + 1;
}

// records and tags of a tile pass, one thread per (sweep, row): loc is the
// item's number in its CTA's list, owner the CTA of a (sweep, tile)
__global__ void __launch_bounds__(256) k_gs_plan(int n, int nsw, int shift, int ng, int reverse, int slots,
                                                 int64_t nnzb, const int* __restrict__ row_ptr,
                                                 const int* __restrict__ col_idx, const int* __restrict__ xptr,
                                                 const int* __restrict__ cta_ptr, const int* __restrict__ owner,
                                                 const int* __restrict__ loc, int4* __restrict__ rec,
                                                 signed char* __restrict__ ltag) {
    const int64_t total = (int64_t)nsw * n;
    for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < total; t += (int64_t)gridDim.x * 256) {
        const int s = (int)(t / n), i = (int)(t - (int64_t)s * n);
        const int *os = owner + (size_t)s * ng, *ls = loc + (size_t)s * n;
        const int o = __ldg(os + (i >> shift)), seq = __ldg(ls + i);
        const int k0 = __ldg(row_ptr + i), k1 = __ldg(row_ptr + i + 1);
        rec[(size_t)__ldg(cta_ptr + o) + seq] = make_int4((i << 3) | s, k0, k1 - k0, __ldg(xptr + i + 1) > __ldg(xptr + i));
        for (int k = k0; k < k1; ++k) {
            const int j = __ldg(col_idx + k);
            int d = 0;
            if ((reverse ? j > i : j < i) && __ldg(os + (j >> shift)) == o) d = seq - __ldg(ls + j);
            ltag[s * nnzb + k] = (signed char)(d > 0 && d <= slots ? d : 0);
        }
    }
}

static void pass_build(mgldg_ctx* ctx, Sched& S, int dir, int nsw, int grid, int tile, int slots, GsPass& P) {
    const int n = S.n;
    MG_REQUIRE(n < (1 << 28) && nsw >= 1 && nsw <= 7, MGLDG_ERR_UNSUPPORTED, "Gauss-Seidel pass too large");
    std::vector<int> lev;
    const int maxlev = gs_pass_levels_host(n, S.nbp, S.nbi, dir, nsw, lev) - 1;
    // counting sort by level; inside a level by sweep, then in sweep order
    std::vector<int> cnt(maxlev + 2, 0);
    for (int l : lev) cnt[l + 1]++;
    for (int l = 0; l <= maxlev; ++l) cnt[l + 1] += cnt[l];
    std::vector<int> items((size_t)nsw * n);
    for (int s = 0; s < nsw; ++s)
        for (int t = 0; t < n; ++t) {
            const int i = dir == 0 ? t : n - 1 - t;
            items[cnt[lev[(size_t)s * n + i]]++] = (i << 3) | s;
        }
    P.nsw = nsw;
    P.dir = dir;
    P.grid = grid;
    P.tile = tile;
    P.nitems = nsw * n;
    P.depth = n ? maxlev + 1 : 0;
    P.slots = slots;
    if (grid > 0) {
        // groups of consecutive rows, one sweep each, go to the CTAs in the
        // order in which the pass reaches them; the records and tags follow
        // from that on the GPU (first V-cycle of a hierarchy with 16,384 rows of
        // 4 x 4, FP32: 1.04 ms with them made and uploaded here, 0.61 ms)
        const int shift = __builtin_ctz((unsigned)tile), ng = (n + tile - 1) >> shift;   // a power of two
        const size_t nrec = std::max<size_t>(1, items.size()), nown = (size_t)nsw * ng;
        const size_t ntag = (size_t)nsw * S.A->h_row_ptr[n];
        // first items of the CTAs, owners, numbers in the CTAs' lists
        std::vector<int> tab(grid + 1 + nown + items.size(), 0);
        int *cta = tab.data(), *owner = cta + grid + 1, *loc = owner + nown;
        std::fill(owner, owner + nown, -1);
        int next = 0;
        for (int it : items) {
            const int i = it >> 3, s = it & 7;
            int& o = owner[(size_t)s * ng + (i >> shift)];
            if (o < 0) {
                o = next;
                next = next + 1 < grid ? next + 1 : 0;
            }
            loc[(size_t)s * n + i] = cta[o + 1]++;
        }
        for (int c = 0; c < grid; ++c) cta[c + 1] += cta[c];
        P.items = dalloc<int>(4 * nrec + tab.size() + (ntag + 3) / 4);
        P.rec = reinterpret_cast<int4*>(P.items);
        P.cta_ptr = P.items + 4 * nrec;
        P.ltag = reinterpret_cast<signed char*>(P.cta_ptr + tab.size());
        upload(ctx, P.cta_ptr, tab.data(), tab.size());
        if (n) {
            const int g = (int)std::min<int64_t>(((int64_t)nsw * n + 255) / 256, ctx->sm_count * 16);
            Launch L(ctx, MGLDG_K_SETUP);
            k_gs_plan<<<g, 256, 0, ctx->stream>>>(n, nsw, shift, ng, dir, slots, (int64_t)S.A->h_row_ptr[n],
                                                  S.A->row_ptr, S.A->col_idx, S.xptr, P.cta_ptr, P.cta_ptr + grid + 1,
                                                  P.cta_ptr + grid + 1 + nown, P.rec, P.ltag);
        }
        check_launch();
        sync(ctx);
        return;
    }
    P.items = dalloc<int>(std::max<size_t>(1, items.size()));
    upload(ctx, P.items, items.data(), items.size());
    sync(ctx);
}

static void pass_free(GsPass& P) {
    dfree(P.items);
}

static GsPass& get_pass(mgldg_ctx* ctx, Sched& S, int dir, int nsw, int grid, int tile, int slots) {
    for (auto& P : S.passes)
        if (P.dir == dir && P.nsw == nsw && P.grid == grid && P.tile == tile && P.slots == slots)
            return P;
    GsPass P;
    try {
        pass_build(ctx, S, dir, nsw, grid, tile, slots, P);
    } catch (...) {
        pass_free(P);
        throw;
    }
    S.passes.push_back(P);
    return S.passes.back();
}

void sched_free(Sched& S) {
    for (auto& P : S.passes) pass_free(P);
    S.passes.clear();
    dfree(S.xptr);
    dfree(S.xidx);
    dfree(S.xp);
    dfree(S.sync);
    S.xptr = S.xidx = nullptr;
    S.xp = nullptr;
    S.sync = nullptr;
}

int gs_take_error(mgldg_ctx* ctx, Sched& S) {
    if (!S.sync) return 0;
    GsSync h;
    download(ctx, &h, S.sync, 1);
    sync(ctx);
    if (h.err) {
        // clear the error word; epochs stay monotone, so the next pass's
        // targets exceed every stale word and the schedule stays valid
        unsigned zero = 0;
        upload(ctx, &S.sync->err, &zero, 1);
        sync(ctx);
        return 1;
    }
    return 0;
}

// the published rows of a schedule, `words` 64-bit words each
static void packed_rows(mgldg_ctx* ctx, Sched& S, int words) {
    if (!S.xp || S.words_per_row != words) {
        dfree(S.xp);
        S.xp = nullptr;
        S.xp = dalloc<unsigned long long>((size_t)std::max(1, S.n) * words);
        S.words_per_row = words;
        MG_CHECK_CUDA(cudaMemsetAsync(S.xp, 0, (size_t)std::max(1, S.n) * words * sizeof(unsigned long long),
                                      ctx->stream));
        // epochs restart below every word
        MG_CHECK_CUDA(cudaMemsetAsync(S.sync, 0, sizeof(GsSync), ctx->stream));
    }
}

template <class T, int B>
static void launch_gs_tiles(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b, T* x,
                            Sched& S, T omega, bool reverse, int nsw) {
    using G = GsTile<T, B>;
    constexpr int WPB = G::WPB, tile = kGsTile<T, B>;
    packed_rows(ctx, S, G::W);
    auto kern = k_gs_tiles<T, B>;
    MG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM));
    int per_sm = 0;
    MG_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WPB * 32, G::SMEM));
    MG_REQUIRE(per_sm > 0, MGLDG_ERR_CUDA, "Gauss-Seidel kernel does not fit on an SM");
    const int64_t groups = (int64_t)nsw * ((S.n + tile - 1) / tile);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(groups, (int64_t)per_sm * ctx->sm_count));
    GsPass& P = get_pass(ctx, S, reverse ? 1 : 0, nsw, grid, tile, (int)G::SLOTS);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(WPB * 32);
    cfg.dynamicSmemBytes = G::SMEM;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs co-resident
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    {
        Launch L(ctx, MGLDG_K_GS);
        MG_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, (const int*)P.cta_ptr, (const int4*)P.rec,
                                         (const signed char*)P.ltag, (int64_t)A->h_row_ptr.back(), nsw,
                                         (const int*)A->col_idx, vals, Dinv, b, x, S.xp, (const int*)S.xptr,
                                         (const int*)S.xidx, S.sync, omega, (int)reverse, S.timeout_ns));
    }
}

template <class T, int B>
static void launch_gs(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b, T* x, Sched& S,
                      T omega, bool reverse, int nsw) {
    constexpr int WPB = 4;
    constexpr int MAXE = 1;
    auto kern = k_gs_pass<T, B, WPB, MAXE>;
    packed_rows(ctx, S, B * Packed<T>::WPV);
    GsPass& P = get_pass(ctx, S, reverse ? 1 : 0, nsw, 0, 0, 0);
    int per_sm = 0;
    MG_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WPB * 32, 0));
    MG_REQUIRE(per_sm > 0, MGLDG_ERR_CUDA, "Gauss-Seidel kernel does not fit on an SM");
    const int grid = std::max(1, std::min((P.nitems + WPB - 1) / WPB, per_sm * ctx->sm_count));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(WPB * 32);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs co-resident
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    {
        Launch L(ctx, MGLDG_K_GS);
        MG_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, P.nitems, (const int*)P.items, nsw, (const int*)A->row_ptr,
                                         (const int*)A->col_idx, vals, Dinv, b, x, S.xp, (const int*)S.xptr,
                                         (const int*)S.xidx, S.sync, omega, (int)reverse, S.timeout_ns));
    }
}

template <class T>
void gs_sweeps(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b, T* x, Sched& S, T omega,
               bool reverse, int nsw) {
    if (S.n == 0 || nsw <= 0) return;
    MG_REQUIRE(A->br == A->bc, MGLDG_ERR_SHAPE, "smoother needs square blocks");
    while (nsw > 0) {
        const int k = std::min(nsw, 4);
        switch (A->br) {
            case 1: launch_gs_tiles<T, 1>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 3: launch_gs_tiles<T, 3>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 4: launch_gs_tiles<T, 4>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 6: launch_gs_tiles<T, 6>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 8: launch_gs_tiles<T, 8>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 9: launch_gs_tiles<T, 9>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 10: launch_gs_tiles<T, 10>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 16: launch_gs_tiles<T, 16>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 25: launch_gs<T, 25>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            case 27: launch_gs<T, 27>(ctx, A, vals, Dinv, b, x, S, omega, reverse, k); break;
            default: throw Error(MGLDG_ERR_UNSUPPORTED, "Gauss-Seidel: unsupported block size");
        }
        nsw -= k;
    }
}
template void gs_sweeps<double>(mgldg_ctx*, const mgldg_bsr*, const double*, const double*, const double*, double*,
                                Sched&, double, bool, int);
template void gs_sweeps<float>(mgldg_ctx*, const mgldg_bsr*, const float*, const float*, const float*, float*, Sched&,
                               float, bool, int);

template <class T, int B>
static void launch_jacobi(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b,
                          const T* xin, T* xout, T omega, bool xzero) {
    constexpr int WPB = 8;
    int grid = std::max(1, std::min((A->nbr + WPB - 1) / WPB, ctx->sm_count * 16));
    {
        Launch L(ctx, MGLDG_K_JACOBI);
        k_jacobi<T, B, WPB><<<grid, WPB * 32, 0, ctx->stream>>>(A->nbr, A->row_ptr, A->col_idx, vals, Dinv, b, xin,
                                                                xout, omega, xzero);
    }
    check_launch();
}

template <class T>
void jacobi_sweep(mgldg_ctx* ctx, const mgldg_bsr* A, const T* vals, const T* Dinv, const T* b, const T* xin,
                  T* xout, T omega, bool xzero) {
    if (A->nbr == 0) return;
    if constexpr (std::is_same<T, float>::value) {
        if (bulk_jacobi_f32(ctx, A, vals, Dinv, b, xin, xout, omega, xzero)) return;
    }
    if (split_jacobi(ctx, A, vals, Dinv, b, xin, xout, omega, xzero)) return;
    if (!A->blk) switch (A->br) {
            case 3: launch_jacobi_rows<T, 3>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
            case 4: launch_jacobi_rows<T, 4>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
            case 6: launch_jacobi_rows<T, 6>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
            case 8: launch_jacobi_rows<T, 8>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
            case 9: launch_jacobi_rows<T, 9>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
            case 10: launch_jacobi_rows<T, 10>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        }
    switch (A->br) {
        case 1: launch_jacobi<T, 1>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 3: launch_jacobi<T, 3>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 4: launch_jacobi<T, 4>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 6: launch_jacobi<T, 6>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 8: launch_jacobi<T, 8>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 9: launch_jacobi<T, 9>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 10: launch_jacobi<T, 10>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 16: launch_jacobi<T, 16>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 25: launch_jacobi<T, 25>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
        case 27: launch_jacobi<T, 27>(ctx, A, vals, Dinv, b, xin, xout, omega, xzero); return;
    }
    throw Error(MGLDG_ERR_UNSUPPORTED, "Jacobi: unsupported block size");
}
bool jacobi_f16(mgldg_ctx* ctx, const mgldg_bsr* A, const float* Dinv, const float* b, const float* xin, float* xout,
                float omega, bool xzero) {
    if (!A->val16 || A->blk || A->nbr == 0 || !f16_shape(A->br, A->bc)) return false;
    return bulk_jacobi_f16(ctx, A, Dinv, b, xin, xout, omega, xzero);
}

template void jacobi_sweep<double>(mgldg_ctx*, const mgldg_bsr*, const double*, const double*, const double*,
                                   const double*, double*, double, bool);
template void jacobi_sweep<float>(mgldg_ctx*, const mgldg_bsr*, const float*, const float*, const float*, const float*,
                                  float*, float, bool);

}  // namespace mg

// ================================================================== C ABI ==
extern "C" int mgldg_gs_levels(int nbr, const int* row_ptr, const int* col_idx, int reverse, int* level,
                               int* order, int* nlevels) {
    if (nbr < 0 || !row_ptr || (nbr > 0 && row_ptr[nbr] > 0 && !col_idx)) return MGLDG_ERR_ARG;
    try {
        std::vector<int> lev, wp, wi, ord;
        int nl = 0;
        mg::gs_levels_host(nbr, row_ptr, col_idx, reverse ? 1 : 0, lev, wp, wi, ord, nl);
        if (level) std::copy(lev.begin(), lev.end(), level);
        if (order) std::copy(ord.begin(), ord.end(), order);
        if (nlevels) *nlevels = nl;
    } catch (...) {
        return MGLDG_ERR_NOMEM;
    }
    return MGLDG_OK;
}

extern "C" int mgldg_gs_pass_levels(int nbr, const int* row_ptr, const int* col_idx, int reverse, int nsw,
                                    int* level, int* nlevels) {
    if (nbr < 0 || !row_ptr || nsw < 1 || nsw > 7 || (nbr > 0 && row_ptr[nbr] > 0 && !col_idx)) return MGLDG_ERR_ARG;
    try {
        std::vector<int> nbp, nbi, lev;
        mg::symmetrised_neighbours(nbr, row_ptr, col_idx, nbp, nbi);
        const int nl = mg::gs_pass_levels_host(nbr, nbp, nbi, reverse ? 1 : 0, nsw, lev);
        if (level) std::copy(lev.begin(), lev.end(), level);
        if (nlevels) *nlevels = nl;
    } catch (...) {
        return MGLDG_ERR_NOMEM;
    }
    return MGLDG_OK;
}

namespace mg {

// One forward sweep over blocks of B, FP64, of a system of two rows of which
// only row 1 is scheduled (`pass` fills the work list): it waits for row 0
// until the time limit.  True if the kernel reported that.
template <int B, class F>
static bool wait_runs_out(mgldg_ctx* ctx, int64_t timeout_ns, F&& pass) {
    std::vector<int> rp{0, 2, 4}, ci{0, 1, 0, 1};
    mgldg_bsr* A = bsr_new(ctx, 2, 2, B, B, rp, ci);
    Sched S;
    double* v = nullptr;   // Dinv, b, x
    bool out = false;
    auto clean = [&]() {
        sched_free(S);
        dfree(v);
        delete A;
    };
    try {
        std::vector<double> av(4 * B * B, 0.0), dv(2 * B * B, 0.0);
        for (int k = 0; k < 4; ++k)
            for (int r = 0; r < B; ++r) av[((size_t)k * B + r) * B + r] = k == 1 || k == 2 ? 1.0 : 2.0;
        for (int r = 0; r < 2 * B; ++r) dv[(size_t)r * B + r % B] = 0.5;
        upload(ctx, A->val, av.data(), av.size());
        v = dalloc<double>(dv.size() + 4 * B);
        double *b = v + dv.size(), *x = b + 2 * B;
        upload(ctx, v, dv.data(), dv.size());
        MG_CHECK_CUDA(cudaMemsetAsync(b, 0, 4 * B * sizeof(double), ctx->stream));
        sched_build(ctx, A, S);
        S.timeout_ns = timeout_ns;
        S.passes.emplace_back();
        GsPass& P = S.passes.back();
        P.nsw = P.nitems = P.depth = 1;
        pass(P);
        gs_sweeps<double>(ctx, A, A->val, v, b, x, S, 1.0, false, 1);
        sync(ctx);
        MG_REQUIRE(S.passes.size() == 1, MGLDG_ERR_ARG, "self-test: the work list was not taken");
        out = gs_take_error(ctx, S) != 0;
        // the context must still work: a plain SpMV
        spmv<double>(ctx, A, 1.0, b, 0.0, nullptr, x);
        sync(ctx);
    } catch (...) {
        clean();
        throw;
    }
    clean();
    return out;
}

}  // namespace mg

// Runs the Gauss-Seidel kernels on two-row systems in which row 1 waits for
// row 0 but row 0 is never scheduled (a pass whose only item is row 1), so
// the wait can only end by its time limit.  Reports the status the kernels
// left and checks that the stream is still usable afterwards.
extern "C" int mgldg_selftest_wait_timeout(mgldg_ctx* ctx, int64_t timeout_ns, int* status) {
    MG_API_BEGIN(ctx)
    MG_REQUIRE(status && timeout_ns > 0 && timeout_ns <= 2000000000LL, MGLDG_ERR_ARG, "bad self-test arguments");
    bool out = true;
    // tiles: as another CTA's row (in global memory), then as its own CTA's (in
    // shared memory), under the number of an item that the list does not have
    for (int tag0 = 0; tag0 >= -1; --tag0)
        out = wait_runs_out<1>(ctx, timeout_ns, [&](GsPass& P) {
            const signed char tag[4] = {0, 0, (signed char)tag0, 0};
            int tab[7] = {(1 << 3) | 0, 2, 2, 0, /* items */ 0, 1, /* tags */ 0};
            std::memcpy(tab + 6, tag, sizeof tag);
            P.grid = 1;
            P.tile = kGsTile<double, 1>;
            P.slots = GsTile<double, 1>::SLOTS;
            P.items = dalloc<int>(7);
            P.rec = reinterpret_cast<int4*>(P.items);
            P.cta_ptr = P.items + 4;
            P.ltag = reinterpret_cast<signed char*>(P.items + 6);
            upload(ctx, P.items, tab, 7);
            sync(ctx);
        }) && out;
    // row by row (blocks of 25 and 27)
    out = wait_runs_out<25>(ctx, timeout_ns, [&](GsPass& P) {
        const int item = (1 << 3) | 0;
        P.items = dalloc<int>(1);
        upload(ctx, P.items, &item, 1);
        sync(ctx);
    }) && out;
    *status = out ? MGLDG_ERR_TIMEOUT : MGLDG_OK;
    MG_API_END
}
