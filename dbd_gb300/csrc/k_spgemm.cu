// k_spgemm.cu -- symbolic and numeric SpGEMM kernels per row category.
//
// Replaces the reference's expansion kernels rowproduct_{sparse,dense,ddense}
// (dbd/for_small_datasets/src/computeGPU.cu:135-294), its global-memory dense
// merge (:296-329) and its compaction kernel collect (:331-341).  The
// reference writes every intermediate product to HBM and re-reads it for an
// FP32 atomic merge into a dense global row, deciding structure by value
// (|partial sum| < 1e-4).  Here no intermediate product touches HBM; each
// bin of rows (by products, size and column window) has its own kernels:
//
//   tiny rows   (P_r <= 32)     one lane per row, products listed in shared
//                               memory, sorted by column in registers and
//                               summed in Gustavson order (bit-exact FP64)
//   narrow rows (small window)  one warp per row over a window of flag bytes
//                               and FP64 accumulators (symbolic: the length of
//                               the union of the B rows' column runs when
//                               each is one run); warp bitmap ranks
//   short rows  (<= 256 nnz)    one warp per row: symbolic by a shared hash
//                               table; numeric by expand-sort-compress in
//                               registers for rows of at most 512 products, else by the
//                               table, compaction and a bitonic sort
//   CTA rows                    the row's A entries staged in shared memory,
//                               warps over consecutive products with several
//                               B loads in flight (warp_range_ld): hash
//                               tables for narrow-span rows, bitmap ranks
//                               for rows within 2^18 columns (sums in shared
//                               memory up to 4096 entries, products reduced
//                               into C in place above)
//   wide rows   (symbolic)      persistent CTAs, a shared bitmap over windows
//                               of up to 2^19 columns that stays zero between
//                               rows, kept for the numeric rank kernels
//   dense rows  (numeric)       persistent CTAs, bitmap ranks over 2^19-column
//                               windows in shared memory, products reduced
//                               into C in place
//
// Structure is decided by index only (a column belongs to a row as soon as a
// product lands on it).  GB300's FP64 pipe is narrow (about two FP64
// instructions per SM per clock), so the numeric kernels spend one FP64
// instruction per product: a fused multiply-add into the accumulator (plain,
// or inside a compare-and-swap loop where lanes may collide), or a multiply
// whose sum the L2 performs (global reductions: rank rows past 4096 entries and
// dense rows), or, in warp rows of at most 256 products, sorts add up.  The tiny
// path rounds each product (__dmul_rn) and adds in the oracle's order,
// reproducing it bit for bit; the other paths differ from it by summation order
// and by the fused roundings, well inside the 1e-12 tolerance.
#include "cta_stage.cuh"
#include "dbd_internal.h"
#include "warp_chunk.cuh"

#include <algorithm>
#include <mutex>
#include <vector>
#include <climits>

namespace dbd {

namespace {

constexpr int32_t EMPTY = -1;

constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x >> 1); }

__device__ __forceinline__ uint32_t hslot(int32_t c, int shift) {
    return ((uint32_t)c * 0x9E3779B1u) >> shift;
}

// *acc += a * b with one rounding, atomically (a compare-and-swap loop around
// one DFMA; shared or global memory).
__device__ __forceinline__ void atomic_fma(double *acc, double a, double b) {
    unsigned long long *p = reinterpret_cast<unsigned long long *>(acc);
    unsigned long long old = *reinterpret_cast<volatile unsigned long long *>(p), seen;
    do {
        seen = old;
        old = atomicCAS(p, seen, (unsigned long long)__double_as_longlong(
                                     __fma_rn(a, b, __longlong_as_double((long long)seen))));
    } while (old != seen);
}

// A column's offset in its row's window: true when inside [0, limit), else
// records DEV_OUT_OF_WINDOW (the window came from B's row ranges, so this
// only fires when B changed after it was loaded) and the product is skipped.
__device__ __forceinline__ bool in_window(uint32_t rel, uint32_t limit, int *err) {
    if (rel < limit) return true;
    raise(err, DEV_OUT_OF_WINDOW);
    return false;
}

// ---------------------------------------------------------------------------
// Warp-level enumeration of the products of up to 32 consecutive A entries
// (Chunk, load_chunk and chunk_owner in warp_chunk.cuh): product t
// (0 <= t < total) comes from the lane whose inclusive length prefix first
// exceeds t.
// ---------------------------------------------------------------------------
// Steps of B loads a wide-row warp keeps in flight on rows past the touch list.
constexpr int kWideLoads = 4;
// Steps of B loads a warp-hash row keeps in flight.
constexpr int kHashWarpLoads = 2;
// Warp-hash rows of at most this many products are sorted instead of hashed.
// Up to kEscMax every product is rounded before it is added; past it, to
// kFusedMax, the sums are fused multiply-adds, as the table's are: such rows
// have columns of several products by necessity (they hold at most 256 entries),
// whose rms error would be 0.62 units of the last place instead of 0.54
// (against exact sums).
constexpr int kEscMax = 256, kFusedMax = 512;
constexpr int kEscShift = 8, kFusedShift = 9;  // bits of a product's number in their keys
// Mean B row length from which their products are listed by groups of lanes, at
// which both ways take the same time: 100k rows of about 200 products, groups
// against one flat sequence, mean 3 289 and 262 us, 4 246 and 225, 5 221 and 227,
// 6 218 and 221, 8 195 and 198, 12 158 and 172.
constexpr int kEscGroupLen = 6;

// Position in B of product t and the lane its entry is on (all lanes call;
// results valid when t < total).
__device__ __forceinline__ int32_t chunk_pos(const Chunk &c, int32_t t, double *a_out, int32_t *owner = nullptr) {
    const int o = chunk_owner(c, t);
    if (a_out) *a_out = __shfl_sync(FULL, c.a, o);
    if (owner) *owner = o;
    return t + __shfl_sync(FULL, c.bs - (c.incl - c.len), o);
}

// ---------------------------------------------------------------------------
// Block-level helpers.
// ---------------------------------------------------------------------------
template <int THREADS>
__device__ __forceinline__ int32_t block_min_i32(int32_t v, int32_t *sh) {
#pragma unroll
    for (int d = 16; d; d >>= 1) v = min(v, __shfl_xor_sync(FULL, v, d));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    int32_t r = INT_MAX;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) r = min(r, sh[i]);
    __syncthreads();
    return r;
}

template <int THREADS>
__device__ __forceinline__ int block_sum_i(int v, int *sh) {
#pragma unroll
    for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    int r = 0;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) r += sh[i];
    __syncthreads();
    return r;
}

// B's rows ascend strictly: the host's flag, or for a device-driven launch
// the flag the device computed for this run (bUnsorted).
template <class Args>
__device__ __forceinline__ bool b_sorted(const Args &a) {
    return a.bUnsorted ? *a.bUnsorted == 0 : a.bSorted != 0;
}

// Column and value of a product, as loaded by warp_range_ld.
struct ColVal {
    int32_t c;
    double v;
};

// Sets bit rel of a shared bitmap on lanes with v, one atomicOr per lane.
// Lanes that share a word serialise on it; a segmented OR over runs of such
// lanes (one atomic per run) costs more instructions than that saves, on
// sparse and dense power-law windows alike.
__device__ __forceinline__ void or_bit(uint32_t *bm, bool v, uint32_t rel) {
    if (v) atomicOr(&bm[rel >> 5], 1u << (rel & 31));
}

// Writes the columns of a ranked bitmap with the work balanced by output
// position: thread t writes out[r] = colbase + 32 w + b for the output ranks
// r in [t tot / T, (t + 1) tot / T) below lim, a contiguous run.  The bitmap
// is cut into THREADS groups of G consecutive words (G <= 32); tbase[g] is
// the rank of group g's first column and tmask[g] the mask of its non-empty
// words (both in shared memory).  A thread finds the group holding its
// first rank by binary search, then walks words and bits in order.  (When
// the columns are written by the thread that owns their words instead, a
// thread over a dense stretch of the row writes up to 32 G columns while
// its neighbours write few, and the CTA waits for it.)  The run goes out in
// aligned 16-byte stores, its ragged ends one column at a time: each lane
// of a warp writes its own run, so per-column stores would cost a memory
// transaction per column.
template <int THREADS>
__device__ __forceinline__ void write_columns_balanced(const uint32_t *bits, const int32_t *tbase,
                                                       const uint32_t *tmask, int G, int32_t tot, int32_t *out,
                                                       int64_t lim, int64_t colbase) {
    const int tid = threadIdx.x;
    const int32_t r0 = (int32_t)((int64_t)tot * tid / THREADS);
    const int32_t r1 = (int32_t)min((int64_t)tot * (tid + 1) / THREADS, lim);
    if (r0 >= r1) return;
    // The last group whose first rank is at most r0 holds rank r0 (the
    // next group starts above it, so this one is not empty).
    int lo = 0, hi = THREADS - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tbase[mid] <= r0) lo = mid;
        else hi = mid - 1;
    }
    int g = lo;
    uint32_t m = tmask[g];
    int32_t p = tbase[g];
    int w = G * g + __ffs(m) - 1;
    uint32_t word = bits[w];
    while (p + __popc(word) <= r0) {
        p += __popc(word);
        m &= m - 1u;
        w = G * g + __ffs(m) - 1;
        word = bits[w];
    }
    for (; p < r0; ++p) word &= word - 1u;  // drop the bits before rank r0
    auto next = [&]() -> int32_t {
        while (!word) {
            m &= m - 1u;
            while (!m) m = tmask[++g];
            w = G * g + __ffs(m) - 1;
            word = bits[w];
        }
        const int b = __ffs(word) - 1;
        word &= word - 1u;
        return (int32_t)(colbase + (w << 5) + b);
    };
    // out + r is 16-byte aligned when (k0 + r) % 4 == 0.
    const uint32_t k0 = (uint32_t)(reinterpret_cast<uintptr_t>(out) >> 2) & 3u;
    for (; p < r1 && ((k0 + (uint32_t)p) & 3u); ++p) __stcs(out + p, next());
    for (; p + 4 <= r1; p += 4) {
        const int32_t q0 = next(), q1 = next(), q2 = next(), q3 = next();
        __stcs(reinterpret_cast<int4 *>(out + p), make_int4(q0, q1, q2, q3));
    }
    for (; p < r1; ++p) __stcs(out + p, next());
}

template <int GROUP, int ROWS>
__device__ __forceinline__ void group_sync() {
    if constexpr (ROWS > 1) {
        static_assert(GROUP == 32, "multi-row CTAs use one warp per row");
        __syncwarp();
    } else {
        __syncthreads();
    }
}

template <int TABLE>
__device__ __forceinline__ int hash_insert_key(int32_t *keys, int32_t col, int *err) {
    constexpr int SHIFT = 32 - ilog2(TABLE);
    uint32_t h = hslot(col, SHIFT);
#pragma unroll 1
    for (int probe = 0; probe < TABLE; ++probe) {
        const int32_t k = ((volatile int32_t *)keys)[h];
        if (k == col) return 0;
        if (k == EMPTY) {
            const int32_t old = atomicCAS(&keys[h], EMPTY, col);
            if (old == EMPTY) return 1;
            if (old == col) return 0;
        }
        h = (h + 1) & (TABLE - 1);
    }
    raise(err, DEV_TABLE_FULL);
    return 0;
}

template <int TABLE>
__device__ __forceinline__ int hash_insert_slot(int32_t *keys, int32_t col, int *err) {
    constexpr int SHIFT = 32 - ilog2(TABLE);
    uint32_t h = hslot(col, SHIFT);
#pragma unroll 1
    for (int probe = 0; probe < TABLE; ++probe) {
        const int32_t k = ((volatile int32_t *)keys)[h];
        if (k == col) return (int)h;
        if (k == EMPTY) {
            const int32_t old = atomicCAS(&keys[h], EMPTY, col);
            if (old == EMPTY || old == col) return (int)h;
        }
        h = (h + 1) & (TABLE - 1);
    }
    raise(err, DEV_TABLE_FULL);
    return -1;
}

__device__ __forceinline__ int warp_sum_i(int v) {
#pragma unroll
    for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
    return v;
}

// ======================================================================
// Symbolic kernels: rowNnz[row] = number of distinct columns of C's row.
// ======================================================================

// Tiny rows (P_r <= 32, |A_r| <= 32): one lane per row.  The lane lists the
// B positions (and A values) of its row's products in Gustavson order in its
// own column of a warp's shared array (entry i of lane l at kTinyPitch i + l:
// no bank conflicts where the lanes walk in step, nor along one lane's
// entries), loads eight products at a time, sorts them in registers by
// (column, position in that order) and sums each run of equal columns, which
// is Gustavson's order.  The sort is Batcher's odd-even merge sort (Knuth,
// TAOCP vol. 3, 5.2.2) of 8, 16 or 32 keys, 32 bits each: 2 instructions a
// comparator, no memory, no divergence.
//
// A warp per row, the form before, spends the same instructions on one row
// that this spends on 32, holds one row's chain of dependent loads in flight
// instead of 32, and (numeric) issues 32 FP64 additions per row, 16 clocks of
// the SM's FP64 pipe each, where a row needs one per product: 512 clocks a
// row set its time.  2.1M five-point rows (25 products each): symbolic
// 574 -> 88 us, numeric 4401 -> 393 us; 4096 rows: symbolic 8 -> 6 us, numeric
// 17 -> 17 us.  (Merging the products into a sorted list in shared
// memory instead of sorting registers: 95, 422 and 19 us.)
constexpr int kTinyPitch = 33;
constexpr int kTinyWords = kTinyMax * kTinyPitch;
constexpr int kSymTinyWarps = 4;  // 16.5 KB a CTA
constexpr int kNumTinyWarps = 2;  // 24.8 KB a CTA

// Batcher's merge exchange: the comparators of stage (P, K), then the next.
template <int N, int P, int K, class T>
__device__ __forceinline__ void merge_exchange(T (&key)[N]) {
#pragma unroll
    for (int x = K % P; x < N - K; ++x) {
        if ((x - K % P) % (2 * K) < K && x / (2 * P) == (x + K) / (2 * P)) {
            const T lo = min(key[x], key[x + K]), hi = max(key[x], key[x + K]);
            key[x] = lo;
            key[x + K] = hi;
        }
    }
    if constexpr (K > 1) merge_exchange<N, P, K / 2>(key);
    else if constexpr (2 * P < N) merge_exchange<N, 2 * P, 2 * P>(key);
}

// Lists this lane's products: their positions in B, at most kTinyMax, and
// (NUM) their A values.  Returns how many.
template <bool NUM>
__device__ __forceinline__ int tiny_list(const CsrDev &A, const CsrDev &B, int32_t row, bool live, int32_t *pos,
                                         double *val) {
    int32_t e = 0, e1 = 0;
    if (live) {
        e = __ldg(&A.ptr[row]);
        e1 = __ldg(&A.ptr[row + 1]);
    }
    int n = 0;
    for (; e < e1; e += 4) {
        int32_t k[4], bs[4], len[4];
        double av[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            k[u] = e + u < e1 ? __ldg(&A.idx[e + u]) : -1;
            if constexpr (NUM) av[u] = e + u < e1 ? __ldg(&A.val[e + u]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            bs[u] = k[u] >= 0 ? __ldg(&B.ptr[k[u]]) : 0;
            len[u] = k[u] >= 0 ? __ldg(&B.ptr[k[u] + 1]) - bs[u] : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int stop = min(n + len[u], kTinyMax);
            for (int32_t q = bs[u]; n < stop; ++q, ++n) {
                pos[kTinyPitch * n] = q;
                if constexpr (NUM) val[kTinyPitch * n] = av[u];
            }
        }
    }
    return n;
}

// Distinct columns among a lane's n <= N listed products.
template <int N>
__device__ __forceinline__ int tiny_count(const CsrDev &B, int n, const int32_t *pos) {
    uint32_t key[N];
#pragma unroll
    for (int i = 0; i < N; ++i) key[i] = i < n ? (uint32_t)__ldg(&B.idx[pos[kTinyPitch * i]]) : 0xffffffffu;
    merge_exchange<N, 1, 1>(key);
    int m = n > 0 ? 1 : 0;
#pragma unroll
    for (int i = 1; i < N; ++i) m += i < n && key[i] != key[i - 1];
    return m;
}

// The sum starts at zero: a first product of -0 gives +0.
__device__ __forceinline__ double first_term(double p) { return __double_as_longlong(p) == LLONG_MIN ? 0.0 : p; }

// A lane's n <= N listed products (positions in col, A values in val) merged:
// afterwards col and val hold its distinct columns less `shift`, ascending,
// and their sums.  Returns how many.  Columns are in [base, base + 2^27).
template <int N>
__device__ __forceinline__ int tiny_sum(const CsrDev &B, int n, int32_t base, int32_t shift, int32_t *col,
                                        double *val) {
    uint32_t key[N];
#pragma unroll
    for (int i0 = 0; i0 < N; i0 += 8) {
        double v[8];
#pragma unroll
        for (int i = i0; i < i0 + 8; ++i) {
            const int32_t q = i < n ? col[kTinyPitch * i] : 0;
            key[i] = i < n ? (uint32_t)(__ldg(&B.idx[q]) - base) << 5 | (uint32_t)i : 0xffffffffu;
            v[i - i0] = i < n ? __ldg(&B.val[q]) : 0.0;
        }
#pragma unroll
        for (int i = i0; i < i0 + 8; ++i)
            if (i < n) val[kTinyPitch * i] = __dmul_rn(val[kTinyPitch * i], v[i - i0]);
    }
    merge_exchange<N, 1, 1>(key);
    double p[N];
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = i < n ? val[kTinyPitch * (int)(key[i] & 31u)] : 0.0;
    int m = 0;
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (i < n) {
            const bool head = i == 0 || (key[i] >> 5) != (key[i > 0 ? i - 1 : 0] >> 5);
            if (head) {
                acc = first_term(p[i]);
                col[kTinyPitch * m] = (int32_t)(key[i] >> 5) + (base - shift);
                ++m;
            } else {
                acc = __dadd_rn(acc, p[i]);
            }
            val[kTinyPitch * (m - 1)] = acc;
        }
    }
    return m;
}

// The same for rows over 2^27 columns or more, whose keys would not fit 32
// bits: products are merged one by one into the sorted list [0, m), which
// never passes the product being taken.
__device__ __noinline__ int tiny_sum_wide(const CsrDev &B, int n, int32_t shift, int32_t *col, double *val) {
    int m = 0;
    for (int i = 0; i < n; ++i) {
        const int32_t q = col[kTinyPitch * i];
        const int32_t c = __ldg(&B.idx[q]) - shift;
        const double p = __dmul_rn(val[kTinyPitch * i], __ldg(&B.val[q]));
        int j = m;
        while (j > 0 && col[kTinyPitch * (j - 1)] > c) --j;
        if (j > 0 && col[kTinyPitch * (j - 1)] == c) {
            val[kTinyPitch * (j - 1)] = __dadd_rn(val[kTinyPitch * (j - 1)], p);
            continue;
        }
        for (int x = m; x > j; --x) {
            col[kTinyPitch * x] = col[kTinyPitch * (x - 1)];
            val[kTinyPitch * x] = val[kTinyPitch * (x - 1)];
        }
        col[kTinyPitch * j] = c;
        val[kTinyPitch * j] = first_term(p);
        ++m;
    }
    return m;
}

__device__ __forceinline__ void sym_tiny_rows(const SymArgs &a, int32_t begin, int32_t count, int64_t vb) {
    __shared__ int32_t cols[kSymTinyWarps][kTinyWords];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int64_t item = (vb * kSymTinyWarps + g) * 32 + lane;
    const bool live = item < count;
    const int32_t row = live ? a.list[begin + item] : 0;
    int32_t *pos = cols[g] + lane;
    const int n = tiny_list<false>(a.A, a.B, row, live, pos, nullptr);
    const int most = __reduce_max_sync(FULL, n);
    const int m = most <= 8    ? tiny_count<8>(a.B, n, pos)
                  : most <= 16 ? tiny_count<16>(a.B, n, pos)
                               : tiny_count<kTinyMax>(a.B, n, pos);
    if (live) a.rowNnz[row] = m;
}

__global__ void __launch_bounds__(32 * kSymTinyWarps) k_sym_tiny(SymArgs a, int32_t begin, int32_t count) {
    sym_tiny_rows(a, begin, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
__global__ void __launch_bounds__(32 * kSymTinyWarps) k_sym_tiny_dd(SymArgs a, int bin) {
    const int32_t begin = a.binStart[bin], count = a.binStart[bin + 1] - begin;
    for (int64_t vb = blockIdx.x; vb * (32 * kSymTinyWarps) < count; vb += gridDim.x) {
        sym_tiny_rows(a, begin, count, vb);
        __syncthreads();
    }
}

// Warp hash rows: one warp per row, ROWS rows per CTA, TABLE keys per row.
template <int ROWS, int TABLE>
__device__ __forceinline__ void sym_hash_warp_rows(const SymArgs &a, int32_t begin, int32_t count, int64_t vb) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)vb * ROWS + g;
    if (item >= count) return;
    int32_t *keys = reinterpret_cast<int32_t *>(smem) + (size_t)g * TABLE;
    const int32_t row = a.list[begin + item];
    for (int i = lane; i < TABLE; i += 32) keys[i] = EMPTY;
    __syncwarp();
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    int cnt = 0;
    for (int32_t e = e0; e < e1; e += 32) {
        const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
        for (int32_t t0 = 0; t0 < c.total; t0 += 32 * kHashWarpLoads) {
            int32_t col[kHashWarpLoads];
#pragma unroll
            for (int u = 0; u < kHashWarpLoads; ++u) {
                col[u] = -1;
                const int32_t t = t0 + 32 * u + lane;
                if (t0 + 32 * u < c.total) {
                    const int32_t j = chunk_pos(c, t, nullptr);
                    if (t < c.total) col[u] = __ldg(&a.B.idx[j]);
                }
            }
#pragma unroll
            for (int u = 0; u < kHashWarpLoads; ++u)
                if (col[u] >= 0) cnt += hash_insert_key<TABLE>(keys, col[u], a.err);
        }
    }
    cnt = warp_sum_i(cnt);
    if (lane == 0) a.rowNnz[row] = cnt;
}

template <int ROWS, int TABLE>
__global__ void __launch_bounds__(32 * ROWS) k_sym_hash_warp(SymArgs a, int32_t begin, int32_t count) {
    sym_hash_warp_rows<ROWS, TABLE>(a, begin, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int ROWS, int TABLE>
__global__ void __launch_bounds__(32 * ROWS) k_sym_hash_warp_dd(SymArgs a, int bin) {
    const int32_t begin = a.binStart[bin], count = a.binStart[bin + 1] - begin;
    for (int64_t vb = blockIdx.x; vb * ROWS < count; vb += gridDim.x) {
        sym_hash_warp_rows<ROWS, TABLE>(a, begin, count, vb);
        __syncthreads();
    }
}

// CTA hash rows: one CTA per row, products spread over all threads.
template <int THREADS, int TABLE>
__device__ __forceinline__ void sym_hash_cta_rows(const SymArgs &a, int32_t begin, int64_t vb) {
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    __shared__ int32_t sh[THREADS / 32];
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    int32_t *keys = reinterpret_cast<int32_t *>(smem + L::bytes);
    const int tid = threadIdx.x;
    const int32_t row = a.list[begin + vb];
    for (int i = tid; i < TABLE; i += THREADS) keys[i] = EMPTY;
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    int cnt = 0;
    for (int32_t eb = e0; eb < e1; eb += THREADS) {
        int nb;
        const int32_t total =
            stage_entries<THREADS, false>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, nullptr, &nb, sh);
        int32_t tb, te;
        warp_share<THREADS>(total, &tb, &te);
        warp_range_ld<4>(
            pre, bst, nb, tb, te, [&](int32_t pos) { return __ldg(&a.B.idx[pos]); },
            [&](bool v, int32_t col, int) {
                if (v) cnt += hash_insert_key<TABLE>(keys, col, a.err);
            });
        __syncthreads();
    }
    cnt = block_sum_i<THREADS>(cnt, sh);
    if (tid == 0) a.rowNnz[row] = cnt;
}

template <int THREADS, int TABLE>
__global__ void __launch_bounds__(THREADS) k_sym_hash_cta(SymArgs a, int32_t begin) {
    sym_hash_cta_rows<THREADS, TABLE>(a, begin, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int THREADS, int TABLE>
__global__ void __launch_bounds__(THREADS) k_sym_hash_cta_dd(SymArgs a, int bin) {
    const int32_t begin = a.binStart[bin], count = a.binStart[bin + 1] - begin;
    for (int64_t vb = blockIdx.x; vb < count; vb += gridDim.x) {
        sym_hash_cta_rows<THREADS, TABLE>(a, begin, vb);
        __syncthreads();
    }
}

// or_bit that also counts and records: returns the number of bits this
// lane newly set (its bit, if the word's old value lacked it), and appends
// every word it finds zero to touched[] (through *nt; entries past cap are
// dropped, *nt still counts them).  Lanes that share a bit or a word
// serialise on its atomic, so exactly one of them counts the bit and one
// records the word.
__device__ __forceinline__ int or_bits_count(uint32_t *bm, bool v, uint32_t rel, int32_t *touched, int *nt,
                                             int cap) {
    if (!v) return 0;
    const uint32_t bit = 1u << (rel & 31);
    const uint32_t old = atomicOr(&bm[rel >> 5], bit);
    if (cap > 0 && old == 0u) {
        const int k = atomicAdd(nt, 1);
        if (k < cap) touched[k] = (int32_t)(rel >> 5);
    }
    return (old & bit) ? 0 : 1;
}

// Words a wide-row window clears one by one: past a quarter of the window a
// full clear is as cheap.
__host__ __device__ __forceinline__ int wide_touch_cap(int winBits) {
    return min(kWideTouchMax, (winBits >> 5) / 4);
}

// Column slabs that a wide row is cut into, an item each; 0 for a row that is
// not (fewer than a.cutP products, one slab, or B's rows not ascending).
__device__ __forceinline__ int sym_cut_slabs(const SymArgs &a, int32_t row) {
    if (a.rowP[row] < a.cutP || !b_sorted(a)) return 0;
    const int64_t base = (int64_t)(a.rowLo[row] >> 5) << 5;
    const int64_t ns = (((int64_t)a.rowHi[row] + 1 - base) + (1 << kSlabShift) - 1) >> kSlabShift;
    return ns > 1 && ns <= kMaxSlabs ? (int)ns : 0;
}

// Items of the wide rows list[begin, begin + n) that are cut.  A cut row's count
// starts at zero here, and its slab counts get their slot.
__global__ void __launch_bounds__(256) k_sym_items(SymArgs a, int32_t begin, int32_t n) {
    const int32_t i = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const int32_t row = a.list[begin + i];
    const int k = sym_cut_slabs(a, row);
    if (k == 0) return;
    const uint32_t at = atomicAdd(&a.ctr[CTR_SYM_ITEMS], (uint32_t)k);
    for (int s = 0; s < k; ++s) a.items[at + s] = SymItem{i, (int16_t)s, (int16_t)(s + 1)};
    a.rowNnz[row] = 0;
    if (a.slabCnt) {
        int32_t sl = (int32_t)atomicAdd(&a.ctr[CTR_HEAVY], 1u);
        if (sl >= a.heavyCap) sl = -1;
        a.heavySlot[row] = sl;
    }
}

// Wide rows: persistent CTAs take rows from a counter (heavy rows spread
// over the whole grid).  A shared bitmap over windows of winBits columns
// stays zero between rows: every window records the words it touched and
// clears only those (the whole window when more than kWideTouchMax were
// touched).  The row's size is the sum of newly set bits, so no popcount
// pass over the window either: a row costs its products, not its span.
// The largest rows, cut by column, are items of a launch of their own (ITEMS,
// built by k_sym_items): a piece sets, counts and keeps its slabs' columns and
// adds its count to the row's.
// 10,240 rows of R-MAT 2^21, two of which hold 3.7M products each: 2.00 ->
// 1.14 ms (1.84 with 32-bit window arithmetic alone).
template <int THREADS, bool ITEMS>
__global__ void __launch_bounds__(THREADS) k_sym_wide(SymArgs a, int32_t begin, int32_t count, int winBits) {
    if (!ITEMS && begin < 0) {  // device-driven: the bin's rows from the bin table
        begin = a.binStart[SB_WIDE];
        count = a.binStart[SB_WIDE + 1] - begin;
    }
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    __shared__ int32_t sh[THREADS / 32];
    __shared__ int nt;
    __shared__ int32_t next;
    __shared__ int32_t slot;
    __shared__ int32_t slabSh[kWideWindowBitsMax >> kSlabShift];
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    uint32_t *bm = reinterpret_cast<uint32_t *>(smem + L::bytes);
    int32_t *touched = reinterpret_cast<int32_t *>(bm + (winBits >> 5));
    const int cap = wide_touch_cap(winBits);
    int32_t *cur = touched + cap;  // per staged entry: its B cursor across windows
    const int tid = threadIdx.x;
    for (int i = tid; i < (winBits >> 5); i += THREADS) bm[i] = 0u;
    if constexpr (ITEMS) count = *(volatile int32_t *)&a.ctr[CTR_SYM_ITEMS];
    for (;;) {
        if (tid == 0) next = (int32_t)atomicAdd(&a.ctr[ITEMS ? CTR_SYM_NEXT : CTR_SYM_WIDE], 1u);
        __syncthreads();
        int32_t item = next;
        if (item >= count) break;
        SymItem it{item, -1, -1};
        if constexpr (ITEMS) {
            it = a.items[item];
            item = it.idx;
        }
        const int32_t row = a.list[begin + item];
        if (!ITEMS && a.items && sym_cut_slabs(a, row) > 0) {  // its pieces are items
            __syncthreads();  // every thread has read `next` before it changes
            continue;
        }
        constexpr bool piece = ITEMS;
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        // The row's window [lo, hi], in windows of winBits columns from lo's word.
        const int32_t rlo = a.rowLo[row], rhi = a.rowHi[row];
        const int sw = span_words(rlo, rhi);
        const int64_t base = (int64_t)(rlo >> 5) << 5;
        const int64_t start = piece ? base + ((int64_t)it.s0 << kSlabShift) : base;
        const int64_t end = piece ? min((int64_t)rhi + 1, base + ((int64_t)it.s1 << kSlabShift)) : (int64_t)rhi + 1;
        // Rows with more products than the list holds touch more words than
        // it holds as a rule: they set their bits with plain ORs (no old
        // values, no bookkeeping) and count, keep and clear the window in one
        // sweep over its words.
        const int rowCap = a.rowP[row] <= cap ? cap : 0;
        const bool keep = a.wideBits && sw <= kRankWordsMax;
        // Heavy rows record their entries per slab of 2^kSlabShift columns
        // (from `base`), for the numeric pass to cut them into pieces.
        if (tid == 0 && piece) slot = a.heavySlot ? a.heavySlot[row] : -1;
        if (tid == 0 && !piece) {
            int32_t sl = -1;
            const int64_t nslabs = ((end - base) + (1 << kSlabShift) - 1) >> kSlabShift;
            if (a.slabCnt && !rowCap && a.rowP[row] >= kHeavyP && winBits >= (1 << kSlabShift) &&
                nslabs <= kMaxSlabs) {
                sl = (int32_t)atomicAdd(&a.ctr[CTR_HEAVY], 1u);
                if (sl >= a.heavyCap) sl = -1;
            }
            slot = sl;
            if (a.heavySlot) a.heavySlot[row] = sl;
        }
        int cnt = 0;
        // Rows over several windows enumerate, per window, only the part of
        // each B row inside it (B's rows ascending).
        const bool clip = b_sorted(a) && (piece || end - base > (int64_t)winBits);
        const bool once = e1 - e0 <= THREADS;  // one batch: its cursors carry over the windows
        for (int64_t c_lo = start; c_lo < end; c_lo += winBits) {
            const int words = (int)min((int64_t)winBits, end - c_lo + 31) >> 5;
            // Columns of this window (a whole row has none past its end).
            const uint32_t lim = ITEMS ? (uint32_t)min((int64_t)winBits, end - c_lo) : (uint32_t)winBits;
            if (tid == 0) nt = rowCap ? 0 : cap + 1;
            if (tid < (kWideWindowBitsMax >> kSlabShift)) slabSh[tid] = 0;
            __syncthreads();
            for (int32_t eb = e0; eb < e1; eb += THREADS) {
                int nb;
                const int32_t total =
                    stage_entries<THREADS, false>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, nullptr, &nb, sh, clip,
                                                  c_lo, c_lo + lim, once ? cur : nullptr, once && c_lo != start);
                int32_t tb, te;
                warp_share<THREADS>(total, &tb, &te);
                if (rowCap) {
                    warp_range_ld<kWideLoads>(
                        pre, bst, nb, tb, te, [&](int32_t pos) { return __ldg(&a.B.idx[pos]); },
                        [&](bool v, int32_t col, int) {
                            const uint32_t rel = (uint32_t)col - (uint32_t)c_lo;  // below c_lo it wraps past lim
                            cnt += or_bits_count(bm, v && rel < lim, rel, touched, &nt, rowCap);
                        });
                } else {
                    warp_range_ld<kWideLoads>(
                        pre, bst, nb, tb, te, [&](int32_t pos) { return __ldg(&a.B.idx[pos]); },
                        [&](bool v, int32_t col, int) {
                            const uint32_t rel = (uint32_t)col - (uint32_t)c_lo;
                            if (v && rel < lim) atomicOr(&bm[rel >> 5], 1u << (rel & 31));
                        });
                }
                __syncthreads();
            }
            if (!rowCap) {
                uint32_t *dst = keep ? a.wideBits + (size_t)item * kRankWordsMax + ((c_lo - base) >> 5) : nullptr;
                const int32_t sl = slot;
                if (sl < 0) {
                    for (int i = tid; i < words; i += THREADS) {
                        const uint32_t x = bm[i];
                        cnt += __popc(x);
                        if (dst) __stcs(&dst[i], x);
                        bm[i] = 0u;
                    }
                } else {
                    // Groups of 32 consecutive words per thread (a slab is 64
                    // groups); lanes start at different words of their group
                    // so that a warp's loads hit 32 banks.
                    const int lane = tid & 31;
                    for (int g = tid; 32 * g < words; g += THREADS) {
                        int c = 0;
                        for (int k = 0; k < 32; ++k) {
                            const int i = 32 * g + ((k + lane) & 31);
                            if (i < words) {
                                const uint32_t x = bm[i];
                                c += __popc(x);
                                if (dst) __stcs(&dst[i], x);
                                bm[i] = 0u;
                            }
                        }
                        cnt += c;
                        if (c) atomicAdd(&slabSh[(32 * g) >> (kSlabShift - 5)], c);
                    }
                    __syncthreads();
                    const int s0 = (int)((c_lo - base) >> kSlabShift);
                    const int ns = (words + (1 << (kSlabShift - 5)) - 1) >> (kSlabShift - 5);
                    for (int t = tid; t < ns; t += THREADS) a.slabCnt[(size_t)sl * kMaxSlabs + s0 + t] = slabSh[t];
                }
                if (keep && tid == 0) a.wideSlot[row] = item;
                __syncthreads();
                continue;
            }
            if (keep) {
                // One window covers the row here; keep its bitmap for the numeric pass.
                uint32_t *dst = a.wideBits + (size_t)item * kRankWordsMax;
                for (int i = tid; i < sw; i += THREADS) __stcs(&dst[i], bm[i]);
                if (tid == 0) a.wideSlot[row] = item;
                __syncthreads();
            }
            const int n = nt;
            if (n <= cap) {
                for (int i = tid; i < n; i += THREADS) bm[touched[i]] = 0u;
            } else {
                for (int i = tid; i < words; i += THREADS) bm[i] = 0u;
            }
            __syncthreads();
        }
        cnt = block_sum_i<THREADS>(cnt, sh);
        if (tid == 0) {
            if (piece) atomicAdd(&a.rowNnz[row], cnt);
            else a.rowNnz[row] = cnt;
        }
    }
}

// Size of a row of C whose B rows are each one contiguous run of columns
// (banded and stencil matrices), with the runs' first columns non-decreasing
// in A's entry order: the length of the union of the runs, by a prefix
// maximum of the runs' last columns (the run of entry i adds the part of
// [first_i, last_i] beyond every earlier run's end).  One warp, 32 entries a
// step, no per-column work.  Returns false (count unset) when some B row is
// not one run or the first columns decrease; B's rows must ascend strictly.
// The runs' ends come from the row ranges, loaded beside the row pointers
// (B's columns would have to wait for them), and a step whose runs' ends
// do not decrease either (a band's) needs no prefix maxima.  970k rows of 65
// entries: 577 -> 344 us.
__device__ __forceinline__ bool interval_union_count(const CsrDev &A, const CsrDev &B, const int2 *range, int32_t e0,
                                                     int32_t e1, int lane, int *count) {
    int32_t endMax = INT32_MIN, firstMax = INT32_MIN;  // over the entries of earlier steps
    int add = 0;  // this lane's part of the union
    for (int32_t eb = e0; eb < e1; eb += 32) {
        const int32_t k = eb + lane < e1 ? __ldg(&A.idx[eb + lane]) : -1;
        const int32_t len = k >= 0 ? __ldg(&B.ptr[k + 1]) - __ldg(&B.ptr[k]) : 0;
        const int2 r = k >= 0 ? __ldg(&range[k]) : make_int2(0, 0);
        const bool has = len > 0;
        const int32_t f = has ? r.x : INT32_MIN, l = has ? r.y : INT32_MIN;
        const bool run = !has || l - f == len - 1;
        int32_t fPrev = __shfl_up_sync(FULL, f, 1), lPrev = __shfl_up_sync(FULL, l, 1);
        if (lane == 0) {
            fPrev = firstMax;
            lPrev = endMax;
        }
        const int last = min(31, e1 - eb - 1);
        if (__all_sync(FULL, lane > last || (has && run && f >= fPrev && l >= lPrev))) {
            if (has) add += (int)((long long)l - max((long long)f - 1, (long long)lPrev));
            firstMax = __shfl_sync(FULL, f, last);
            endMax = __shfl_sync(FULL, l, last);
            continue;
        }
        // Inclusive prefix maxima of the first and last columns over lanes.
        int32_t fm = f, lm = l;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t yf = __shfl_up_sync(FULL, fm, d), yl = __shfl_up_sync(FULL, lm, d);
            if (lane >= d) {
                fm = max(fm, yf);
                lm = max(lm, yl);
            }
        }
        fPrev = __shfl_up_sync(FULL, fm, 1);
        lPrev = __shfl_up_sync(FULL, lm, 1);
        if (lane == 0) {
            fPrev = INT32_MIN;
            lPrev = INT32_MIN;
        }
        fPrev = max(fPrev, firstMax);
        lPrev = max(lPrev, endMax);
        if (!__all_sync(FULL, run && (!has || f >= fPrev))) return false;
        if (has) add += (int)max(0LL, (long long)l - max((long long)f - 1, (long long)lPrev));
        firstMax = max(firstMax, __shfl_sync(FULL, fm, 31));
        endMax = max(endMax, __shfl_sync(FULL, lm, 31));
    }
    *count = warp_sum_i(add);
    return true;
}

// Products of one row for one warp, calling f(j, av) for every product (B
// position j, A value av) on the lane that owns it: 32 products of up to 32
// A entries per step (Chunk).  Callers with long B rows walk them row-wise
// themselves.
template <class F>
__device__ __forceinline__ void warp_products(const CsrDev &A, const CsrDev &B, int32_t e0, int32_t e1, int lane,
                                              F &&f) {
    for (int32_t e = e0; e < e1; e += 32) {
        const Chunk c = load_chunk(A, B, e, e1, lane);
        for (int32_t t0 = 0; t0 < c.total; t0 += 32) {
            const int32_t t = t0 + lane;
            double av;
            const int32_t j = chunk_pos(c, t, &av);
            if (t < c.total) f(j, av);
        }
    }
}

// Average B row length from which a row is enumerated row-wise.
constexpr int kRowwiseMinLen = 16;

// Narrow rows (window of at most kWarpSpanWords words): one warp per row,
// one flag byte per column of the window in shared memory; the row's size is
// the number of flags set.
template <int ROWS>
__device__ __forceinline__ void sym_flagw_rows(const SymArgs &a, int32_t begin, int32_t count, int64_t vb) {
    constexpr int kWords = kWarpSpanWords * 8;  // 32 flag bytes per window word
    __shared__ uint32_t fls[ROWS][kWords];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)vb * ROWS + g;
    if (item >= count) return;
    uint32_t *fw = fls[g];
    uint8_t *fb = reinterpret_cast<uint8_t *>(fw);
    const int32_t row = a.list[begin + item];
    const int32_t rlo = a.rowLo[row];
    const int32_t base = (rlo >> 5) << 5;
    const int sw = min(span_words(rlo, a.rowHi[row]), kWarpSpanWords);
    const uint32_t nb = (uint32_t)sw * 32u;
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    const bool rowwise = a.rowP[row] >= (int64_t)kRowwiseMinLen * (e1 - e0);
    int *err = a.err;
    const int32_t *bidx = a.B.idx;
    if (rowwise && b_sorted(a)) {
        int cnt;
        if (interval_union_count(a.A, a.B, a.bRange, e0, e1, lane, &cnt)) {
            if (lane == 0) a.rowNnz[row] = cnt;
            return;
        }
    }
    for (int i = lane; i < sw * 8; i += 32) fw[i] = 0u;
    __syncwarp();
    if (rowwise) {
        // One A entry at a time.  A B row whose columns form one contiguous
        // run (banded and stencil matrices) flags its run a word (4 columns)
        // per lane; any other B row flags a column per lane.
        for (int32_t eb = e0; eb < e1; eb += 32) {
            // Each lane loads its entry's B row bounds and first and last
            // columns up front, so the entries below need no loads of their
            // own before flagging.
            int32_t bs = 0, len = 0, fc = 0, lc = 0;
            if (eb + lane < e1) {
                const int32_t k = a.A.idx[eb + lane];
                bs = a.B.ptr[k];
                len = a.B.ptr[k + 1] - bs;
                if (len > 0) {
                    fc = __ldg(&bidx[bs]);
                    lc = __ldg(&bidx[bs + len - 1]);
                }
            }
            const int n = min(32, e1 - eb);
            for (int q = 0; q < n; ++q) {
                const int32_t bq = __shfl_sync(FULL, bs, q);
                const int32_t lq = __shfl_sync(FULL, len, q);
                const int32_t first = __shfl_sync(FULL, fc, q), last = __shfl_sync(FULL, lc, q);
                if (lq == 0) continue;
                const uint32_t r0 = (uint32_t)(first - base), r1 = (uint32_t)(last - base);
                if (b_sorted(a) && last - first == lq - 1 && r0 < nb && r1 < nb) {
                    for (uint32_t w = (r0 >> 2) + lane; w <= (r1 >> 2); w += 32) {
                        uint32_t m = 0x01010101u;
                        if (w == (r0 >> 2)) m &= 0xffffffffu << (8 * (r0 & 3));
                        if (w == (r1 >> 2)) m &= 0xffffffffu >> (8 * (3 - (r1 & 3)));
                        atomicOr(&fw[w], m);
                    }
                } else {
                    for (int32_t i = lane; i < lq; i += 32) {
                        const uint32_t rel = (uint32_t)(bidx[bq + i] - base);
                        if (in_window(rel, nb, err)) fb[rel] = 1;
                    }
                }
                __syncwarp();
            }
        }
    } else {
        warp_products(a.A, a.B, e0, e1, lane, [&](int32_t j, double) {
            const uint32_t rel = (uint32_t)(bidx[j] - base);
            if (in_window(rel, nb, err)) fb[rel] = 1;
        });
    }
    __syncwarp();
    int cnt = 0;
    for (int i = lane; i < sw * 8; i += 32) cnt += __popc(fw[i]);
    cnt = warp_sum_i(cnt);
    if (lane == 0) a.rowNnz[row] = cnt;
}

template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_sym_flagw(SymArgs a, int32_t begin, int32_t count) {
    sym_flagw_rows<ROWS>(a, begin, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_sym_flagw_dd(SymArgs a, int bin) {
    const int32_t begin = a.binStart[bin], count = a.binStart[bin + 1] - begin;
    for (int64_t vb = blockIdx.x; vb * ROWS < count; vb += gridDim.x) {
        sym_flagw_rows<ROWS>(a, begin, count, vb);
        __syncthreads();
    }
}

// ======================================================================
// Numeric kernels: columns ascending, values in FP64.
// ======================================================================

// Amount subtracted from the columns a row writes (0 unless batched).
__device__ __forceinline__ int32_t col_shift(const NumArgs &a, int32_t row) {
    return a.colShift ? a.colShift[row] : 0;
}

// Tiny rows, numeric: the warp then writes its rows' entries as one flat run, 32
// consecutive ones a step, so that rows next to each other in C go out in whole
// sectors.
__device__ __forceinline__ void num_tiny_rows(const NumArgs &a, int32_t lo, int32_t count, int64_t vb) {
    __shared__ double vals[kNumTinyWarps][kTinyWords];
    __shared__ int32_t cols[kNumTinyWarps][kTinyWords];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int64_t item = (vb * kNumTinyWarps + g) * 32 + lane;
    const bool live = item < count;
    const int32_t row = live ? a.list[lo + item] : 0;
    int32_t *col = cols[g] + lane;
    double *val = vals[g] + lane;
    const int listed = tiny_list<true>(a.A, a.B, row, live, col, val);
    const int most = __reduce_max_sync(FULL, listed);
    const int32_t cbase = live ? a.rowLo[row] : 0;
    const int32_t shift = live ? col_shift(a, row) : 0;
    int m;
    if (__any_sync(FULL, live && listed > 0 && (int64_t)a.rowHi[row] - cbase >= (1 << 27)))
        m = tiny_sum_wide(a.B, listed, shift, col, val);
    else if (most <= 8)
        m = tiny_sum<8>(a.B, listed, cbase, shift, col, val);
    else if (most <= 16)
        m = tiny_sum<16>(a.B, listed, cbase, shift, col, val);
    else
        m = tiny_sum<kTinyMax>(a.B, listed, cbase, shift, col, val);
    int64_t base = 0;
    int n = 0;
    if (live) {
        const int64_t c0 = a.Cp[row];
        const int64_t expect = a.Cp[row + 1] - c0;
        if (m != expect) raise(a.err, DEV_COUNT_MISMATCH);
        n = (int)min((int64_t)m, expect);
        base = c0 - a.outBase;
    }
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += y;
    }
    const int start = incl - n;
    base -= start;  // entry t of the run goes to its row's base + t
    const int total = __shfl_sync(FULL, incl, 31);
    // Consecutive rows share their base, and lanes with entries lead the warp
    // as a rule: entry t is then of the lane that the starts up to t count to
    // (2.1M rows 408 -> 393 us against the search and its shuffles).
    const unsigned have = __ballot_sync(FULL, n > 0);
    const int64_t base0 = __shfl_sync(FULL, base, 0);
    const bool plain = (have & (have + 1u)) == 0u && __all_sync(FULL, n == 0 || base == base0);
    __syncwarp();
    int seen = 0, before = 0;  // rows that start before the step, and where the last of them does
    for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int o, first;
        int64_t to = base0 + t;
        if (plain) {
            const uint32_t at = n > 0 ? (uint32_t)(start - t0) : 32u;
            const uint32_t starts = __reduce_or_sync(FULL, at < 32u ? 1u << at : 0u);
            const uint32_t upto = starts & (FULL >> (31 - lane));
            o = seen + __popc(upto) - 1;
            first = upto ? t0 + 31 - __clz(upto) : before;
            seen += __popc(starts);
            if (starts) before = t0 + 31 - __clz(starts);
        } else {
            o = 0;  // the lane whose row holds entry t
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const int v = __shfl_sync(FULL, incl, o + step - 1);
                if (v <= t) o += step;
            }
            first = __shfl_sync(FULL, start, o);
            to = __shfl_sync(FULL, base, o) + t;
        }
        if (t < total) {
            const int at = kTinyPitch * (t - first) + o;
            a.Ci[to] = cols[g][at];
            a.Cv[to] = vals[g][at];
        }
    }
}

__global__ void __launch_bounds__(32 * kNumTinyWarps) k_num_tiny(NumArgs a, int32_t lo, int32_t count) {
    num_tiny_rows(a, lo, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
__global__ void __launch_bounds__(32 * kNumTinyWarps) k_num_tiny_dd(NumArgs a, int bin) {
    const int32_t lo = a.binStart[bin], count = a.binStart[bin + 1] - lo;
    for (int64_t vb = blockIdx.x; vb * (32 * kNumTinyWarps) < count; vb += gridDim.x) {
        num_tiny_rows(a, lo, count, vb);
        __syncthreads();
    }
}

// Bitonic sort of buf[0, N) ascending by GROUP threads (N a power of two).
template <int GROUP, int ROWS>
__device__ __forceinline__ void group_bitonic(uint64_t *buf, int N, int gt) {
    for (int k = 2; k <= N; k <<= 1) {
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
            for (int i = gt; i < N; i += GROUP) {
                const int ixj = i ^ jj;
                if (ixj > i) {
                    const uint64_t x = buf[i], y = buf[ixj];
                    const bool up = (i & k) == 0;
                    if ((x > y) == up) {
                        buf[i] = y;
                        buf[ixj] = x;
                    }
                }
            }
            group_sync<GROUP, ROWS>();
        }
    }
}

// Compacts the occupied slots of a (keys, vals) table into sbuf (which
// aliases keys) as packed (column, slot) pairs, sorts them and writes the
// row.  GROUP threads per row; all of them call.
template <int GROUP, int ROWS, int TABLE>
__device__ __forceinline__ void table_write_sorted(const NumArgs &a, int32_t row, int32_t *keys, const double *vals,
                                                   int *gcnt, int gt) {
    constexpr int KPT = TABLE / GROUP;
    constexpr int NMAX = TABLE / 2;
    const int lane = threadIdx.x & 31;
    uint64_t *sbuf = reinterpret_cast<uint64_t *>(keys);
    int32_t mk[KPT];
#pragma unroll
    for (int q = 0; q < KPT; ++q) mk[q] = keys[gt + q * GROUP];
    group_sync<GROUP, ROWS>();
#pragma unroll
    for (int q = 0; q < KPT; ++q) {
        const bool occ = mk[q] != EMPTY;
        const unsigned bal = __ballot_sync(FULL, occ);
        int wbase = 0;
        if (lane == 0 && bal) wbase = atomicAdd(gcnt, __popc(bal));
        wbase = __shfl_sync(FULL, wbase, 0);
        if (occ) {
            const int pos = wbase + __popc(bal & ((1u << lane) - 1u));
            if (pos < NMAX) sbuf[pos] = ((uint64_t)(uint32_t)mk[q] << 32) | (uint32_t)(gt + q * GROUP);
        }
    }
    group_sync<GROUP, ROWS>();
    const int n = *gcnt;
    const int64_t expect = a.Cp[row + 1] - a.Cp[row];
    if (gt == 0 && (n != expect || n > NMAX)) raise(a.err, DEV_COUNT_MISMATCH);
    const int nn = min(n, NMAX);
    int N = 1;
    while (N < nn) N <<= 1;
    for (int i = nn + gt; i < N; i += GROUP) sbuf[i] = ~0ull;
    group_sync<GROUP, ROWS>();
    group_bitonic<GROUP, ROWS>(sbuf, N, gt);
    const int64_t obase = a.Cp[row] - a.outBase;
    const int32_t shift = col_shift(a, row);
    const int wn = (int)min((int64_t)nn, expect);
    for (int i = gt; i < wn; i += GROUP) {
        const uint64_t v = sbuf[i];
        a.Ci[obase + i] = (int32_t)(v >> 32) - shift;
        a.Cv[obase + i] = vals[(uint32_t)v];
    }
}

// Shared bytes per warp of the warp hash kernel: keys and values (which rows
// sorted in registers use for their products) and those rows' entries.  6.5 KB
// per warp.
constexpr size_t warp_hash_bytes(int table) { return 13 * (size_t)table; }

// Sorts 32 R keys ascending over a warp's registers: key[r] of lane l is the
// (R l + r)-th afterwards.  Each lane sorts its own R (merge_exchange); then
// runs of neighbouring lanes are merged: the first step of a merge compares
// mirrored positions, the others positions one stride apart (Batcher's
// bitonic merge, all comparators the same way round), strides of R and more
// by shuffles, shorter ones inside the lane.  R need not be a power of two: the
// runs' lengths halve down to a lane's R, which it sorts again.
template <int R, class K>
__device__ __forceinline__ void warp_sort(K (&key)[R]) {
    const int lane = threadIdx.x & 31;
    merge_exchange<R, 1, 1>(key);
#pragma unroll
    for (int m = 2; m <= 32; m <<= 1) {  // runs of m lanes
        K other[R];
#pragma unroll
        for (int r = 0; r < R; ++r) other[r] = __shfl_xor_sync(FULL, key[R - 1 - r], m - 1);
        // The lower lane keeps the smaller key: one compare against the lane's
        // side and one select (a minimum, a maximum and a select otherwise).
        const bool low = (lane & (m >> 1)) == 0;
#pragma unroll
        for (int r = 0; r < R; ++r) key[r] = (other[r] < key[r]) == low ? other[r] : key[r];
#pragma unroll
        for (int d = m >> 2; d >= 1; d >>= 1) {
            const bool lo = (lane & d) == 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const K x = __shfl_xor_sync(FULL, key[r], d);
                key[r] = (x < key[r]) == lo ? x : key[r];
            }
        }
        if constexpr ((R & (R - 1)) == 0) {
#pragma unroll
            for (int d = R >> 1; d >= 1; d >>= 1) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if ((r & d) == 0) {
                        const K lo = min(key[r], key[r + d]), hi = max(key[r], key[r + d]);
                        key[r] = lo;
                        key[r + d] = hi;
                    }
                }
            }
        } else {
            merge_exchange<R, 1, 1>(key);
        }
    }
}

// Where a warp keeps entry p of up to 256 it writes R consecutive ones a lane
// and reads 32 consecutive ones a step: rotated by p / 32 in its group of 32,
// so that neither hits a bank more than twice.
__device__ __forceinline__ int rotated(int p) { return (p & ~31) | ((p + (p >> 5)) & 31); }

// Rows of at most kEscMax products by one warp without a hash table (expand,
// sort, compress): every product's value goes to shared memory (esc_list) and
// its (column, product) key is sorted in registers, 32 R of them (esc_sort,
// warp_sort), which puts equal columns next to each other in Gustavson order.
// A lane sums the runs inside its R keys; a run over several lanes is finished
// by the lane that holds its first key, from the others' leading sums.  The
// row's entries are gathered in shared memory and written 32 consecutive ones
// a step.
//
// A bucket counting sort in shared memory with each lane writing R
// consecutive entries, the form before, was bound by the L1: 60M bank
// conflicts and 20M store requests for 100k rows of 256 products (91% of L1
// throughput busy): 455 -> 190 us, 550k rows of about 144 products 1611 ->
// 954 us.  What bounds it now is instruction issue (65% busy, the ALU 68%) and
// latency, at 32 warps an SM (64 registers, 6 KB a warp; at 92 registers and
// 20 warps 272 us).  kbuf and pv hold a product each; columns lie in
// [rlo, rlo + 2^(bits of K - kEscShift)).
//
// SHIFT is the bits of a product's number in its key.  With ent (rows past
// kEscMax products, of at most 256 entries) pv takes the B values and ent the
// products' entries, for esc_fused.
template <int SHIFT, class K>
__device__ __forceinline__ void esc_list(const NumArgs &a, int32_t e0, int32_t e1, int n, int32_t rlo, K *kbuf,
                                         double *pv, uint8_t *ent) {
    const int lane = threadIdx.x & 31;
    int32_t tb = 0;  // products of the earlier chunks
    if (n >= kEscGroupLen * (e1 - e0)) {
        // Eight lanes an entry, two entries a group and two products of each
        // a lane in flight: no search for a product's entry.
        const int sub = lane & 7, grp = lane >> 3;
        for (int32_t e = e0; e < e1; e += 32) {
            const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
            const int32_t ex = tb + c.incl - c.len;
            const int ne = min(32, e1 - e);
            for (int q = 0; q < ne; q += 8) {
                int32_t at[2], t[2], len[2];
                double av[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int o = q + 4 * h + grp;  // lanes past the chunk's entries hold none
                    at[h] = __shfl_sync(FULL, c.bs, o);
                    len[h] = __shfl_sync(FULL, c.len, o);
                    t[h] = __shfl_sync(FULL, ex, o);
                    av[h] = __shfl_sync(FULL, c.a, o);
                    len[h] = min(len[h], n - t[h]);
                }
                const int32_t most = max(len[0], len[1]);
                for (int32_t i0 = sub; i0 < most; i0 += 16) {
                    int32_t col[4];
                    double bv[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int h = u >> 1, i = i0 + 8 * (u & 1);
                        col[u] = i < len[h] ? __ldg(&a.B.idx[at[h] + i]) : 0;
                        bv[u] = i < len[h] ? __ldg(&a.B.val[at[h] + i]) : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int h = u >> 1, i = i0 + 8 * (u & 1);
                        if (i < len[h]) {
                            const int x = t[h] + i;
                            kbuf[x] = (K)(uint32_t)(col[u] - rlo) << SHIFT | (K)x;
                            pv[x] = ent ? bv[u] : __dmul_rn(av[h], bv[u]);
                            if (ent) ent[x] = (uint8_t)(e - e0 + q + 4 * h + grp);
                        }
                    }
                }
            }
            tb += c.total;
        }
    } else {
        constexpr int U = 4;  // steps of B loads in flight
        for (int32_t e = e0; e < e1; e += 32) {
            const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
            for (int32_t t0 = 0; t0 < c.total; t0 += 32 * U) {
                int32_t j[U], own[U];
                double av[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    j[u] = -1;
                    av[u] = 0.0;
                    own[u] = 0;
                    const int32_t t = t0 + 32 * u + lane;
                    if (t0 + 32 * u < c.total) {
                        const int32_t jj = chunk_pos(c, t, &av[u], &own[u]);
                        if (t < c.total && tb + t < n) j[u] = jj;
                    }
                }
                int32_t col[U];
                double bv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    col[u] = j[u] >= 0 ? __ldg(&a.B.idx[j[u]]) : 0;
                    bv[u] = j[u] >= 0 ? __ldg(&a.B.val[j[u]]) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (j[u] >= 0) {
                        const int t = tb + t0 + 32 * u + lane;
                        kbuf[t] = (K)(uint32_t)(col[u] - rlo) << SHIFT | (K)t;
                        pv[t] = ent ? bv[u] : __dmul_rn(av[u], bv[u]);
                        if (ent) ent[t] = (uint8_t)(e - e0 + own[u]);
                    }
                }
            }
            tb += c.total;
        }
    }
    __syncwarp();
}

template <int R, class K>
__device__ __forceinline__ void esc_sort(const NumArgs &a, int32_t row, int n, int32_t rlo, K *kbuf, double *pv) {
    constexpr int SHIFT = kEscShift;
    constexpr K NONE = ~K(0);
    const int lane = threadIdx.x & 31;
    K key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) key[r] = 32 * r + lane < n ? kbuf[32 * r + lane] : NONE;
    warp_sort<R>(key);
    // Values, and which keys start a column's run.
    double v[R];
    uint32_t heads = 0;
    const K before = __shfl_up_sync(FULL, key[R - 1], 1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool valid = R * lane + r < n;
        v[r] = valid ? pv[min((int)(key[r] & (K)((1 << SHIFT) - 1)), 32 * R - 1)] : 0.0;
        const K prev = r > 0 ? key[r > 0 ? r - 1 : 0] : before;
        if (valid && ((r == 0 && lane == 0) || (key[r] >> SHIFT) != (prev >> SHIFT))) heads |= 1u << r;
    }
    __syncwarp();
    // Sums of the runs in this lane, each left in its last key's v: lead is
    // the part of an earlier lane's run, the run of the last head may go on.
    double lead = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool more = R * lane + r < n && !((heads >> r) & 1u);
        if (!__any_sync(FULL, more)) continue;  // an addition takes the FP64 pipe 16 clocks, needed or not
        if (more) {
            if ((heads & ((1u << r) - 1u)) == 0u) lead += v[r];
            else v[r] += v[r > 0 ? r - 1 : 0];
        }
    }
    // Lanes whose last key's run goes on take the following lanes' leads.
    const bool leads = R * lane < n && !(heads & 1u);  // this lane starts inside a run
    const unsigned goOn = __ballot_sync(FULL, leads);
    const unsigned bare = __ballot_sync(FULL, heads == 0u);
    double more = 0.0;
    bool open = heads != 0u && lane < 31 && ((goOn >> (lane + 1)) & 1u);
    const bool goesOn = open;
    for (int d = 1; __any_sync(FULL, open); ++d) {
        const double x = __shfl_down_sync(FULL, lead, d);
        if (open) {
            more += x;
            open = lane + d < 31 && ((bare >> (lane + d)) & 1u) && ((goOn >> (lane + d + 1)) & 1u);
        }
    }
    // Ranks, then the row gathered in order.
    const int mine = __popc(heads);
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += y;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    const int64_t obase = a.Cp[row] - a.outBase;
    const int64_t expect = a.Cp[row + 1] - a.Cp[row];
    if (lane == 0 && total != expect) raise(a.err, DEV_COUNT_MISMATCH);
    int32_t *cbuf = reinterpret_cast<int32_t *>(kbuf);
    int p = incl - mine;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if ((heads >> r) & 1u) cbuf[rotated(p++)] = (int32_t)(key[r] >> SHIFT);
        // The run's last key in this lane: the next one is a head or there is none.
        const bool ends = R * lane + r < n && (r == R - 1 || R * lane + r + 1 >= n || ((heads >> (r + 1)) & 1u));
        if (ends && (heads & ((2u << r) - 1u))) {
            if (goesOn && p == incl) v[r] += more;
            pv[rotated(p - 1)] = v[r];
        }
    }
    __syncwarp();
    const int32_t shift = col_shift(a, row) - rlo;
    const int wn = (int)min((int64_t)total, expect);
    for (int i = lane; i < wn; i += 32) {
        a.Ci[obase + i] = cbuf[rotated(i)] - shift;
        a.Cv[obase + i] = pv[rotated(i)];
    }
}

// The same for rows of kEscMax to kFusedMax products, whose columns have several
// products by necessity (they hold at most kNumWarpMax entries): every sum is one
// chain of fused multiply-adds, as in the table.  A lane sums the runs that
// start in it; where its keys begin inside a run it goes on from the sum of the
// lane before, once that one has it.  20k rows of about 400 products 323 us by
// the table, 121 so (143 with rounded products).
__device__ __forceinline__ void esc_fused(const NumArgs &a, int32_t row, int32_t e0, int n, int32_t rlo, uint32_t *kbuf,
                                          double *pv, const uint8_t *ent) {
    constexpr int R = kFusedMax / 32, SHIFT = kFusedShift;
    const int lane = threadIdx.x & 31;
    uint32_t key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) key[r] = 32 * r + lane < n ? kbuf[32 * r + lane] : ~0u;
    warp_sort<R>(key);
    const int have = min(max(n - R * lane, 0), R);  // this lane's keys
    uint32_t heads = 0;
    const uint32_t before = __shfl_up_sync(FULL, key[R - 1], 1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t prev = r > 0 ? key[r > 0 ? r - 1 : 0] : before;
        if (r < have && ((r == 0 && lane == 0) || (key[r] >> SHIFT) != (prev >> SHIFT))) heads |= 1u << r;
    }
    const int first = heads ? __ffs(heads) - 1 : have;  // keys before it continue the run of the lane before
    const int begins = __shfl_down_sync(FULL, first > 0 ? 1 : 0, 1);
    const bool goesOn = lane < 31 && begins;  // the last run does, in the next lane
    const int mine = __popc(heads);
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += y;
    }
    const int64_t obase = a.Cp[row] - a.outBase;
    const int32_t expect = (int32_t)(a.Cp[row + 1] - a.Cp[row]);
    if (lane == 31 && incl != expect) raise(a.err, DEV_COUNT_MISMATCH);
    const int32_t shift = col_shift(a, row) - rlo;
    auto fused = [&](uint32_t k, double acc) {
        const int x = (int)(k & ((1u << SHIFT) - 1u));
        return __fma_rn(__ldg(&a.A.val[e0 + ent[x]]), pv[x], acc);
    };
    // Entries go out lane by lane: such rows are few (a batch's tail), and the
    // registers and shared memory for their order would be every row's.
    int p = incl - mine;
    double acc = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r < first || r >= have) continue;
        const bool head = (heads >> r) & 1u;
        acc = fused(key[r], head ? 0.0 : acc);
        if (head && p < expect) a.Ci[obase + p] = (int32_t)(key[r] >> SHIFT) - shift;
        p += head;
        const bool ends = r + 1 == have ? !goesOn : ((heads >> (r + 1)) & 1u) != 0u;
        if (ends && p <= expect) a.Cv[obase + p - 1] = acc;
    }
    bool wait = first > 0;
    bool known = !wait || heads != 0u;  // the sum so far of this lane's last run
    while (__any_sync(FULL, wait)) {
        const double from = __shfl_up_sync(FULL, acc, 1);
        const bool ready = __shfl_up_sync(FULL, known ? 1 : 0, 1);
        if (!wait || !ready) continue;
        double lead = from;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r < first) lead = fused(key[r], lead);
        if (heads == 0u) acc = lead;
        if ((heads != 0u || !goesOn) && incl - mine <= expect) a.Cv[obase + incl - mine - 1] = lead;
        known = true;
        wait = false;
    }
}

template <int ROWS, int TABLE>
__device__ __forceinline__ void num_hash_warp_rows(const NumArgs &a, int32_t lo, int32_t count, int64_t vb) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int gcnt[ROWS];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)vb * ROWS + g;
    if (item >= count) return;
    unsigned char *base_ptr = smem + (size_t)g * warp_hash_bytes(TABLE);
    int32_t *keys = reinterpret_cast<int32_t *>(base_ptr);
    double *vals = reinterpret_cast<double *>(base_ptr + 4 * (size_t)TABLE);
    const int32_t row = a.list[lo + item];
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    // Expand-sort-compress where the products fit the registers and the
    // columns the keys; the table takes the others.
    static_assert(TABLE >= 2 * kEscMax && TABLE >= kFusedMax && (1 << kEscShift) >= kEscMax &&
                      (1 << kFusedShift) >= kFusedMax, "the arrays and keys hold the products");
    const int64_t P = a.rowP[row];
    const int32_t rlo = a.rowLo[row];
    const int64_t span = (int64_t)a.rowHi[row] - rlo + 1;
    uint32_t *kb = reinterpret_cast<uint32_t *>(keys);
    if (P <= kEscMax) {
        // Two sizes and one listing: warps of an SM that run different code
        // miss the instruction cache.  550k rows of 60 to 280 products: 0.95 ms;
        // with six sizes of 2 to 16 keys a lane, each with its own listing,
        // 2.05 ms.
        if (span < ((int64_t)1 << (32 - kEscShift))) {
            esc_list<kEscShift, uint32_t>(a, e0, e1, (int)P, rlo, kb, vals, nullptr);
            if (P <= 192) esc_sort<6, uint32_t>(a, row, (int)P, rlo, kb, vals);
            else esc_sort<8, uint32_t>(a, row, (int)P, rlo, kb, vals);
        } else {
            unsigned long long *kb64 = reinterpret_cast<unsigned long long *>(keys);
            esc_list<kEscShift, unsigned long long>(a, e0, e1, (int)P, rlo, kb64, vals, nullptr);
            esc_sort<8, unsigned long long>(a, row, (int)P, rlo, kb64, vals);
        }
        return;
    }
    if (P <= kFusedMax && e1 - e0 <= 256 && span < ((int64_t)1 << (32 - kFusedShift))) {
        uint8_t *ent = reinterpret_cast<uint8_t *>(vals + TABLE);
        esc_list<kFusedShift, uint32_t>(a, e0, e1, (int)P, rlo, kb, vals, ent);
        esc_fused(a, row, e0, (int)P, rlo, kb, vals, ent);
        return;
    }
    for (int i = lane; i < TABLE; i += 32) {
        keys[i] = EMPTY;
        vals[i] = 0.0;
    }
    if (lane == 0) gcnt[g] = 0;
    __syncwarp();
    for (int32_t e = e0; e < e1; e += 32) {
        const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
        // kHashWarpLoads steps at a time: positions first, then all their B
        // loads, then the inserts.
        for (int32_t t0 = 0; t0 < c.total; t0 += 32 * kHashWarpLoads) {
            int32_t j[kHashWarpLoads], col[kHashWarpLoads];
            double av[kHashWarpLoads], bv[kHashWarpLoads];
#pragma unroll
            for (int u = 0; u < kHashWarpLoads; ++u) {
                j[u] = -1;
                av[u] = 0.0;
                const int32_t t = t0 + 32 * u + lane;
                if (t0 + 32 * u < c.total) {
                    const int32_t jj = chunk_pos(c, t, &av[u]);
                    if (t < c.total) j[u] = jj;
                }
            }
#pragma unroll
            for (int u = 0; u < kHashWarpLoads; ++u) {
                col[u] = j[u] >= 0 ? __ldg(&a.B.idx[j[u]]) : 0;
                bv[u] = j[u] >= 0 ? __ldg(&a.B.val[j[u]]) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kHashWarpLoads; ++u) {
                if (j[u] >= 0) {
                    const int s = hash_insert_slot<TABLE>(keys, col[u], a.err);
                    if (s >= 0) atomic_fma(&vals[s], av[u], bv[u]);
                }
            }
        }
    }
    __syncwarp();
    table_write_sorted<32, ROWS, TABLE>(a, row, keys, vals, &gcnt[g], lane);
}

template <int ROWS, int TABLE>
__global__ void __launch_bounds__(32 * ROWS, 8) k_num_hash_warp(NumArgs a, int32_t lo, int32_t count) {
    num_hash_warp_rows<ROWS, TABLE>(a, lo, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int ROWS, int TABLE>
__global__ void __launch_bounds__(32 * ROWS, 8) k_num_hash_warp_dd(NumArgs a, int bin) {
    const int32_t lo = a.binStart[bin], count = a.binStart[bin + 1] - lo;
    for (int64_t vb = blockIdx.x; vb * ROWS < count; vb += gridDim.x) {
        num_hash_warp_rows<ROWS, TABLE>(a, lo, count, vb);
        __syncthreads();
    }
}

// CTA hash rows: one CTA per row, products spread over all threads.
template <int THREADS, int TABLE>
__device__ __forceinline__ void num_hash_cta_rows(const NumArgs &a, int32_t lo, int64_t vb) {
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    __shared__ int32_t sh[THREADS / 32];
    __shared__ int gcnt;
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    double *av = reinterpret_cast<double *>(smem + L::av);
    int32_t *keys = reinterpret_cast<int32_t *>(smem + L::bytes);
    double *vals = reinterpret_cast<double *>(smem + L::bytes + 4 * (size_t)TABLE);
    const int tid = threadIdx.x;
    const int32_t row = a.list[lo + vb];
    for (int i = tid; i < TABLE; i += THREADS) {
        keys[i] = EMPTY;
        vals[i] = 0.0;
    }
    if (tid == 0) gcnt = 0;
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    for (int32_t eb = e0; eb < e1; eb += THREADS) {
        int nb;
        const int32_t total =
            stage_entries<THREADS, true>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, av, &nb, sh);
        int32_t tb, te;
        warp_share<THREADS>(total, &tb, &te);
        warp_range_ld<4>(
            pre, bst, nb, tb, te,
            [&](int32_t pos) { return ColVal{__ldg(&a.B.idx[pos]), __ldg(&a.B.val[pos])}; },
            [&](bool v, const ColVal &x, int e) {
                if (v) {
                    const int s = hash_insert_slot<TABLE>(keys, x.c, a.err);
                    if (s >= 0) atomic_fma(&vals[s], av[e], x.v);
                }
            });
        __syncthreads();
    }
    table_write_sorted<THREADS, 1, TABLE>(a, row, keys, vals, &gcnt, tid);
}

template <int THREADS, int TABLE>
__global__ void __launch_bounds__(THREADS) k_num_hash_cta(NumArgs a, int32_t lo) {
    num_hash_cta_rows<THREADS, TABLE>(a, lo, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int THREADS, int TABLE>
__global__ void __launch_bounds__(THREADS) k_num_hash_cta_dd(NumArgs a, int bin) {
    const int32_t lo = a.binStart[bin], count = a.binStart[bin + 1] - lo;
    for (int64_t vb = blockIdx.x; vb < count; vb += gridDim.x) {
        num_hash_cta_rows<THREADS, TABLE>(a, lo, vb);
        __syncthreads();
    }
}

// Rank rows (windows of at most 2^18 columns): one CTA per row.  The row's
// columns are bits of a shared bitmap over its window (kept by the symbolic
// pass, or set here by a pass over the products); a scan of the words' counts
// ranks every pair of words, which gives a column's position in C's row by
// one 64-bit load and a bit count.  Columns are written balanced by position,
// and a pass over the products adds each one at its rank.  No hashing, no
// sorting.
//
// P is the type of the pairs' ranks: 16 bits for the rows of the small CTAs
// (at most kNumCtaLMax entries).  Their sums are fused multiply-adds in shared
// memory (compare-and-swap loops), kRankVals entries a pass over the products,
// written out in whole sectors; with 75 KB a CTA at the widest window three of
// them share an SM, five at 2^16 columns.  The compare-and-swap loops bound
// them: four of a lane's in flight together, or more CTAs of a smaller
// kRankVals, are no faster (57k rows of R-MAT 2^18 1.99 ms; 2.02 and 2.19), and
// 384 or 512 threads a CTA are slower (2.19, 2.49).  The same rows reduced into
// C in place, as the large ones are, take 1.36 ms but round every product
// before it is added: 0.64 units of the last place instead of 0.56 (rms, R-MAT
// 2^14, against exact sums).  57k rows of 2^18 3.13 ms before the ranks were 16
// bits and taken by warp steps, 18k of 2^16 0.75 -> 0.39.
//
// The larger rows (512 threads, two CTAs an SM) add into C in place by FP64
// reductions at L2 and are bound by the reductions' 25 sectors a step and
// by what of C and B stays in L2 meanwhile: C's values are zeroed right before
// the products, not earlier (33k rows of 2^18 4.76 -> 4.60 ms; 5.01 with the
// ranks a group of words a thread), and a third CTA an SM, which 2^16 gains
// 3% from, costs 2^18 6%.
constexpr int kRankSThreads = 256;  // rows of at most tune.rankSharedMax entries
constexpr int kRankLThreads = 512;
constexpr int kRankVals = 3960;  // with 2^18 columns, a third of an SM's shared memory
// CTAs an SM is to hold: 48 registers a thread for the small ones.
__host__ __device__ constexpr int rank_ctas(int threads) { return threads == kRankSThreads ? 5 : 2; }

// Where the rank kernel's bitmap starts behind the staging area.
__host__ __device__ constexpr size_t rank_bits_at(int threads) {
    const size_t staged =
        threads == kRankSThreads ? StageLayout<kRankSThreads>::bytes : StageLayout<kRankLThreads>::bytes;
    return staged / 16 * 16 + 16;
}

template <int THREADS, class P>
__device__ __forceinline__ void num_rank_rows(const NumArgs &a, int32_t lo, int maxWords, int64_t vb) {
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    constexpr int NW = THREADS / 32;
    __shared__ int32_t sh[NW];
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    double *av = reinterpret_cast<double *>(smem + L::av);
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem + rank_bits_at(THREADS));
    constexpr bool kShared = sizeof(P) == 2;  // the row's values in shared memory
    double *vals = reinterpret_cast<double *>(bits + maxWords);
    P *pairRank = reinterpret_cast<P *>(bits + maxWords + (kShared ? 2 * kRankVals : 0));
    // Per group of words, the rank of its first column and its non-empty
    // words, kept in the staging area (idle between the passes).
    static_assert(8 * THREADS <= L::bytes && kRankWordsMax <= 32 * THREADS, "rank groups");
    int32_t *tbase = pre;
    uint32_t *tmask = reinterpret_cast<uint32_t *>(pre + THREADS);
    const int tid = threadIdx.x;
    const int32_t row = a.list[lo + vb];
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    const int32_t expect = (int32_t)(a.Cp[row + 1] - a.Cp[row]);  // at most the window's 2^18 columns
    const int64_t obase = a.Cp[row] - a.outBase;
    // The row's window: words [rw0, rw0 + nwords) of C's columns.
    const int32_t rlo = a.rowLo[row];
    const int32_t rw0 = rlo >> 5;
    const int nwords = min(span_words(rlo, a.rowHi[row]), maxWords);
    const int32_t cbase = rw0 << 5;
    const int32_t obc = cbase - col_shift(a, row);  // column written for bit 0
    double *cv = a.Cv + obase;

    const bool kept = a.wideBits && sym_bin_of(a.rowP[row], e1 - e0, nwords, a.tune) == SB_WIDE;
    if (!kept) {
        for (int i = tid; 4 * i < nwords; i += THREADS) reinterpret_cast<uint4 *>(bits)[i] = make_uint4(0u, 0u, 0u, 0u);
        for (int32_t eb = e0; eb < e1; eb += THREADS) {
            int nb;
            const int32_t total =
                stage_entries<THREADS, false>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, nullptr, &nb, sh);
            int32_t tb, te;
            warp_share<THREADS>(total, &tb, &te);
            warp_range_ld<4>(
                pre, bst, nb, tb, te, [&](int32_t pos) { return __ldg(&a.B.idx[pos]); },
                [&](bool v, int32_t col, int) {
                    const uint32_t rel = v ? (uint32_t)(col - cbase) : 0u;
                    or_bit(bits, v && in_window(rel, (uint32_t)nwords * 32u, a.err), rel);
                });
            __syncthreads();
        }
    }

    // A warp ranks 32 groups of wpt words (a power of two of at least 4 with
    // THREADS * wpt >= nwords), 128 consecutive words a step, four a lane.
    // (With a group a thread, wide windows pay 8- and 16-way bank conflicts
    // at each load and store: 57k rows of 2^18 1.74 ms instead of 1.39.)
    int wpt = 4, lg = 2;
    while (wpt * THREADS < nwords) wpt <<= 1, ++lg;
    const int lane = tid & 31, n4 = wpt >> 2;
    const int w0 = (tid >> 5) * 32 * wpt + 4 * lane;
    int32_t cnt = 0;
    const uint32_t *src = kept ? a.wideBits + (size_t)a.wideSlot[row] * kRankWordsMax : nullptr;
#pragma unroll 4
    for (int j = 0; j < n4; ++j) {
        const int i = w0 + 128 * j;
        if (i < nwords) {
            uint4 v;
            if (kept) {
                v = __ldcs(reinterpret_cast<const uint4 *>(src + i));
                // Words past the window hold another row's bits.
                if (i + 1 >= nwords) v.y = 0u;
                if (i + 2 >= nwords) v.z = 0u;
                if (i + 3 >= nwords) v.w = 0u;
                *reinterpret_cast<uint4 *>(bits + i) = v;
            } else {
                v = *reinterpret_cast<const uint4 *>(bits + i);
            }
            cnt += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
    }
    int32_t tot;
    int32_t run = __shfl_sync(FULL, block_excl_scan<THREADS>(cnt, &tot, sh), 0);
    if (tid == 0 && tot != expect) raise(a.err, DEV_COUNT_MISMATCH);
#pragma unroll 2
    for (int j = 0; j < n4; ++j) {
        const int i = w0 + 128 * j;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (i < nwords) v = *reinterpret_cast<const uint4 *>(bits + i);
        const int32_t c2 = __popc(v.x) + __popc(v.y), c4 = c2 + __popc(v.z) + __popc(v.w);
        int32_t x = c4;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t y = __shfl_up_sync(FULL, x, d);
            if (lane >= d) x += y;
        }
        const int32_t p = run + x - c4;
        run += __shfl_sync(FULL, x, 31);
        if (i < nwords) {
            pairRank[i >> 1] = (P)p;
            pairRank[(i >> 1) + 1] = (P)(p + c2);
        }
        uint32_t mask = ((v.x ? 1u : 0u) | (v.y ? 2u : 0u) | (v.z ? 4u : 0u) | (v.w ? 8u : 0u))
                        << (4 * (lane & (n4 - 1)));
        for (int d = 1; d < n4; d <<= 1) mask |= __shfl_xor_sync(FULL, mask, d);
        if ((lane & (n4 - 1)) == 0) {
            tbase[i >> lg] = p;
            tmask[i >> lg] = mask;
        }
    }
    __syncthreads();
    write_columns_balanced<THREADS>(bits, tbase, tmask, wpt, tot, a.Ci + obase, expect, obc);
    // Every product, as add(its rank, A value, B value).
    auto products = [&](auto &&add) {
        for (int32_t eb = e0; eb < e1; eb += THREADS) {
            int nb;
            const int32_t total =
                stage_entries<THREADS, true>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, av, &nb, sh);
            int32_t tb, te;
            warp_share<THREADS>(total, &tb, &te);
            warp_range_ld<4>(
                pre, bst, nb, tb, te,
                [&](int32_t pos) { return ColVal{__ldg(&a.B.idx[pos]), __ldg(&a.B.val[pos])}; },
                [&](bool v, const ColVal &x, int e) {
                    const uint32_t c = (uint32_t)(x.c - cbase);
                    if (v && c < (uint32_t)nwords * 32u) {
                        const uint2 word = *reinterpret_cast<const uint2 *>(bits + (c >> 6) * 2u);
                        const uint32_t below = (1u << (c & 31u)) - 1u;
                        add((uint32_t)pairRank[c >> 6] + ((c & 32u) ? __popc(word.x) + __popc(word.y & below)
                                                                    : __popc(word.x & below)),
                            av[e], x.v);
                    }
                });
            __syncthreads();
        }
    };
    if constexpr (kShared) {
        for (int32_t r0 = 0; r0 < expect; r0 += kRankVals) {  // once, but for the largest rows
            const int n = min(expect - r0, kRankVals);
            for (int i = tid; i < n; i += THREADS) vals[i] = 0.0;
            __syncthreads();
            products([&](uint32_t r, double x, double y) {
                r -= (uint32_t)r0;
                if (r < (uint32_t)n) atomic_fma(&vals[r], x, y);
            });
            for (int i = tid; i < n; i += THREADS) cv[r0 + i] = vals[i];
            __syncthreads();
        }
    } else {
        // C's values start at zero.
        for (int i = tid; i < expect; i += THREADS) cv[i] = 0.0;
        __syncthreads();
        products([&](uint32_t r, double x, double y) {
            if (r < (uint32_t)expect) atomicAdd(&cv[r], __dmul_rn(x, y));
        });
    }
}

template <int THREADS, class P>
__global__ void __launch_bounds__(THREADS, rank_ctas(THREADS)) k_num_rank(NumArgs a, int32_t lo, int maxWords) {
    num_rank_rows<THREADS, P>(a, lo, maxWords, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int THREADS, class P>
__global__ void __launch_bounds__(THREADS, rank_ctas(THREADS)) k_num_rank_dd(NumArgs a, int bin, int maxWords) {
    const int32_t lo = a.binStart[bin], count = a.binStart[bin + 1] - lo;
    for (int64_t vb = blockIdx.x; vb < count; vb += gridDim.x) {
        num_rank_rows<THREADS, P>(a, lo, maxWords, vb);
        __syncthreads();
    }
}

// The columns [r0, r1] of a row's window that fall in 32-column word w, as bits.
__device__ __forceinline__ uint32_t run_bits(int w, int r0, int r1) {
    const int lo = max(r0, 32 * w), hi = min(r1, 32 * w + 31);
    return lo <= hi ? (0xffffffffu >> (31 - (hi - lo))) << (lo & 31) : 0u;
}

// Narrowest rows (window of at most kDenseWarpWords words): one warp per row
// with a dense FP64 accumulator and a flag byte per column of the window in
// shared memory.  Row-wise enumeration over strictly ascending B rows adds
// each column's products in A's entry order with plain fused multiply-adds
// (deterministic); otherwise atomic ones.  The flags give the columns in
// order, 32 of them a step: no bitmap ranks, no sorting.
//
// The FP64 pipe bounds it: a warp's multiply-add takes 16 clocks of the SM's,
// however many lanes it has, and taking one A entry at a time gives the 65
// columns of a band's B row three of them where two would nearly do.  Where
// 32 consecutive entries' B rows are each one run of 32 columns or more
// (banded matrices), their products are taken as one flat sequence, 32 a
// step.  A step then holds the end of one run and the start of the next,
// which share no column when the next run starts at least 32 columns before
// the other's end or behind it (checked per chunk); columns and flags follow
// from the runs' ends, so B's indices are not read.  A band's rows take 2.05
// steps an entry instead of 3: 970k rows of 4225 products 10.95 -> 7.86 ms
// (6.5 ms at the pipe's rate).
//
// Few rows leave most of the pipe idle and are bound by a warp's chain of steps:
// up to kDensewFew rows an SM take the products six steps at a time, which,
// where they lie in one entry, share no column and need no order among them
// (512 rows of 512 entries of 512 products 1560 -> 1105 us, 1245 entry by entry;
// 2000 rows of 256 of 256 458 -> 398).  With 5000 such rows that is slower (898
// us instead of 767), the pipe being busy and the registers fewer.
constexpr int kDensewFew = 16;

template <int ROWS, int U>
__device__ __forceinline__ void num_densew_rows(const NumArgs &a, int32_t lo, int32_t count, int64_t vb) {
    constexpr int kCols = kDenseWarpWords * 32;
    __shared__ double vs[ROWS][kCols];
    __shared__ __align__(16) uint32_t fls[ROWS][kCols / 4];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)vb * ROWS + g;
    if (item >= count) return;
    double *vals = vs[g];
    uint32_t *fw = fls[g];
    uint8_t *fb = reinterpret_cast<uint8_t *>(fw);
    const int32_t row = a.list[lo + item];
    const int32_t rlo = a.rowLo[row];
    const int32_t cbase = (rlo >> 5) << 5;
    const int sw = min(span_words(rlo, a.rowHi[row]), kDenseWarpWords);
    const uint32_t nb = (uint32_t)sw * 32u;
    const int64_t expect = a.Cp[row + 1] - a.Cp[row];
    const int64_t obase = a.Cp[row] - a.outBase;
    for (int i = lane; i < (int)nb; i += 32) vals[i] = 0.0;
    for (int i = lane; i < sw * 8; i += 32) fw[i] = 0u;
    __syncwarp();
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    const bool rowwise = a.rowP[row] >= (int64_t)kRowwiseMinLen * (e1 - e0);
    const bool plain = rowwise && b_sorted(a);
    int *err = a.err;
    const int32_t *bidx = a.B.idx;
    const double *bval = a.B.val;
    uint32_t runs = 0u;  // word `lane` of the window: columns of the runs taken flat
    auto add = [&](uint32_t rel, double av, double bv) {
        if (in_window(rel, nb, err)) {
            if (plain) vals[rel] = __fma_rn(av, bv, vals[rel]);
            else atomic_fma(&vals[rel], av, bv);
            fb[rel] = 1;
        }
    };
    if (rowwise) {
        for (int32_t eb = e0; eb < e1; eb += 32) {
            int32_t bs = 0, len = 0, first = 0, last = -1;  // the B row and its run's ends in the window
            double avl = 0.0;
            if (eb + lane < e1) {
                const int32_t k = a.A.idx[eb + lane];
                bs = a.B.ptr[k];
                len = a.B.ptr[k + 1] - bs;
                avl = a.A.val[eb + lane];
                if (plain && len > 0) {
                    first = __ldg(&bidx[bs]) - cbase;
                    last = __ldg(&bidx[bs + len - 1]) - cbase;
                }
            }
            const int n = min(32, e1 - eb);
            bool flat = plain;
            if (plain) {
                const int d = __shfl_down_sync(FULL, first, 1) - first;
                const bool run = len >= 32 && last - first == len - 1 && first >= 0 && last < (int)nb;
                const bool apart = lane + 1 >= n || d <= len - 32 || d >= len;
                flat = __all_sync(FULL, lane >= n || (run && apart));
            }
            if (flat) {
                int32_t incl = len;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int32_t y = __shfl_up_sync(FULL, incl, d);
                    if (lane >= d) incl += y;
                }
                const int32_t total = __shfl_sync(FULL, incl, 31);
                for (int q = 0; q < n; ++q)
                    runs |= run_bits(lane, __shfl_sync(FULL, first, q), __shfl_sync(FULL, last, q));
                // Product t of entry q: position posAt + t in B, column relAt + t.
                const int32_t posAt = bs - (incl - len), relAt = first - (incl - len);
                int q = 0;
                int32_t end = __shfl_sync(FULL, incl, 0);
                int32_t p0 = __shfl_sync(FULL, posAt, 0), p1 = __shfl_sync(FULL, posAt, 1);
                int32_t c0 = __shfl_sync(FULL, relAt, 0), c1 = __shfl_sync(FULL, relAt, 1);
                double a0 = __shfl_sync(FULL, avl, 0), a1 = __shfl_sync(FULL, avl, 1);
                for (int32_t t0 = 0; t0 < total; t0 += 32 * U) {  // U steps' loads in flight together
                    int32_t rel[U];
                    double av[U], bv[U];
                    const int q0 = q;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int32_t s = t0 + 32 * u, t = s + lane;
                        if (s >= end && s < total) {  // the step starts in the next entry (none is shorter than a step)
                            ++q;
                            end = __shfl_sync(FULL, incl, q);
                            p0 = p1;
                            c0 = c1;
                            a0 = a1;
                            p1 = __shfl_sync(FULL, posAt, q + 1);
                            c1 = __shfl_sync(FULL, relAt, q + 1);
                            a1 = __shfl_sync(FULL, avl, q + 1);
                        }
                        const bool next = t >= end;
                        rel[u] = t < total ? (next ? c1 : c0) + t : -1;
                        av[u] = next ? a1 : a0;
                        bv[u] = t < total ? __ldg(&bval[(next ? p1 : p0) + t]) : 0.0;
                    }
                    if (U > 3 && q == q0 && t0 + 32 * U <= end) {
                        // All in one entry: no column twice.
                        double x[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) x[u] = vals[rel[u]];
#pragma unroll
                        for (int u = 0; u < U; ++u) vals[rel[u]] = __fma_rn(av[u], bv[u], x[u]);
                        __syncwarp();
                        continue;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (rel[u] >= 0) vals[rel[u]] = __fma_rn(av[u], bv[u], vals[rel[u]]);
                        __syncwarp();
                    }
                }
                continue;
            }
            // One A entry at a time; each lane loads up to four of the B row's
            // products before using any, so their loads are in flight together.
            for (int q = 0; q < n; ++q) {
                const int32_t bq = __shfl_sync(FULL, bs, q);
                const int32_t lq = __shfl_sync(FULL, len, q);
                const double aq = __shfl_sync(FULL, avl, q);
                for (int32_t i0 = 0; i0 < lq; i0 += 128) {
                    int32_t c[4];
                    double v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int32_t i = i0 + 32 * u + lane;
                        c[u] = i < lq ? bidx[bq + i] : INT_MIN;
                        v[u] = i < lq ? bval[bq + i] : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (c[u] != INT_MIN) add((uint32_t)(c[u] - cbase), aq, v[u]);
                }
                __syncwarp();
            }
        }
    } else {
        warp_products(a.A, a.B, e0, e1, lane,
                      [&](int32_t j, double av) { add((uint32_t)(bidx[j] - cbase), av, bval[j]); });
    }
    __syncwarp();
    const int32_t obc = cbase - col_shift(a, row);  // column written for flag 0
    int64_t p = 0;
    for (int w = 0; w < sw; ++w) {
        const uint32_t word = __shfl_sync(FULL, runs, w);
        const bool set = fb[32 * w + lane] != 0 || ((word >> lane) & 1u);
        const unsigned bal = __ballot_sync(FULL, set);
        const int64_t at = p + __popc(bal & ((1u << lane) - 1u));
        if (set && at < expect) {
            a.Ci[obase + at] = obc + 32 * w + lane;
            a.Cv[obase + at] = vals[32 * w + lane];
        }
        p += __popc(bal);
    }
    if (lane == 0 && p != expect) raise(a.err, DEV_COUNT_MISMATCH);
}

template <int ROWS, int U>
__global__ void __launch_bounds__(32 * ROWS) k_num_densew(NumArgs a, int32_t lo, int32_t count) {
    num_densew_rows<ROWS, U>(a, lo, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_num_densew_dd(NumArgs a, int bin) {
    const int32_t lo = a.binStart[bin], count = a.binStart[bin + 1] - lo;
    for (int64_t vb = blockIdx.x; vb * ROWS < count; vb += gridDim.x) {
        num_densew_rows<ROWS, 3>(a, lo, count, vb);
        __syncthreads();
    }
}

// Narrow rows (window of at most kWarpSpanWords words, at most kNumWarpMax
// entries): one warp per row with the window's bitmap, word ranks and the
// row's values in shared memory; the rank kernel's method at warp scale.
template <int ROWS>
__device__ __forceinline__ void num_rankw_rows(const NumArgs &a, int32_t lo, int32_t count, int64_t vb) {
    static_assert(kWarpSpanWords == 64, "two bitmap words per lane");
    __shared__ uint32_t bms[ROWS][kWarpSpanWords];
    __shared__ int32_t wps[ROWS][kWarpSpanWords];
    __shared__ double vs[ROWS][kNumWarpMax];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)vb * ROWS + g;
    if (item >= count) return;
    uint32_t *bm = bms[g];
    int32_t *wp = wps[g];
    double *vals = vs[g];
    const int32_t row = a.list[lo + item];
    const int32_t cbase = (a.rowLo[row] >> 5) << 5;
    const int32_t obc = cbase - col_shift(a, row);  // column written for bit 0
    const int64_t expect = a.Cp[row + 1] - a.Cp[row];
    const int64_t obase = a.Cp[row] - a.outBase;
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    for (int i = lane; i < kWarpSpanWords; i += 32) bm[i] = 0u;
    for (int i = lane; i < kNumWarpMax; i += 32) vals[i] = 0.0;
    __syncwarp();
    for (int32_t e = e0; e < e1; e += 32) {
        const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
        for (int32_t t0 = 0; t0 < c.total; t0 += 32) {
            const int32_t t = t0 + lane;
            const int32_t j = chunk_pos(c, t, nullptr);
            const uint32_t rel = t < c.total ? (uint32_t)(a.B.idx[j] - cbase) : 0u;
            const bool v = t < c.total && in_window(rel, kWarpSpanWords * 32, a.err);
            or_bit(bm, v, rel);
        }
    }
    __syncwarp();
    const int32_t p0 = __popc(bm[lane]), p1 = __popc(bm[lane + 32]);
    int32_t i0 = p0, i1 = p1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int32_t y0 = __shfl_up_sync(FULL, i0, d), y1 = __shfl_up_sync(FULL, i1, d);
        if (lane >= d) {
            i0 += y0;
            i1 += y1;
        }
    }
    const int32_t half = __shfl_sync(FULL, i0, 31);
    const int32_t total = half + __shfl_sync(FULL, i1, 31);
    wp[lane] = i0 - p0;
    wp[lane + 32] = half + i1 - p1;
    if (lane == 0 && total != expect) raise(a.err, DEV_COUNT_MISMATCH);
    __syncwarp();
    for (int w = lane; w < kWarpSpanWords; w += 32) {
        uint32_t word = bm[w];
        int64_t p = wp[w];
        while (word) {
            const int b = __ffs(word) - 1;
            word &= word - 1u;
            if (p < expect) a.Ci[obase + p] = obc + (w << 5) + b;
            ++p;
        }
    }
    for (int32_t e = e0; e < e1; e += 32) {
        const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
        for (int32_t t0 = 0; t0 < c.total; t0 += 32) {
            const int32_t t = t0 + lane;
            double av;
            const int32_t j = chunk_pos(c, t, &av);
            const int32_t col = t < c.total ? a.B.idx[j] - cbase : 0;
            if (t < c.total && (uint32_t)col < (uint32_t)(kWarpSpanWords * 32)) {
                const int w = col >> 5;
                const int r = wp[w] + __popc(bm[w] & ((1u << (col & 31)) - 1u));
                if (r < kNumWarpMax) atomic_fma(&vals[r], av, a.B.val[j]);
            }
        }
    }
    __syncwarp();
    const int64_t nout = min(expect, (int64_t)kNumWarpMax);
    for (int64_t i = lane; i < nout; i += 32) a.Cv[obase + i] = vals[i];
}

template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_num_rankw(NumArgs a, int32_t lo, int32_t count) {
    num_rankw_rows<ROWS>(a, lo, count, blockIdx.x);
}

// The same rows launched device-driven: the bin's rows from the bin table
// on the device, covered by a grid-stride loop.
template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_num_rankw_dd(NumArgs a, int bin) {
    const int32_t lo = a.binStart[bin], count = a.binStart[bin + 1] - lo;
    for (int64_t vb = blockIdx.x; vb * ROWS < count; vb += gridDim.x) {
        num_rankw_rows<ROWS>(a, lo, count, vb);
        __syncthreads();
    }
}

// A segmented OR over runs of lanes that share a word that also marks, in a summary bitmap (one bit per word),
// every word it finds zero.  All lanes call.
__device__ __forceinline__ void or_bits_mark(uint32_t *bm, uint32_t *sum, bool v, uint32_t rel) {
    const int lane = threadIdx.x & 31;
    const int32_t w = v ? (int32_t)(rel >> 5) : -1 - lane;
    uint32_t acc = v ? 1u << (rel & 31) : 0u;
    bool head = v;
    if (__any_sync(FULL, __shfl_up_sync(FULL, w, 1) == w && lane > 0)) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t ow = __shfl_down_sync(FULL, w, d);
            const uint32_t ob = __shfl_down_sync(FULL, acc, d);
            if (lane + d < 32 && ow == w) acc |= ob;
        }
        const int32_t pw = __shfl_up_sync(FULL, w, 1);
        head = v && (lane == 0 || pw != w);
    }
    if (head && atomicOr(&bm[w], acc) == 0u) atomicOr(&sum[w >> 5], 1u << (w & 31));
}

// Rows of at most kNumWarpMax entries whose window spans at most
// kMidSpanWords words: persistent warps, one row at a time, the rank method
// over the row's own window.  A summary bitmap (one bit per window word)
// lists the words the row touched, so word ranks, output and the clean-up
// for the next row visit only those words: a row costs its products and
// entries, not its span.  No hash table, no sort.
template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_num_rankm(NumArgs a, int32_t lo, int32_t count) {
    if (lo < 0) {  // device-driven: the bin's rows from the bin table
        lo = a.binStart[NB_RANKM];
        count = a.binStart[NB_RANKM + 1] - lo;
    }
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int kSumWords = kMidSpanWords / 32;
    constexpr size_t kWarpBytes =
        8 * (size_t)kNumWarpMax + 4 * (size_t)kMidSpanWords + 4 * (size_t)kSumWords + 2 * (size_t)kMidSpanWords;
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double *vals = reinterpret_cast<double *>(smem + g * kWarpBytes);
    uint32_t *bm = reinterpret_cast<uint32_t *>(vals + kNumWarpMax);
    uint32_t *sum = bm + kMidSpanWords;
    uint16_t *wp = reinterpret_cast<uint16_t *>(sum + kSumWords);
    for (int i = lane; i < kMidSpanWords; i += 32) bm[i] = 0u;
    for (int i = lane; i < kSumWords; i += 32) sum[i] = 0u;
    for (int i = lane; i < kNumWarpMax; i += 32) vals[i] = 0.0;
    __syncwarp();
    const int64_t warps = (int64_t)gridDim.x * ROWS;
    for (int64_t item = (int64_t)blockIdx.x * ROWS + g; item < count; item += warps) {
        const int32_t row = a.list[lo + item];
        const int32_t rlo = a.rowLo[row];
        const int32_t cbase = (rlo >> 5) << 5;
        const int nw = min(span_words(rlo, a.rowHi[row]), kMidSpanWords);
        const uint32_t nbits = (uint32_t)nw * 32u;
        const int32_t obc = cbase - col_shift(a, row);  // column written for bit 0
        const int64_t expect = a.Cp[row + 1] - a.Cp[row];
        const int64_t obase = a.Cp[row] - a.outBase;
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        for (int32_t e = e0; e < e1; e += 32) {
            const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
            for (int32_t t0 = 0; t0 < c.total; t0 += 32) {
                const int32_t t = t0 + lane;
                const int32_t j = chunk_pos(c, t, nullptr);
                const uint32_t rel = t < c.total ? (uint32_t)(a.B.idx[j] - cbase) : 0u;
                const bool v = t < c.total && in_window(rel, nbits, a.err);
                or_bits_mark(bm, sum, v, rel);
            }
        }
        __syncwarp();
        // Lane l owns window words [64 l, 64 l + 64): summary words 2l, 2l + 1.
        const uint32_t s0 = sum[2 * lane], s1 = sum[2 * lane + 1];
        int cnt = 0;
        for (uint32_t m = s0; m; m &= m - 1u) cnt += __popc(bm[64 * lane + __ffs(m) - 1]);
        for (uint32_t m = s1; m; m &= m - 1u) cnt += __popc(bm[64 * lane + 32 + __ffs(m) - 1]);
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += y;
        }
        const int total = __shfl_sync(FULL, incl, 31);
        if (lane == 0 && total != expect) raise(a.err, DEV_COUNT_MISMATCH);
        int64_t p = incl - cnt;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            for (uint32_t m = h ? s1 : s0; m; m &= m - 1u) {
                const int w = 64 * lane + 32 * h + __ffs(m) - 1;
                wp[w] = (uint16_t)p;
                uint32_t word = bm[w];
                while (word) {
                    const int b = __ffs(word) - 1;
                    word &= word - 1u;
                    if (p < expect) a.Ci[obase + p] = obc + (w << 5) + b;
                    ++p;
                }
            }
        }
        __syncwarp();
        for (int32_t e = e0; e < e1; e += 32) {
            const Chunk c = load_chunk(a.A, a.B, e, e1, lane);
            for (int32_t t0 = 0; t0 < c.total; t0 += 32) {
                const int32_t t = t0 + lane;
                double av;
                const int32_t j = chunk_pos(c, t, &av);
                const int32_t col = t < c.total ? a.B.idx[j] - cbase : 0;
                if (t < c.total && (uint32_t)col < nbits) {
                    const int w = col >> 5;
                    const int r = wp[w] + __popc(bm[w] & ((1u << (col & 31)) - 1u));
                    if (r < kNumWarpMax) atomic_fma(&vals[r], av, a.B.val[j]);
                }
            }
        }
        __syncwarp();
        const int nout = (int)min(expect, (int64_t)kNumWarpMax);
        for (int i = lane; i < nout; i += 32) {
            a.Cv[obase + i] = vals[i];
            vals[i] = 0.0;
        }
        // Leave the bitmap and summary clean for the next row.
        for (uint32_t m = s0; m; m &= m - 1u) bm[64 * lane + __ffs(m) - 1] = 0u;
        for (uint32_t m = s1; m; m &= m - 1u) bm[64 * lane + 32 + __ffs(m) - 1] = 0u;
        sum[2 * lane] = 0u;
        sum[2 * lane + 1] = 0u;
        __syncwarp();
    }
}

// Work items of the dense bin for list[lo, lo + n): one per row, except that
// a row of more than kPieceNnz entries whose slab counts the symbolic pass
// recorded (B's rows ascending) is cut at slab boundaries into pieces of
// about kPieceNnz entries and at most kPieceSlabs slabs.  Every item is
// independent: it knows its columns and where its entries start in C's row.
__global__ void __launch_bounds__(256) k_dense_items(NumArgs a, int32_t lo, int32_t n) {
    const int32_t i = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const int32_t row = a.list[lo + i];
    const int64_t nnz = a.Cp[row + 1] - a.Cp[row];
    const int32_t sl = a.heavySlot[row];
    auto put = [&](int s0, int s1, int32_t cnt, int64_t off) {
        const uint32_t k = atomicAdd(&a.ctr[CTR_ITEMS], 1u);
        if (k >= (uint32_t)a.itemCap) {
            raise(a.err, DEV_TABLE_FULL);
            return;
        }
        a.items[k] = DenseItem{row, (int16_t)s0, (int16_t)s1, cnt, off};
    };
    if (sl < 0 || !b_sorted(a) || nnz <= kPieceNnz) {
        put(-1, -1, (int32_t)min(nnz, (int64_t)INT32_MAX), 0);
        return;
    }
    const int64_t base = (int64_t)(a.rowLo[row] >> 5) << 5;
    const int ns = (int)((((int64_t)a.rowHi[row] + 1 - base) + (1 << kSlabShift) - 1) >> kSlabShift);
    const int32_t *sc = a.slabCnt + (size_t)sl * kMaxSlabs;
    int s0 = 0;
    int32_t acc = 0;
    int64_t off = 0;
    for (int s = 0; s < ns; ++s) {
        const int32_t c = sc[s];
        if (s > s0 && (acc + c > kPieceNnz || s - s0 == kPieceSlabs)) {
            put(s0, s, acc, off);
            off += acc;
            acc = 0;
            s0 = s;
        }
        acc += c;
    }
    put(s0, ns, acc, off);
}

// Dense rows (windows wider than the CTA rank kernel's): persistent CTAs,
// two per SM, take rows from a counter and apply the rank method over
// windows of WIN words of the row's span (2^19 columns in shared memory).
// Per window: a pass over the row's products sets the bits inside the
// window; its words are counted and ranked 128 a warp and step (a 16-bit
// offset each from a 32-bit base per 256 words), and 32-word groups get the
// rank of their first column and the mask of their non-empty words, from
// which C's columns are written (each thread a contiguous run of them).  A
// second pass adds every product inside the window into C's row in place at
// its rank (FP64 L2 reductions).  Bound by instruction issue and the
// reductions' 24 sectors a step (10,240 rows of R-MAT 2^21: 7 GB of DRAM
// traffic and 59% of L1's throughput in 3.6 ms).  With a 32-word group a
// thread, whose non-empty words it then visited one by one, the warp waited for the
// fullest group: 3.92 -> 3.77 ms.  Half as many CTAs of 1024 threads and twice the
// window: 4.07.
template <int THREADS, int WIN>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_num_rankwin(NumArgs a, int32_t lo, int32_t count) {
    static_assert(WIN == 32 * THREADS, "whole groups of 256 words per warp");
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    constexpr int NW = THREADS / 32;
    __shared__ int32_t sh[NW];
    __shared__ int32_t next;
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    double *av = reinterpret_cast<double *>(smem + L::av);
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem + rank_bits_at(THREADS));
    uint16_t *wpre = reinterpret_cast<uint16_t *>(bits + WIN);
    int32_t *gbase = reinterpret_cast<int32_t *>(wpre + WIN);
    int32_t *tbase = gbase + WIN / 256;                          // per thread: rank of its first column
    uint32_t *tmask = reinterpret_cast<uint32_t *>(tbase + THREADS);  // per thread: its non-empty words
    int32_t *cur = reinterpret_cast<int32_t *>(tmask + THREADS);      // per staged entry: its B cursor
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i < WIN; i += THREADS) bits[i] = 0u;
    // With work items (heavy rows cut into pieces), the items the builder
    // wrote before this launch; otherwise the bin's rows.
    if (lo < 0) {  // device-driven: the bin's rows from the bin table
        lo = a.binStart[NB_DENSE];
        count = a.binStart[NB_DENSE + 1] - lo;
    }
    const int32_t nitems = a.items ? (int32_t)min(*(volatile uint32_t *)&a.ctr[CTR_ITEMS], (uint32_t)a.itemCap)
                                   : count;
    for (;;) {
        if (tid == 0) next = (int32_t)atomicAdd(&a.ctr[CTR_NUM_RANKWIN], 1u);
        __syncthreads();
        if (next >= nitems) break;
        const int32_t item = next;
        DenseItem it{0, -1, -1, 0, 0};
        if (a.items) it = a.items[item];
        const int32_t row = a.items ? it.row : a.list[lo + item];
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        const int64_t expect = a.Cp[row + 1] - a.Cp[row];
        const int64_t obase = a.Cp[row] - a.outBase;
        const int32_t shift = col_shift(a, row);
        int64_t end = (int64_t)a.rowHi[row] + 1;
        int64_t start = (int64_t)(a.rowLo[row] >> 5) << 5;
        int64_t run = 0, expectEnd = expect;
        if (it.s0 >= 0) {
            // A piece: the row's columns [start + s0 slabs, start + s1 slabs).
            const int64_t b = start;
            start = b + ((int64_t)it.s0 << kSlabShift);
            end = min(end, b + ((int64_t)it.s1 << kSlabShift));
            run = it.off;
            expectEnd = it.off + it.cnt;
        }
        // Rows over several windows and pieces enumerate, per window, only
        // the part of each B row inside it (B's rows ascending).
        const bool clip = b_sorted(a) && (it.s0 >= 0 || end - start > (int64_t)WIN * 32);
        for (int64_t c_lo = start; c_lo < end; c_lo += (int64_t)WIN * 32) {
            const int nwords = (int)min((int64_t)WIN, (end - c_lo + 31) >> 5);
            const uint32_t nbits = (uint32_t)nwords * 32u;
            const int64_t c_hi = c_lo + nbits;
            // Pass 1: the window's bits.  A row (or piece) of at most THREADS
            // entries is staged once, with its A values, and pass 2 reuses
            // the staging (no second round of loads and clipping searches).
            const bool once = e1 - e0 <= THREADS;
            int nb1 = 0;
            int32_t total1 = 0;
            for (int32_t eb = e0; eb < e1; eb += THREADS) {
                int nb;
                const int32_t total =
                    once ? stage_entries<THREADS, true>(a.A, a.B, eb, e1 - eb, pre, bst, av, &nb, sh, clip, c_lo, c_hi,
                                                        cur, c_lo != start)
                         : stage_entries<THREADS, false>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, nullptr, &nb,
                                                         sh, clip, c_lo, c_hi);
                nb1 = nb;
                total1 = total;
                int32_t tb, te;
                warp_share<THREADS>(total, &tb, &te);
                warp_range_ld<4>(
                    pre, bst, nb, tb, te, [&](int32_t pos) { return __ldg(&a.B.idx[pos]); },
                    [&](bool v, int32_t col, int) {
                        const uint32_t rel = (uint32_t)col - (uint32_t)c_lo;
                        or_bit(bits, v && rel < nbits, rel);
                    });
                __syncthreads();
            }
            // The words' ranks, 128 words a warp and step, four a lane, and
            // per 32 words the rank of the first column and the non-empty
            // words.
            const int w0 = (tid >> 5) * (WIN / NW) + 4 * lane;
            int32_t cnt = 0;
#pragma unroll
            for (int j = 0; j < WIN / NW / 128; ++j) {
                const uint4 v = *reinterpret_cast<const uint4 *>(bits + w0 + 128 * j);
                cnt += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            }
            int32_t tot;
            int32_t p0 = __shfl_sync(FULL, block_excl_scan<THREADS>(cnt, &tot, sh), 0), gb = p0;
#pragma unroll 2
            for (int j = 0; j < WIN / NW / 128; ++j) {
                const int i = w0 + 128 * j;
                const uint4 v = *reinterpret_cast<const uint4 *>(bits + i);
                const int32_t c1 = __popc(v.x), c2 = c1 + __popc(v.y), c3 = c2 + __popc(v.z), c4 = c3 + __popc(v.w);
                int32_t x = c4;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int32_t y = __shfl_up_sync(FULL, x, d);
                    if (lane >= d) x += y;
                }
                const int32_t p = p0 + x - c4;
                if ((j & 1) == 0) {  // a group of 256 words starts
                    gb = p0;
                    if (lane == 0) gbase[i >> 8] = p0;
                }
                p0 += __shfl_sync(FULL, x, 31);
                const int32_t q = p - gb;
                *reinterpret_cast<ushort4 *>(wpre + i) = make_ushort4(
                    (uint16_t)q, (uint16_t)(q + c1), (uint16_t)(q + c2), (uint16_t)(q + c3));
                uint32_t mask = ((v.x ? 1u : 0u) | (v.y ? 2u : 0u) | (v.z ? 4u : 0u) | (v.w ? 8u : 0u))
                                << (4 * (lane & 7));
#pragma unroll
                for (int d = 1; d < 8; d <<= 1) mask |= __shfl_xor_sync(FULL, mask, d);
                if ((lane & 7) == 0) {
                    tbase[i >> 5] = p;
                    tmask[i >> 5] = mask;
                }
            }
            __syncthreads();
            // C's columns, balanced over the threads by output position.
            write_columns_balanced<THREADS>(bits, tbase, tmask, 32, tot, a.Ci + obase + run, expect - run,
                                            c_lo - shift);
            for (int64_t i = tid; i < tot && run + i < expect; i += THREADS) a.Cv[obase + run + i] = 0.0;
            __syncthreads();
            // Pass 2: the window's products into C's row in place (ranks
            // within a window and its columns fit 32 bits).
            double *cv = a.Cv + obase + run;
            const uint32_t lim = (uint32_t)max((int64_t)0, min(expect - run, (int64_t)INT_MAX));
            for (int32_t eb = e0; eb < e1; eb += THREADS) {
                int nb = nb1;
                const int32_t total =
                    once ? total1
                         : stage_entries<THREADS, true>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, av, &nb, sh,
                                                        clip, c_lo, c_hi);
                int32_t tb, te;
                warp_share<THREADS>(total, &tb, &te);
                warp_range_ld<4>(
                    pre, bst, nb, tb, te,
                    [&](int32_t pos) { return ColVal{__ldg(&a.B.idx[pos]), __ldg(&a.B.val[pos])}; },
                    [&](bool v, const ColVal &x, int e) {
                        const uint32_t c = (uint32_t)x.c - (uint32_t)c_lo;
                        if (v && c < nbits) {
                            const uint32_t w = c >> 5;
                            const uint32_t r = (uint32_t)gbase[w >> 8] + wpre[w] +
                                               __popc(bits[w] & ((1u << (c & 31)) - 1u));
                            if (r < lim) atomicAdd(&cv[r], __dmul_rn(av[e], x.v));
                        }
                    });
                __syncthreads();
            }
            // Leave the bitmap zero.
            for (int i = tid; 4 * i < nwords; i += THREADS)
                reinterpret_cast<uint4 *>(bits)[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            run += tot;
        }
        if (tid == 0 && run != expectEnd) raise(a.err, DEV_COUNT_MISMATCH);
        __syncthreads();  // every thread has read `next` before it changes
    }
}

// Dense rows in one product pass: persistent CTAs (one per scratch row) take
// rows from a counter; per window of WIN words of the row's span (2^19 columns)
// one pass over the row's products sets each product's column bit in a
// shared bitmap and adds the product into the CTA's FP64 scratch row in
// global memory, indexed by column (an L2 reduction whose result is not
// read back).  Then each warp compacts its 1024 words of the window, word
// by word in column order: the 32 lanes are the word's 32 columns, so C's
// columns and values go out as contiguous runs (coalesced), the values read
// from the scratch row at the same 32 consecutive columns, which the warp
// zeroes behind it, leaving the scratch row and the bitmap zero for the next
// window.  Compared with the rank method this enumerates every product once
// instead of twice and writes C once, coalesced, instead of zeroing it and
// reducing into it in place.
template <int THREADS, int WIN>
__global__ void __launch_bounds__(THREADS) k_num_dscr(NumArgs a, int32_t lo, int32_t count) {
    static_assert(WIN == 32 * THREADS, "one 32-word group per thread");
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    constexpr int NW = THREADS / 32;
    __shared__ int32_t sh[NW];
    __shared__ int32_t next;
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    double *av = reinterpret_cast<double *>(smem + L::av);
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem + L::bytes);
    double *scr = a.scr + (size_t)blockIdx.x * (size_t)a.scrStride;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t lt = (1u << lane) - 1u;
    for (int i = tid; i < WIN; i += THREADS) bits[i] = 0u;
    for (;;) {
        if (tid == 0) next = (int32_t)atomicAdd(&a.ctr[CTR_NUM_DSCR], 1u);
        __syncthreads();
        if (next >= count) break;
        const int32_t item = next;
        const int32_t row = a.list[lo + item];
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        const int64_t expect = a.Cp[row + 1] - a.Cp[row];
        const int64_t obase = a.Cp[row] - a.outBase;
        const int32_t shift = col_shift(a, row);
        const int64_t end = (int64_t)a.rowHi[row] + 1;
        const int64_t start = (int64_t)(a.rowLo[row] >> 5) << 5;
        const bool clip = b_sorted(a) && end - start > (int64_t)WIN * 32;
        int64_t run = 0;
        for (int64_t c_lo = start; c_lo < end; c_lo += (int64_t)WIN * 32) {
            const int nwords = (int)min((int64_t)WIN, (end - c_lo + 31) >> 5);
            const uint32_t nbits = min((uint32_t)nwords * 32u, (uint32_t)a.scrStride);
            const int64_t c_hi = c_lo + nbits;
            // The pass: bits in shared memory, products into the scratch row.
            for (int32_t eb = e0; eb < e1; eb += THREADS) {
                int nb;
                const int32_t total = stage_entries<THREADS, true>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, av,
                                                                   &nb, sh, clip, c_lo, c_hi);
                int32_t tb, te;
                warp_share<THREADS>(total, &tb, &te);
                warp_range_ld<4>(
                    pre, bst, nb, tb, te,
                    [&](int32_t pos) { return ColVal{__ldg(&a.B.idx[pos]), __ldg(&a.B.val[pos])}; },
                    [&](bool v, const ColVal &x, int e) {
                        const uint32_t rel = v ? (uint32_t)((int64_t)x.c - c_lo) : 0u;
                        const bool in = v && rel < nbits;
                        or_bit(bits, in, rel);
                        if (in) atomicAdd(&scr[rel], __dmul_rn(av[e], x.v));
                    });
                __syncthreads();
            }
            // Word counts: thread t holds words [32 t, 32 t + 32).
            uint32_t mask = 0;
            int32_t cnt = 0;
#pragma unroll 8
            for (int k = 0; k < 32; ++k) {
                const int q = (k + lane) & 31;
                const uint32_t x = bits[32 * tid + q];
                if (x) mask |= 1u << q;
                cnt += __popc(x);
            }
            int32_t tot;
            const int32_t base = block_excl_scan<THREADS>(cnt, &tot, sh);
            // Compaction: the warp walks its lanes' non-empty words in column
            // order; lane b takes column 32 w + b of word w.
            for (int src = 0; src < 32; ++src) {
                uint32_t m = __shfl_sync(FULL, mask, src);
                int64_t p = run + __shfl_sync(FULL, base, src);
                while (m) {
                    const int w = 32 * (32 * (tid >> 5) + src) + __ffs(m) - 1;
                    m &= m - 1u;
                    const uint32_t word = bits[w];
                    const int64_t q = p + __popc(word & lt);
                    if ((word >> lane) & 1u) {
                        double *s = &scr[32 * w + lane];
                        if (q < expect) {
                            __stcs(&a.Ci[obase + q], (int32_t)(c_lo + 32 * w + lane - shift));
                            __stcs(&a.Cv[obase + q], __ldcg(s));
                        }
                        __stcg(s, 0.0);
                    }
                    p += __popc(word);
                }
            }
            __syncthreads();  // every warp has read its words before they clear
            for (uint32_t m = mask; m; m &= m - 1u) bits[32 * tid + __ffs(m) - 1] = 0u;
            __syncthreads();
            run += tot;
        }
        if (tid == 0 && run != expect) raise(a.err, DEV_COUNT_MISMATCH);
        __syncthreads();  // every thread has read `next` before it changes
    }
}

// Dense rows with a global slot: persistent CTAs, one slot each, take rows
// from a counter; the rank method over the whole row, its bitmap and word
// ranks in the slot (two bits per column of C, so the slots of all CTAs stay
// in L2 for millions of columns) and the summary bitmap (one bit per bitmap
// word) in shared memory.  Pass 1 sets every product's column bit by an L2
// reduction (no round trip) and its word's summary bit in shared memory.  The word ranks are computed over the summary
// bits of the row's window in order (the row's entries plus its span / 1024),
// which also writes C's columns.  Pass 2 adds every product into C's row in
// place at its rank (FP64 L2 reductions).  The clean-up clears the words it
// set.  Reads after reductions go to L2 (__ldcg), past the SM's L1.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_num_gdense(NumArgs a, int32_t lo, int32_t count) {
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    constexpr int NW = THREADS / 32;
    __shared__ int32_t sh[NW];
    __shared__ int32_t next;
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    double *av = reinterpret_cast<double *>(smem + L::av);
    uint32_t *sum = reinterpret_cast<uint32_t *>(smem + L::bytes);
    const int tid = threadIdx.x;
    uint32_t *bits = a.gBits + (size_t)blockIdx.x * (a.gStride >> 5);
    uint32_t *wpre = a.gWpre + (size_t)blockIdx.x * (a.gStride >> 5);
    const uint32_t ncols = (uint32_t)min(a.gStride, a.B.n);
    int *err = a.err;
    for (int i = tid; i < (int)(a.gStride >> 10); i += THREADS) sum[i] = 0u;
    for (;;) {
        if (tid == 0) next = (int32_t)atomicAdd(&a.ctr[CTR_NUM_GDENSE], 1u);
        __syncthreads();
        const int32_t item = next;
        if (item >= count) break;
        const int32_t row = a.list[lo + item];
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        const int64_t expect = a.Cp[row + 1] - a.Cp[row];
        const int64_t obase = a.Cp[row] - a.outBase;
        const int32_t shift = col_shift(a, row);
        // Pass 1: bits.
        for (int32_t eb = e0; eb < e1; eb += THREADS) {
            int nb;
            const int32_t total =
                stage_entries<THREADS, false>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, nullptr, &nb, sh);
            int32_t tb, te;
            warp_share<THREADS>(total, &tb, &te);
            warp_range_ld<4>(
                pre, bst, nb, tb, te, [&](int32_t pos) { return __ldg(&a.B.idx[pos]); },
                [&](bool v, int32_t col, int) {
                    if (v) {
                        const uint32_t c = (uint32_t)col;
                        if (in_window(c, ncols, err)) {
                            atomicOr(&bits[c >> 5], 1u << (c & 31));
                            atomicOr(&sum[c >> 10], 1u << ((c >> 5) & 31));  // shared
                        }
                    }
                });
            __syncthreads();
        }
        __threadfence();
        __syncthreads();
        // Word ranks and C's columns; thread t owns a contiguous run of the
        // window's summary words.
        const int32_t s0 = a.rowLo[row] >> 10, s1 = a.rowHi[row] >> 10;
        const int nsum = s1 - s0 + 1;
        const int per = (nsum + THREADS - 1) / THREADS;
        const int q0 = s0 + min(nsum, tid * per), q1 = s0 + min(nsum, tid * per + per);
        int cnt = 0;
        for (int q = q0; q < q1; ++q)
            for (uint32_t m = sum[q]; m; m &= m - 1u) cnt += __popc(__ldcg(&bits[q * 32 + __ffs(m) - 1]));
        int32_t tot;
        int64_t pos = block_excl_scan<THREADS>(cnt, &tot, sh);
        if (tid == 0 && tot != expect) raise(a.err, DEV_COUNT_MISMATCH);
        for (int q = q0; q < q1; ++q) {
            for (uint32_t m = sum[q]; m; m &= m - 1u) {
                const int w = q * 32 + __ffs(m) - 1;
                __stcg(&wpre[w], (uint32_t)pos);
                uint32_t word = __ldcg(&bits[w]);
                while (word) {
                    const int b = __ffs(word) - 1;
                    word &= word - 1u;
                    if (pos < expect) a.Ci[obase + pos] = w * 32 + b - shift;
                    ++pos;
                }
            }
        }
        for (int64_t i = tid; i < expect; i += THREADS) __stcg(&a.Cv[obase + i], 0.0);
        __threadfence();
        __syncthreads();
        // Pass 2: values in place at their ranks.
        for (int32_t eb = e0; eb < e1; eb += THREADS) {
            int nb;
            const int32_t total =
                stage_entries<THREADS, true>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, av, &nb, sh);
            int32_t tb, te;
            warp_share<THREADS>(total, &tb, &te);
            warp_range_ld<4>(
                pre, bst, nb, tb, te,
                [&](int32_t p) { return ColVal{__ldg(&a.B.idx[p]), __ldg(&a.B.val[p])}; },
                [&](bool v, const ColVal &x, int e) {
                    if (v) {
                        const uint32_t c = (uint32_t)x.c;
                        if (c < ncols) {
                            const int w = (int)(c >> 5);
                            const int64_t r =
                                (int64_t)__ldcg(&wpre[w]) + __popc(__ldcg(&bits[w]) & ((1u << (c & 31)) - 1u));
                            if (r < expect) atomicAdd(&a.Cv[obase + r], __dmul_rn(av[e], x.v));
                        }
                    }
                });
            __syncthreads();
        }
        // Clean-up: the words this row set, then its summary words.
        for (int q = q0; q < q1; ++q) {
            for (uint32_t m = sum[q]; m; m &= m - 1u) __stcg(&bits[q * 32 + __ffs(m) - 1], 0u);
            sum[q] = 0u;
        }
        __threadfence();
        __syncthreads();
    }
}

// Dense rows: one CTA per row sweeps windows of W columns.  Every A entry
// keeps a cursor into its B row and the next column at or past it, in shared
// memory for rows of at most ECAP entries and in a.state otherwise.  Per
// window, each warp reads the next columns of 32 entries at a time (one
// coalesced load), and only entries with products inside the window are
// worked on: the warp scans that entry's B row from its cursor 32 products
// per step (with B rows ascending the products inside the window are a
// prefix, found by ballot).  No block barrier runs per entry, only per
// window.  Without sorted B rows every window rescans whole B rows and
// filters.  The window is zeroed once and every written column is zeroed as
// it is written out, so a window costs its products and C entries, not its
// width.
template <int THREADS, int W, int ECAP, bool SORTED>
__global__ void __launch_bounds__(THREADS) k_num_dense(NumArgs a, int32_t lo) {
    extern __shared__ __align__(16) unsigned char smem[];
    static_assert(W / 32 <= THREADS, "one bitmap word per thread");
    constexpr int NW = THREADS / 32;
    double *dense = reinterpret_cast<double *>(smem);
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem + 8 * (size_t)W);
    int32_t *scur = reinterpret_cast<int32_t *>(smem + 8 * (size_t)W + W / 8);
    int32_t *snext = scur + ECAP;
    __shared__ int32_t sh[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int32_t row = a.list[lo + blockIdx.x];
    const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
    const int32_t nA = e1 - e0;
    const bool resident = nA <= ECAP;
    int32_t *cur_of = resident ? scur : a.state + e0;              // cursor per A entry
    int32_t *next_of = resident ? snext : a.state + a.A.nnz + e0;  // next column per A entry
    const int64_t expect = a.Cp[row + 1] - a.Cp[row];
    const int64_t obase = a.Cp[row] - a.outBase;
    const int32_t shift = col_shift(a, row);
    for (int i = tid; i < W; i += THREADS) dense[i] = 0.0;
    for (int i = tid; i < W / 32; i += THREADS) bits[i] = 0u;

    // Initial state of every entry.
    int32_t mymin = INT_MAX;
    for (int32_t i = tid; i < nA; i += THREADS) {
        const int32_t k = a.A.idx[e0 + i];
        const int32_t s = a.B.ptr[k], t = a.B.ptr[k + 1];
        int32_t nx = INT_MAX;
        if constexpr (SORTED) {
            if (s < t) nx = a.B.idx[s];
        } else {
            for (int32_t q = s; q < t; ++q) nx = min(nx, a.B.idx[q]);
        }
        mymin = min(mymin, nx);
        cur_of[i] = s;
        next_of[i] = nx;
    }
    int32_t cmin = block_min_i32<THREADS>(mymin, sh);
    int64_t run = 0;
    while (cmin != INT_MAX) {
        const int32_t c_lo = (cmin / W) * W;
        const int64_t c_hi = (int64_t)c_lo + W;
        mymin = INT_MAX;
        for (int32_t g = warp * 32; g < nA; g += NW * 32) {
            const int32_t nxl = g + lane < nA ? next_of[g + lane] : INT_MAX;
            unsigned act = __ballot_sync(FULL, nxl < c_hi);
            if (nxl >= c_hi) mymin = min(mymin, nxl);
            while (act) {
                const int q = __ffs(act) - 1;
                act &= act - 1u;
                const int32_t i = g + q;
                const int32_t k = a.A.idx[e0 + i];
                const int32_t end = a.B.ptr[k + 1];
                const double av = a.A.val[e0 + i];
                int32_t cur = SORTED ? cur_of[i] : a.B.ptr[k];
                int32_t nxt = INT_MAX;
                if constexpr (SORTED) {
                    for (;;) {
                        const int32_t p = cur + lane;
                        const int32_t c = p < end ? a.B.idx[p] : INT_MAX;
                        const bool v = c < c_hi;
                        const unsigned m = __ballot_sync(FULL, v);
                        // cursors never point below the window (it starts at the
                        // smallest next column); the guard keeps a malformed row
                        // inside shared memory all the same
                        const int rel = v ? max(c - c_lo, 0) : 0;
                        if (v) atomic_fma(&dense[rel], av, a.B.val[p]);
                        or_bit(bits, v, (uint32_t)rel);
                        const int n = __popc(m);
                        cur += n;
                        if (n < 32) {
                            nxt = __shfl_sync(FULL, c, n);
                            break;
                        }
                    }
                } else {
                    for (int32_t q0 = cur; q0 < end; q0 += 32) {
                        const int32_t p = q0 + lane;
                        const int32_t c = p < end ? a.B.idx[p] : INT_MAX;
                        const bool v = c >= c_lo && c < c_hi;
                        const int rel = v ? c - c_lo : 0;
                        if (v) atomic_fma(&dense[rel], av, a.B.val[p]);
                        or_bit(bits, v, (uint32_t)rel);
                        if (!v && c >= c_hi) nxt = min(nxt, c);
                    }
#pragma unroll
                    for (int d = 16; d; d >>= 1) nxt = min(nxt, __shfl_xor_sync(FULL, nxt, d));
                }
                mymin = min(mymin, nxt);
                if (lane == 0) {
                    if constexpr (SORTED) cur_of[i] = cur;
                    next_of[i] = nxt;
                }
            }
        }
        __syncthreads();
        uint32_t word = tid < W / 32 ? bits[tid] : 0u;
        if (tid < W / 32) bits[tid] = 0u;
        int32_t tot;
        const int32_t off = block_excl_scan<THREADS>(__popc(word), &tot, sh);
        int64_t pos = run + off;
        while (word) {
            const int b = __ffs(word) - 1;
            word &= word - 1u;
            const int rel = tid * 32 + b;
            if (pos < expect) {
                a.Ci[obase + pos] = c_lo - shift + rel;
                a.Cv[obase + pos] = dense[rel];
            }
            dense[rel] = 0.0;
            ++pos;
        }
        run += tot;
        cmin = block_min_i32<THREADS>(mymin, sh);
    }
    if (tid == 0 && run != expect) raise(a.err, DEV_COUNT_MISMATCH);
}

// Configurations and their dynamic shared memory.
constexpr int kSymWarpRows = 8;
constexpr int kNumWarpRows = 4;
constexpr int kSymCtaThreads = 256;
constexpr int kNumCtaSThreads = 256;
constexpr int kNumCtaLThreads = 512;
constexpr int kDenseThreads = 512;
constexpr int kDenseStage = 1024;  // entries whose cursors stay in shared memory
constexpr int kWideThreads = 512;       // two or more CTAs per SM
constexpr size_t kSmemSymWarp = (size_t)kSymWarpRows * kSymWarpTable * 4;
constexpr size_t kSmemSymCta = StageLayout<kSymCtaThreads>::bytes + (size_t)kSymCtaTable * 4;
constexpr size_t kSmemNumWarp = (size_t)kNumWarpRows * warp_hash_bytes(kNumWarpTable);
constexpr size_t kSmemNumCtaS = StageLayout<kNumCtaSThreads>::bytes + (size_t)kNumCtaSTable * 12;
constexpr size_t kSmemNumCtaL = StageLayout<kNumCtaLThreads>::bytes + (size_t)kNumCtaLTable * 12;
constexpr size_t kSmemDense = (size_t)kDenseWindow * 8 + kDenseWindow / 8 + (size_t)kDenseStage * 8;
constexpr size_t kSmemWideBase = StageLayout<kWideThreads>::bytes;
constexpr int kBitwRows = 8;
constexpr int kRankwRows = 8;
constexpr int kDensewRows = 4;  // 8 rows a CTA: 8.2 ms where 4 take 7.9
constexpr int kGdenseThreads = 512;
constexpr int kRankWinThreads = 512;  // two CTAs per SM: one works while the other waits at a barrier
constexpr int kRankWinWords = 16384;  // 2^19 columns per window
constexpr size_t kSmemRankWin = rank_bits_at(kRankWinThreads) + 6 * (size_t)kRankWinWords +
                                4 * (size_t)(kRankWinWords / 256) + 12 * (size_t)kRankWinThreads;
constexpr size_t kSmemGdenseBase = StageLayout<kGdenseThreads>::bytes;
constexpr size_t kSmemDscr = StageLayout<kRankWinThreads>::bytes + 4 * (size_t)kRankWinWords;
constexpr int kRankmRows = 5;  // 14.6 KiB per warp: three CTAs (15 warps) per SM
constexpr size_t kSmemRankm =
    (size_t)kRankmRows * (6 * (size_t)kMidSpanWords + 4 * (size_t)(kMidSpanWords / 32) + 8 * (size_t)kNumWarpMax);

}  // namespace

// Dynamic shared memory of the rank kernel: staging, bitmap and pair ranks of
// maxWords words, and the small CTAs' values.
static size_t smem_rank(int threads, int maxWords) {
    const bool small = threads == kRankSThreads;
    return rank_bits_at(threads) + 4 * (size_t)maxWords + (small ? 2 : 4) * (size_t)(maxWords / 2) +
           (small ? 8 * (size_t)kRankVals : 0);
}

// Words of the rank kernels' bitmap: the threshold's, or all of C's columns
// where they take fewer (a multiple of 4, as threads own aligned quads).
static int rank_words(const Tuning &t, int64_t ncols) {
    return (int)((std::min<int64_t>(t.rankWordsMax, ncols / 32 + 1) + 3) / 4 * 4);
}

void init_kernel_attributes() {
    cudaFuncSetAttribute(k_sym_hash_warp<kSymWarpRows, kSymWarpTable>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemSymWarp);
    cudaFuncSetAttribute(k_sym_hash_cta<kSymCtaThreads, kSymCtaTable>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemSymCta);
    for (const void *fn : {(const void *)k_sym_wide<kWideThreads, false>, (const void *)k_sym_wide<kWideThreads, true>})
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kSmemWideBase + kWideWindowBitsMax / 8 + 4 * (size_t)kWideTouchMax +
                                   4 * kWideThreads));
    cudaFuncSetAttribute(k_num_hash_warp<kNumWarpRows, kNumWarpTable>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemNumWarp);
    cudaFuncSetAttribute(k_num_hash_cta<kNumCtaSThreads, kNumCtaSTable>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemNumCtaS);
    cudaFuncSetAttribute(k_num_hash_cta<kNumCtaLThreads, kNumCtaLTable>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemNumCtaL);
    cudaFuncSetAttribute(k_num_dense<kDenseThreads, kDenseWindow, kDenseStage, true>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemDense);
    cudaFuncSetAttribute(k_num_dense<kDenseThreads, kDenseWindow, kDenseStage, false>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemDense);
    cudaFuncSetAttribute(k_num_rank<kRankSThreads, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_rank(kRankSThreads, kRankWordsMax));
    cudaFuncSetAttribute(k_num_rank<kRankLThreads, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_rank(kRankLThreads, kRankWordsMax));
    cudaFuncSetAttribute(k_num_rankm<kRankmRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemRankm);
    cudaFuncSetAttribute(k_num_rankwin<kRankWinThreads, kRankWinWords>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemRankWin);
    cudaFuncSetAttribute(k_num_dscr<kRankWinThreads, kRankWinWords>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemDscr);
    cudaFuncSetAttribute(k_num_gdense<kGdenseThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(kSmemGdenseBase + 4 * (size_t)kGdenseSumMax));
    // The device-driven forms of the same kernels.
    cudaFuncSetAttribute(k_sym_hash_warp_dd<kSymWarpRows, kSymWarpTable>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemSymWarp);
    cudaFuncSetAttribute(k_sym_hash_cta_dd<kSymCtaThreads, kSymCtaTable>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemSymCta);
    cudaFuncSetAttribute(k_num_hash_warp_dd<kNumWarpRows, kNumWarpTable>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemNumWarp);
    cudaFuncSetAttribute(k_num_hash_cta_dd<kNumCtaSThreads, kNumCtaSTable>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemNumCtaS);
    cudaFuncSetAttribute(k_num_hash_cta_dd<kNumCtaLThreads, kNumCtaLTable>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemNumCtaL);
    cudaFuncSetAttribute(k_num_rank_dd<kRankSThreads, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_rank(kRankSThreads, kRankWordsMax));
    cudaFuncSetAttribute(k_num_rank_dd<kRankLThreads, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_rank(kRankLThreads, kRankWordsMax));
}

// Loads every symbolic and numeric kernel of this file now.  CUDA loads
// kernels lazily (on first launch) by default; a caller that must not have
// the CUDA driver allocate during a later call (the allocation-free entry point)
// has them loaded at its set-up instead.  Returns the first error.
cudaError_t preload_spgemm_kernels() {
    const void *fns[] = {
        (const void *)k_sym_tiny,
        (const void *)k_sym_flagw<kBitwRows>,
        (const void *)k_sym_hash_warp<kSymWarpRows, kSymWarpTable>,
        (const void *)k_sym_hash_cta<kSymCtaThreads, kSymCtaTable>,
        (const void *)k_sym_items,
        (const void *)k_sym_wide<kWideThreads, false>,
        (const void *)k_sym_wide<kWideThreads, true>,
        (const void *)k_num_tiny,
        (const void *)k_num_hash_warp<kNumWarpRows, kNumWarpTable>,
        (const void *)k_num_densew<kDensewRows, 3>,
        (const void *)k_num_densew<kDensewRows, 6>,
        (const void *)k_num_rankm<kRankmRows>,
        (const void *)k_num_rankw<kRankwRows>,
        (const void *)k_num_rank<kRankSThreads, uint16_t>,
        (const void *)k_num_rank<kRankLThreads, int32_t>,
        (const void *)k_num_hash_cta<kNumCtaSThreads, kNumCtaSTable>,
        (const void *)k_num_hash_cta<kNumCtaLThreads, kNumCtaLTable>,
        (const void *)k_num_rankwin<kRankWinThreads, kRankWinWords>,
        (const void *)k_dense_items,
        (const void *)k_num_dscr<kRankWinThreads, kRankWinWords>,
        (const void *)k_num_gdense<kGdenseThreads>,
        (const void *)k_num_dense<kDenseThreads, kDenseWindow, kDenseStage, true>,
        (const void *)k_num_dense<kDenseThreads, kDenseWindow, kDenseStage, false>,
    };
    for (const void *f : fns) {
        cudaFuncAttributes fa;
        const cudaError_t e = cudaFuncGetAttributes(&fa, f);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

static int wide_window_bits(int64_t ncols) {
    int64_t w = 32;
    while (w < ncols && w < kWideWindowBitsMax) w <<= 1;
    return (int)w;
}

static size_t smem_wide(int winBits) {
    return kSmemWideBase + (size_t)winBits / 8 + 4 * (size_t)wide_touch_cap(winBits) + 4 * kWideThreads;
}

static int64_t wide_grid(int winBits, int sms) {
    const int per_sm = std::max(1, std::min(2048 / kWideThreads, (int)((227 * 1024) / (smem_wide(winBits) + 1024))));
    return (int64_t)std::max(sms, 1) * per_sm;
}

void launch_symbolic_items(const SymArgs &a, int32_t begin, int32_t n, cudaStream_t s, int *launches) {
    const int wb = wide_window_bits(a.B.n);
    k_sym_items<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(a, begin, n);
    k_sym_wide<kWideThreads, true>
        <<<(unsigned)wide_grid(wb, a.numSms), kWideThreads, smem_wide(wb), s>>>(a, begin, 0, wb);
    *launches += 2;
}

// Symbolic kernel of bin b over list[begin, begin + n).
void launch_symbolic_bin(const SymArgs &a, int bin, int32_t begin, int32_t n, cudaStream_t s,
                         int *launches) {
    if (n <= 0) return;
    switch (bin) {
        case SB_TINY:
            k_sym_tiny<<<(unsigned)ceil_div(n, 32 * kSymTinyWarps), 32 * kSymTinyWarps, 0, s>>>(a, begin, n);
            break;
        case SB_BITW:
            k_sym_flagw<kBitwRows><<<(unsigned)ceil_div(n, kBitwRows), 32 * kBitwRows, 0, s>>>(a, begin, n);
            break;
        case SB_HWARP:
            k_sym_hash_warp<kSymWarpRows, kSymWarpTable>
                <<<(unsigned)ceil_div(n, kSymWarpRows), 32 * kSymWarpRows, kSmemSymWarp, s>>>(a, begin, n);
            break;
        case SB_HCTA:
            k_sym_hash_cta<kSymCtaThreads, kSymCtaTable><<<(unsigned)n, kSymCtaThreads, kSmemSymCta, s>>>(a, begin);
            break;
        case SB_WIDE: {
            // Persistent: as many CTAs as fit on the GPU at once (two per SM
            // with the widest window), rows taken from a counter.
            const int wb = wide_window_bits(a.B.n);
            const int grid = (int)std::min<int64_t>(n, wide_grid(wb, a.numSms));
            k_sym_wide<kWideThreads, false><<<(unsigned)grid, kWideThreads, smem_wide(wb), s>>>(a, begin, n, wb);
            break;
        }
        default:
            return;
    }
    ++*launches;
}

// Resident CTAs of kernel fn on the whole GPU (the grid of a device-driven
// launch, which strides over however many rows its bin holds).
// The occupancy is looked up once per kernel and shared-memory size, so
// that launches inside a stream capture query nothing.
static int resident_grid(const void *fn, int threads, size_t smem, int sms) {
    struct Entry {
        const void *fn;
        size_t smem;
        int per_sm;
    };
    static std::mutex mu;
    static std::vector<Entry> cache;
    std::lock_guard<std::mutex> lk(mu);
    for (const Entry &e : cache)
        if (e.fn == fn && e.smem == smem) return e.per_sm * std::max(sms, 1);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    cache.push_back(Entry{fn, smem, per_sm});
    return per_sm * std::max(sms, 1);
}

void launch_symbolic_bin_dd(const SymArgs &a, int bin, cudaStream_t s, int *launches) {
    switch (bin) {
        case SB_TINY: {
            const void *fn = (const void *)k_sym_tiny_dd;
            k_sym_tiny_dd<<<resident_grid(fn, 32 * kSymTinyWarps, 0, a.numSms), 32 * kSymTinyWarps, 0, s>>>(a, bin);
            break;
        }
        case SB_BITW: {
            const void *fn = (const void *)k_sym_flagw_dd<kBitwRows>;
            k_sym_flagw_dd<kBitwRows><<<resident_grid(fn, 32 * kBitwRows, 0, a.numSms), 32 * kBitwRows, 0, s>>>(a, bin);
            break;
        }
        case SB_HWARP: {
            const void *fn = (const void *)k_sym_hash_warp_dd<kSymWarpRows, kSymWarpTable>;
            k_sym_hash_warp_dd<kSymWarpRows, kSymWarpTable>
                <<<resident_grid(fn, 32 * kSymWarpRows, kSmemSymWarp, a.numSms), 32 * kSymWarpRows, kSmemSymWarp, s>>>(
                    a, bin);
            break;
        }
        case SB_HCTA: {
            const void *fn = (const void *)k_sym_hash_cta_dd<kSymCtaThreads, kSymCtaTable>;
            k_sym_hash_cta_dd<kSymCtaThreads, kSymCtaTable>
                <<<resident_grid(fn, kSymCtaThreads, kSmemSymCta, a.numSms), kSymCtaThreads, kSmemSymCta, s>>>(a, bin);
            break;
        }
        case SB_WIDE: {
            const int wb = wide_window_bits(a.B.n);
            const size_t smem = smem_wide(wb);
            const void *fn = (const void *)k_sym_wide<kWideThreads, false>;
            k_sym_wide<kWideThreads, false>
                <<<(unsigned)resident_grid(fn, kWideThreads, smem, a.numSms), kWideThreads, smem, s>>>(a, -1, 0, wb);
            break;
        }
        default:
            return;
    }
    ++*launches;
}

// Device-driven numeric launch of bin `bin` (rows from a.binStart on the
// device): persistent grids, the dense bin on rank windows without pieces.
void launch_numeric_bin_dd(const NumArgs &a, int bin, cudaStream_t s, int *launches) {
    switch (bin) {
        case NB_TINY: {
            const void *fn = (const void *)k_num_tiny_dd;
            k_num_tiny_dd<<<resident_grid(fn, 32 * kNumTinyWarps, 0, a.numSms), 32 * kNumTinyWarps, 0, s>>>(a, bin);
            break;
        }
        case NB_HWARP: {
            const void *fn = (const void *)k_num_hash_warp_dd<kNumWarpRows, kNumWarpTable>;
            k_num_hash_warp_dd<kNumWarpRows, kNumWarpTable>
                <<<resident_grid(fn, 32 * kNumWarpRows, kSmemNumWarp, a.numSms), 32 * kNumWarpRows, kSmemNumWarp, s>>>(
                    a, bin);
            break;
        }
        case NB_DENSEW: {
            const void *fn = (const void *)k_num_densew_dd<kDensewRows>;
            k_num_densew_dd<kDensewRows><<<resident_grid(fn, 32 * kDensewRows, 0, a.numSms), 32 * kDensewRows, 0, s>>>(
                a, bin);
            break;
        }
        case NB_RANKM: {
            const int grid = std::max(a.numSms, 1) * 3;
            k_num_rankm<kRankmRows><<<(unsigned)grid, 32 * kRankmRows, kSmemRankm, s>>>(a, -1, 0);
            break;
        }
        case NB_RANKW: {
            const void *fn = (const void *)k_num_rankw_dd<kRankwRows>;
            k_num_rankw_dd<kRankwRows><<<resident_grid(fn, 32 * kRankwRows, 0, a.numSms), 32 * kRankwRows, 0, s>>>(
                a, bin);
            break;
        }
        case NB_RANKS: {
            const int words = rank_words(a.tune, a.B.n);
            const size_t smem = smem_rank(kRankSThreads, words);
            const void *fn = (const void *)k_num_rank_dd<kRankSThreads, uint16_t>;
            k_num_rank_dd<kRankSThreads, uint16_t>
                <<<resident_grid(fn, kRankSThreads, smem, a.numSms), kRankSThreads, smem, s>>>(a, bin, words);
            break;
        }
        case NB_RANKL: {
            const int words = rank_words(a.tune, a.B.n);
            const size_t smem = smem_rank(kRankLThreads, words);
            const void *fn = (const void *)k_num_rank_dd<kRankLThreads, int32_t>;
            k_num_rank_dd<kRankLThreads, int32_t>
                <<<resident_grid(fn, kRankLThreads, smem, a.numSms), kRankLThreads, smem, s>>>(a, bin, words);
            break;
        }
        case NB_HCTA_S: {
            const void *fn = (const void *)k_num_hash_cta_dd<kNumCtaSThreads, kNumCtaSTable>;
            k_num_hash_cta_dd<kNumCtaSThreads, kNumCtaSTable>
                <<<resident_grid(fn, kNumCtaSThreads, kSmemNumCtaS, a.numSms), kNumCtaSThreads, kSmemNumCtaS, s>>>(a,
                                                                                                               bin);
            break;
        }
        case NB_HCTA_L: {
            const void *fn = (const void *)k_num_hash_cta_dd<kNumCtaLThreads, kNumCtaLTable>;
            k_num_hash_cta_dd<kNumCtaLThreads, kNumCtaLTable>
                <<<resident_grid(fn, kNumCtaLThreads, kSmemNumCtaL, a.numSms), kNumCtaLThreads, kSmemNumCtaL, s>>>(a,
                                                                                                               bin);
            break;
        }
        case NB_DENSE: {
            cudaMemsetAsync(a.ctr + CTR_NUM_RANKWIN, 0, sizeof(uint32_t), s);
            const void *fn = (const void *)k_num_rankwin<kRankWinThreads, kRankWinWords>;
            k_num_rankwin<kRankWinThreads, kRankWinWords>
                <<<resident_grid(fn, kRankWinThreads, kSmemRankWin, a.numSms), kRankWinThreads, kSmemRankWin, s>>>(a, -1,
                                                                                                              0);
            break;
        }
        default:
            return;
    }
    ++*launches;
}

// Looks up the grids of every device-driven launch for these thresholds and
// B's column count ahead of any stream capture.
void prepare_dd_grids(const Tuning &t, int64_t bcols, int sms) {
    const int wb = wide_window_bits(bcols);
    resident_grid((const void *)k_sym_tiny_dd, 32 * kSymTinyWarps, 0, sms);
    resident_grid((const void *)k_sym_flagw_dd<kBitwRows>, 32 * kBitwRows, 0, sms);
    resident_grid((const void *)k_sym_hash_warp_dd<kSymWarpRows, kSymWarpTable>, 32 * kSymWarpRows, kSmemSymWarp, sms);
    resident_grid((const void *)k_sym_hash_cta_dd<kSymCtaThreads, kSymCtaTable>, kSymCtaThreads, kSmemSymCta, sms);
    resident_grid((const void *)k_sym_wide<kWideThreads, false>, kWideThreads, smem_wide(wb), sms);
    resident_grid((const void *)k_num_tiny_dd, 32 * kNumTinyWarps, 0, sms);
    resident_grid((const void *)k_num_hash_warp_dd<kNumWarpRows, kNumWarpTable>, 32 * kNumWarpRows, kSmemNumWarp, sms);
    resident_grid((const void *)k_num_densew_dd<kDensewRows>, 32 * kDensewRows, 0, sms);
    resident_grid((const void *)k_num_rankw_dd<kRankwRows>, 32 * kRankwRows, 0, sms);
    resident_grid((const void *)k_num_rank_dd<kRankSThreads, uint16_t>, kRankSThreads,
                  smem_rank(kRankSThreads, rank_words(t, bcols)), sms);
    resident_grid((const void *)k_num_rank_dd<kRankLThreads, int32_t>, kRankLThreads,
                  smem_rank(kRankLThreads, rank_words(t, bcols)), sms);
    resident_grid((const void *)k_num_hash_cta_dd<kNumCtaSThreads, kNumCtaSTable>, kNumCtaSThreads, kSmemNumCtaS, sms);
    resident_grid((const void *)k_num_hash_cta_dd<kNumCtaLThreads, kNumCtaLTable>, kNumCtaLThreads, kSmemNumCtaL, sms);
    resident_grid((const void *)k_num_rankwin<kRankWinThreads, kRankWinWords>, kRankWinThreads, kSmemRankWin, sms);
    resident_grid((const void *)k_num_rankm<kRankmRows>, 32 * kRankmRows, kSmemRankm, sms);
}

void launch_numeric_bin(const NumArgs &a, int bin, int32_t lo, int32_t hi, cudaStream_t s,
                        int *launches) {
    const int32_t n = hi - lo;
    if (n <= 0) return;
    switch (bin) {
        case NB_TINY:
            k_num_tiny<<<(unsigned)ceil_div(n, 32 * kNumTinyWarps), 32 * kNumTinyWarps, 0, s>>>(a, lo, n);
            break;
        case NB_HWARP:
            k_num_hash_warp<kNumWarpRows, kNumWarpTable>
                <<<(unsigned)ceil_div(n, kNumWarpRows), 32 * kNumWarpRows, kSmemNumWarp, s>>>(a, lo, n);
            break;
        case NB_DENSEW:
            if (n <= kDensewFew * std::max(a.numSms, 1))
                k_num_densew<kDensewRows, 6><<<(unsigned)ceil_div(n, kDensewRows), 32 * kDensewRows, 0, s>>>(a, lo, n);
            else
                k_num_densew<kDensewRows, 3><<<(unsigned)ceil_div(n, kDensewRows), 32 * kDensewRows, 0, s>>>(a, lo, n);
            break;
        case NB_RANKM: {
            // Persistent: three CTAs of kRankmRows warps per SM.
            const int grid = (int)std::min<int64_t>(ceil_div(n, kRankmRows), (int64_t)std::max(a.numSms, 1) * 3);
            k_num_rankm<kRankmRows><<<(unsigned)grid, 32 * kRankmRows, kSmemRankm, s>>>(a, lo, n);
            break;
        }
        case NB_RANKW:
            k_num_rankw<kRankwRows><<<(unsigned)ceil_div(n, kRankwRows), 32 * kRankwRows, 0, s>>>(a, lo, n);
            break;
        case NB_RANKS: {
            const int words = rank_words(a.tune, a.B.n);
            k_num_rank<kRankSThreads, uint16_t>
                <<<(unsigned)n, kRankSThreads, smem_rank(kRankSThreads, words), s>>>(a, lo, words);
            break;
        }
        case NB_RANKL: {
            const int words = rank_words(a.tune, a.B.n);
            k_num_rank<kRankLThreads, int32_t>
                <<<(unsigned)n, kRankLThreads, smem_rank(kRankLThreads, words), s>>>(a, lo, words);
            break;
        }
        case NB_HCTA_S:
            k_num_hash_cta<kNumCtaSThreads, kNumCtaSTable><<<(unsigned)n, kNumCtaSThreads, kSmemNumCtaS, s>>>(a, lo);
            break;
        case NB_HCTA_L:
            k_num_hash_cta<kNumCtaLThreads, kNumCtaLTable><<<(unsigned)n, kNumCtaLThreads, kSmemNumCtaL, s>>>(a, lo);
            break;
        case NB_DENSE:
            if (a.tune.denseMethod == 0) {
                cudaMemsetAsync(a.ctr + CTR_NUM_RANKWIN, 0, sizeof(uint32_t), s);
                const int per_sm = std::max(1, (int)((227 * 1024) / (kSmemRankWin + 1024)));
                int64_t work = n;
                if (a.items) {
                    // Heavy rows cut into pieces: the items are built on the
                    // device, so the grid is the persistent one.
                    cudaMemsetAsync(a.ctr + CTR_ITEMS, 0, sizeof(uint32_t), s);
                    k_dense_items<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(a, lo, n);
                    ++*launches;
                    work = (int64_t)a.itemCap;
                }
                const int grid = (int)std::min<int64_t>(work, (int64_t)std::max(a.numSms, 1) * per_sm);
                k_num_rankwin<kRankWinThreads, kRankWinWords>
                    <<<(unsigned)grid, kRankWinThreads, kSmemRankWin, s>>>(a, lo, n);
            } else if (a.tune.denseMethod == 3 && a.scr) {
                cudaMemsetAsync(a.ctr + CTR_NUM_DSCR, 0, sizeof(uint32_t), s);
                const int grid = (int)std::min<int64_t>(n, a.scrSlots);
                k_num_dscr<kRankWinThreads, kRankWinWords><<<(unsigned)grid, kRankWinThreads, kSmemDscr, s>>>(a, lo, n);
            } else if (a.tune.denseMethod == 1 && a.gBits) {
                cudaMemsetAsync(a.ctr + CTR_NUM_GDENSE, 0, sizeof(uint32_t), s);
                const int grid = (int)std::min<int64_t>(n, a.gSlots);
                const size_t smem = kSmemGdenseBase + 4 * (size_t)(a.gStride >> 10);
                k_num_gdense<kGdenseThreads><<<(unsigned)grid, kGdenseThreads, smem, s>>>(a, lo, n);
            } else if (a.bSorted)
                k_num_dense<kDenseThreads, kDenseWindow, kDenseStage, true>
                    <<<(unsigned)n, kDenseThreads, kSmemDense, s>>>(a, lo);
            else
                k_num_dense<kDenseThreads, kDenseWindow, kDenseStage, false>
                    <<<(unsigned)n, kDenseThreads, kSmemDense, s>>>(a, lo);
            break;
        default:
            return;
    }
    ++*launches;
}

}  // namespace dbd
