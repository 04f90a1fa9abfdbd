// Device helpers of the CTA kernels: block scans, a batch of one A row's
// entries staged in shared memory, and a warp's walk over its products.
#pragma once

#include <climits>

#include "dbd_internal.h"
#include "warp_chunk.cuh"

namespace dbd {
namespace {

template <int THREADS>
__device__ __forceinline__ int32_t block_excl_scan(int32_t v, int32_t *total, int32_t *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int32_t y = __shfl_up_sync(FULL, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    int32_t base = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < THREADS / 32; ++i) {
        const int32_t s = sh[i];
        if (i < w) base += s;
        tot += s;
    }
    __syncthreads();
    *total = tot;
    return base + x - v;
}

// Lower bound of target in the ascending bi (the first index whose column
// is >= target), known to lie in [l, h], found by the group of m aligned
// lanes this lane belongs to (m a power of two, lg = log2 m): each step the
// m lanes probe the midpoints of m equal slices of [l, h) at once and the
// range shrinks about m times.  m = 1 is a binary search.  Every lane of
// the warp calls; lanes with l == h wait for their warp.
__device__ __forceinline__ int32_t group_lower_bound(const int32_t *bi, int32_t l, int32_t h, int64_t target,
                                                    int lg) {
    const int lane = threadIdx.x & 31;
    const int m = 1 << lg;
    const int j = lane & (m - 1);
    const int base = lane & ~(m - 1);
    const uint32_t gm = m == 32 ? FULL : (1u << m) - 1u;
    while (__any_sync(FULL, l < h)) {
        const int64_t n = h - l;
        const bool act = l < h;
        const int32_t p = l + (int32_t)((n * (2 * j + 1)) >> (lg + 1));
        const bool below = act && (int64_t)__ldg(&bi[p]) < target;
        const int c = __popc((__ballot_sync(FULL, below) >> base) & gm);
        if (act) {
            // The group's first c probes are below target (bi ascends).
            const int32_t nl = c > 0 ? l + (int32_t)((n * (2 * c - 1)) >> (lg + 1)) + 1 : l;
            const int32_t nh = c < m ? l + (int32_t)((n * (2 * c + 1)) >> (lg + 1)) : h;
            l = nl;
            h = nh;
        }
    }
    return l;
}

// A batch of up to THREADS entries of one A row staged in shared memory,
// keeping only entries whose B row is non-empty: pre[i] = exclusive prefix
// of |B_k| (pre[*nb] = the batch's products), bst[i] = first position of B_k,
// av[i] = A value.  Every staged entry has at least one product, so 32
// consecutive products span at most 32 entries.  Returns the products.
// With clip (B's rows ascending), each entry keeps only the part of its B
// row inside the column window [cLo, cHi), so a row walked window by window
// enumerates each product once.  The two ends of each part are lower-bound
// searches over the B row, which are dependent L2 loads: an entry gets
// as many lanes as the batch leaves free (up to 32), half searching each
// end, so that the CTA waits a few probes instead of two binary searches.
// With cur (a row walked through consecutive windows with the same batch),
// cur[i] carries where entry i's part of the previous window ended, which
// is where this window's starts (carry), and all the entry's lanes search
// the other end.
template <int THREADS, bool VALS>
__device__ __forceinline__ int32_t stage_entries(const CsrDev &A, const CsrDev &B, int32_t eb, int n_in,
                                                 int32_t *pre, int32_t *bst, double *av, int *nb,
                                                 int32_t *sh, bool clip = false, int64_t cLo = 0,
                                                 int64_t cHi = 0, int32_t *cur = nullptr, bool carry = false,
                                                 int32_t *src = nullptr) {
    const int tid = threadIdx.x;
    int32_t len = 0, s = 0;
    double a = 0.0;
    if (!clip) {
        if (tid < n_in) {
            const int32_t k = A.idx[eb + tid];
            s = B.ptr[k];
            len = B.ptr[k + 1] - s;
            if constexpr (VALS) a = A.val[eb + tid];
        }
    } else {
        // Lanes per entry: L = 2^lgL, the largest with n_in L <= THREADS.
        int lgL = 0;
        while (lgL < 5 && n_in * (2 << lgL) <= THREADS) ++lgL;
        const int L = 1 << lgL;
        const int ent = tid >> lgL, sub = tid & (L - 1);
        int32_t rs = 0, rl = 0;
        if (ent < n_in) {
            const int32_t k = A.idx[eb + ent];
            rs = B.ptr[k];
            rl = B.ptr[k + 1] - rs;
        }
        const int32_t *bi = B.idx + rs;
        bool needLo = false, needHi = false;
        int32_t a0 = 0;
        if (rl > 0) {
            if (carry) a0 = cur[ent] - rs;
            else needLo = (int64_t)__ldg(&bi[0]) < cLo;
            needHi = (int64_t)__ldg(&bi[rl - 1]) >= cHi;
        }
        int32_t lo, hi;
        if (carry || L == 1) {
            // One search per group of L lanes (L == 1: both ends in turn);
            // the lanes of a group reach the same bounds.
            int32_t r0 = a0;
            if (!carry) r0 = group_lower_bound(bi, needLo ? 1 : 0, needLo ? rl : 0, cLo, 0);
            lo = r0;
            hi = group_lower_bound(bi, needHi ? r0 : rl, needHi ? rl - 1 : rl, cHi, lgL);
        } else {
            // Lanes [0, L/2) of the group find the start, [L/2, L) the end
            // (one call site: the searches hold warp votes).
            const bool upper = sub >= L / 2;
            const int32_t l0 = upper ? (needHi ? 0 : rl) : (needLo ? 1 : 0);
            const int32_t h0 = upper ? (needHi ? rl - 1 : rl) : (needLo ? rl : 0);
            const int32_t r = group_lower_bound(bi, l0, h0, upper ? cHi : cLo, lgL - 1);
            const int g0 = (tid & 31) & ~(L - 1);
            lo = __shfl_sync(FULL, r, g0);
            hi = __shfl_sync(FULL, r, g0 + L / 2);
        }
        if (ent < n_in && sub == 0) {
            s = rs + lo;
            len = max(0, hi - lo);
            if (cur) cur[ent] = rs + max(hi, lo);
            if constexpr (VALS) a = A.val[eb + ent];
        }
    }
    int32_t total, kept;
    const int32_t ex = block_excl_scan<THREADS>(len, &total, sh);
    const int32_t slot = block_excl_scan<THREADS>(len > 0 ? 1 : 0, &kept, sh);
    if (len > 0) {
        pre[slot] = ex;
        bst[slot] = s;
        if constexpr (VALS) av[slot] = a;
        if (src) src[slot] = eb + tid;  // without clip, a thread's entry is eb + tid
    }
    if (tid == 0) pre[kept] = total;
    *nb = kept;
    __syncthreads();
    return total;
}

// Largest i in [0, nb) with pre[i] <= t.
__device__ __forceinline__ int find_entry(const int32_t *pre, int nb, int32_t t) {
    int lo = 0, hi = nb - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Where a warp's walk over a staged batch stands: the entry e0 of the last
// product placed, its first product p0 and B position b0, and the first
// product p1 of the entry behind it.
struct RangeWalk {
    int e0;
    int32_t p0, b0, p1;
    __device__ __forceinline__ RangeWalk(const int32_t *pre, const int32_t *bst, int nb, int32_t tb) {
        e0 = find_entry(pre, nb, tb);
        p0 = pre[e0];
        b0 = bst[e0];
        p1 = e0 + 1 < nb ? pre[e0 + 1] : INT_MAX;
    }
    // B positions and entries of the U * 32 products from g0 on (below te).  A
    // step whose products all lie in the current entry (long B rows) takes
    // their positions from registers; otherwise the entries' starts within the
    // step make a mask (one OR over the warp), whose bits up to a lane's own
    // give its entry and its place in the entry's B row.  (A 5-step shuffle
    // search among the starts took 15 more instructions and a chain of five
    // shuffles: symbolic wide rows of R-MAT 2^18 1.37 -> 1.26 ms, 2^16 0.52 ->
    // 0.45, dense rows of 2^21 3.70 -> 3.62.)
    template <int U>
    __device__ __forceinline__ void place(const int32_t *pre, const int32_t *bst, int nb, int32_t g0, int32_t te,
                                          int32_t (&pos)[U], int (&ent)[U], bool (&val)[U]) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int32_t t0 = g0 + 32 * u;
            const int32_t t = t0 + lane;
            val[u] = t < te;
            ent[u] = e0;
            pos[u] = b0 + (t - p0);
            if (t0 >= te || p1 > t0 + 31) continue;  // past the range, or all in entry e0
            const int ej = e0 + 1 + lane;
            const uint32_t at = ej < nb ? (uint32_t)(pre[ej] - t0) : 32u;  // not before t0
            const uint32_t starts = __reduce_or_sync(FULL, at < 32u ? 1u << at : 0u);
            const uint32_t upto = starts & (FULL >> (31 - lane));
            const int e = e0 + __popc(upto);
            ent[u] = e;
            pos[u] = bst[e] + (upto ? lane + __clz(upto) - 31 : t - p0);
            e0 += __popc(starts);
            p0 = t0 + 31 - __clz(starts);
            b0 = bst[e0];
            p1 = e0 + 1 < nb ? pre[e0 + 1] : INT_MAX;
        }
    }
};

// One warp walks products [tb, te) of a staged batch, 32 per step, in
// groups of U steps whose B loads are all issued before any is used:
// ld(pos) reads what a product needs from B (read-only loads), use(valid, x,
// e) consumes it on every lane (e = staged entry; meaningful when valid).
// A warp keeps U loads in flight instead of one, which hides the L2 latency
// of B's rows.  use is called by all lanes for each step, so it may hold
// warp collectives.
template <int U, class LD, class USE>
__device__ __forceinline__ void warp_range_ld(const int32_t *pre, const int32_t *bst, int nb, int32_t tb,
                                              int32_t te, LD &&ld, USE &&use) {
    if (tb >= te) return;
    RangeWalk walk(pre, bst, nb, tb);
    for (int32_t g0 = tb; g0 < te; g0 += 32 * U) {
        int32_t pos[U];
        int ent[U];
        bool val[U];
        walk.template place<U>(pre, bst, nb, g0, te, pos, ent, val);
        using T = decltype(ld(0));
        T x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = val[u] ? ld(pos[u]) : T{};
#pragma unroll
        for (int u = 0; u < U; ++u) use(val[u], x[u], ent[u]);
    }
}

// Contiguous share of [0, total) for this warp, in multiples of 32 products.
template <int THREADS>
__device__ __forceinline__ void warp_share(int32_t total, int32_t *tb, int32_t *te) {
    constexpr int NW = THREADS / 32;
    const int64_t per = ((int64_t)total + NW * 32 - 1) / (NW * 32) * 32;
    const int64_t b = (int64_t)(threadIdx.x >> 5) * per;
    *tb = (int32_t)(b < total ? b : (int64_t)total);
    *te = (int32_t)(b + per < total ? b + per : (int64_t)total);
}

// Shared-memory layout of the staged entries (after an 8-aligned prefix).
template <int ECAP>
struct StageLayout {
    static constexpr size_t pre = 0;                              // int32[ECAP + 1]
    static constexpr size_t bst = ((4 * (ECAP + 1)) + 7) / 8 * 8;  // int32[ECAP]
    static constexpr size_t av = bst + ((4 * ECAP) + 7) / 8 * 8;  // double[ECAP]
    static constexpr size_t bytes = av + 8 * ECAP;
};

}  // namespace
}  // namespace dbd
