// Adjoint kernels (no reference counterpart): gradients of a loss with
// respect to the values of A and B over their fixed patterns, given
// G = dL/dC on the pattern of C = A*B that the forward multiply left on the
// device (CSR, columns ascending in every row):
//   dA = mask_A(G * B^T)   dA(i,k) = sum_j G(i,j) * B(k,j)
//   dB = mask_B(A^T * G)   dB(k,j) = sum_i A(i,k) * G(i,j)
// k_adjoint_rows and k_adjoint_cta take both from A's rows (dB by FP64
// reductions); with the deterministic option dB comes from its own pass over B's
// pattern
// (k_entry_rows, the stable radix sort of k_mtx.cu, k_col_ptr, then the
// k_adjoint_db kernels).
#include "cta_stage.cuh"
#include "dbd_internal.h"
#include "warp_chunk.cuh"

#include <algorithm>

namespace dbd {

namespace {

// Position of column k within C's sorted row [lo, hi), or hi.
__device__ __forceinline__ int64_t find_col(const int32_t *__restrict__ ci, int64_t lo, int64_t hi, int32_t k) {
    const int64_t end = hi;
    while (lo < hi) {
        const int64_t mid = lo + ((hi - lo) >> 1);
        if (ci[mid] < k) lo = mid + 1;
        else hi = mid;
    }
    return (lo < end && ci[lo] == k) ? lo : end;
}

// Rows of C of at most NNZ entries: WARPS warps per row of A.  The row's
// columns and G sit in shared memory, so a product's G(i,j) is a binary
// search there instead of one through L2 (each step of which the product
// would wait for); L lanes take one entry of A at a time, 32 / L entries a warp
// and step and two products of each a lane, so that B rows fill the warp without
// an owner search and an entry's dA is one sum over L lanes.  Two FP64
// instructions a product: the fused multiply-add into dA and the multiply whose
// sum into dB the L2 does.  100k rows of 256 products: 380 -> 242 us.
//
// L follows the mean number of products of 32 entries (30k rows of 200 entries of 1,
// 3 and 5 products: 575, 775 and 1025 us with eight lanes whatever the mean, 232,
// 475 and 690 so); rows of a few entries, which fill no step however few lanes
// they get, take more, whose reductions into dB are next to each other (300k
// rows of 3 entries of 3 products 627 -> 484 us).  A single lane gains for
// entries of one product only (932 -> 863 us) and loses for those of three.
//
// Rows of 513 entries and more take four warps a row: 24 KB a CTA for 2048 of
// them, 12 KB for 1024, which leaves the L1 its room (100k rows of 576 products
// 851 -> 736 us).
constexpr int kAdjWarpNnz = 512, kAdjQuadNnz = 1024, kAdjWideNnz = 2048;
constexpr int kAdjWarps = 4;  // a CTA
constexpr int kAdjCtaThreads = 256, kAdjCtaPerSm = 5;

// Which rows of the CTA bins these kernels take (k_adjoint_split), by the steps
// that one warp would walk.  A step is about 0.08 us of an SM's time, a CTA's
// row 1.5 us a batch of its entries and 1.9 ns a product: rows of few steps for
// their products, whose entries are of like lengths, are worth taking.  100k
// rows of 289, 400, 576 and 1024 products in 17 to 32 entries: 1605, 1683, 1766
// and 2031 us by CTAs, 455, 505, 780 and 1137 so.  Longer walks are left to the
// CTAs, as one row would be the last one running: with 24 steps for a warp 20k
// rows of one entry of 400 products take 291 us instead of 233; with 24 for four
// warps and a product in 45 steps, 1209 us instead of 1137 on the last case
// above.  Power-law graphs stay as they are (R-MAT 2^16 1.10 ms; 1.42 if rows
// were taken by their products alone).
constexpr int kAdjWarpSteps = 32, kAdjQuadSteps = 16, kAdjBase = 20, kAdjPer = 30;

// Lanes an entry, for n entries of P products in all (of each no more than 1024
// counted).
__device__ __forceinline__ int adjoint_lanes(int P, int n) {
    if (n <= 4 || P > 8 * n) return 8;
    return n <= 8 || P > 4 * n ? 4 : 2;
}

// Up to 32 entries of a row (from eb on; each lane holds one), L lanes an entry:
// groups q0 / PER, q0 / PER + WARPS, ... of 32 / L entries.
template <int WARPS, int L>
__device__ __forceinline__ void adjoint_entries(const AdjArgs &a, int32_t eb, int ne, int q0, int32_t bs, int32_t len,
                                                double av, int64_t off, const double *g, const int32_t *c, int nc,
                                                int top) {
    constexpr int PER = 32 / L;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1), grp = lane / L;
    const unsigned gmask = ((1u << L) - 1u) << (lane & (32 - L));
    for (int q = PER * q0; q < ne; q += PER * WARPS) {
        const int32_t s = __shfl_sync(FULL, bs, q + grp), l = __shfl_sync(FULL, len, q + grp);
        const double x = __shfl_sync(FULL, av, q + grp);
        double *keep = nullptr;
        if (a.prod) {
            const int64_t o = __shfl_sync(FULL, off, q + grp);
            if (o + l <= a.prodCap) keep = a.prod + o;
            else raise(a.err, DEV_COUNT_MISMATCH);  // the patterns are not the forward's
        }
        double acc = 0.0;
        for (int32_t i0 = sub; i0 < l; i0 += 2 * L) {
            // Two products a lane in flight.
            int32_t k[2];
            double b[2];
            int at[2] = {0, 0};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int32_t i = i0 + L * u;
                k[u] = i < l ? __ldg(&a.B.idx[s + i]) : -1;
                b[u] = i < l ? __ldg(&a.B.val[s + i]) : 0.0;
            }
            for (int step = top; step >= 1; step >>= 1) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (at[u] + step < nc && c[at[u] + step] <= k[u]) at[u] += step;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (k[u] < 0) continue;
                if (nc == 0 || c[at[u]] != k[u]) {
                    raise(a.err, DEV_COUNT_MISMATCH);
                    continue;
                }
                const double gv = g[at[u]];
                acc = __fma_rn(gv, b[u], acc);
                if (a.dB) atomicAdd(&a.dB[s + i0 + L * u], __dmul_rn(x, gv));
                else if (keep) keep[i0 + L * u] = __dmul_rn(x, gv);
            }
        }
#pragma unroll
        for (int d = L / 2; d; d >>= 1) acc += __shfl_xor_sync(gmask, acc, d, L);
        if (sub == 0 && q + grp < ne) a.dA[eb + q + grp] = acc;
    }
}

template <int WARPS>
__device__ __forceinline__ void adjoint_row(const AdjArgs &a, int32_t e0, int32_t e1, int64_t c0, int nc, double *gs,
                                            int32_t *cs) {
    constexpr int T = 32 * WARPS;
    const int lane = threadIdx.x & 31, w = WARPS == 1 ? 0 : threadIdx.x >> 5, tid = 32 * w + lane;
    for (int i = tid; i < nc; i += T) {
        cs[i] = __ldg(&a.Ci[c0 + i]);
        gs[i] = __ldg(&a.G[c0 + i]);
    }
    if constexpr (WARPS == 1) __syncwarp();
    else __syncthreads();
    int top = 1;
    while (2 * top < nc) top <<= 1;
    int q0 = w;  // 32 entries make two groups of two lanes: the next two warps take the next ones'
    for (int32_t eb = e0; eb < e1; eb += 32, q0 = (q0 + WARPS / 2) % WARPS) {
        int32_t bs = 0, len = 0;
        double av = 0.0;
        int64_t off = 0;
        if (eb + lane < e1) {
            if (a.prod) off = __ldg(&a.off[eb + lane]);
            const int32_t k = __ldg(&a.A.idx[eb + lane]);
            bs = __ldg(&a.B.ptr[k]);
            len = __ldg(&a.B.ptr[k + 1]) - bs;
            av = __ldg(&a.A.val[eb + lane]);
        }
        const int ne = min(32, e1 - eb);
        const int lanes = adjoint_lanes(__reduce_add_sync(FULL, min(len, 1024)), ne);
        if (lanes == 2) adjoint_entries<WARPS, 2>(a, eb, ne, q0, bs, len, av, off, gs, cs, nc, top);
        else if (lanes == 4) adjoint_entries<WARPS, 4>(a, eb, ne, q0, bs, len, av, off, gs, cs, nc, top);
        else adjoint_entries<WARPS, 8>(a, eb, ne, q0, bs, len, av, off, gs, cs, nc, top);
    }
}

// Rows list[0, n), or as many as *count says.
template <int WARPS, int NNZ>
__global__ void __launch_bounds__(32 * kAdjWarps) k_adjoint_rows(AdjArgs a, const int32_t *__restrict__ list, int32_t n,
                                                                 const uint32_t *__restrict__ count) {
    constexpr int ROWS = kAdjWarps / WARPS;
    __shared__ double gs[ROWS][NNZ];
    __shared__ int32_t cs[ROWS][NNZ];
    const int r = WARPS == 1 ? threadIdx.x >> 5 : 0;
    if (count) n = (int32_t)min((int64_t)n, (int64_t)*count);
    for (int64_t i = (int64_t)blockIdx.x * ROWS + r; i < n; i += (int64_t)gridDim.x * ROWS) {
        const int32_t row = list[i];
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        const int64_t c0 = a.Cp[row], nc = a.Cp[row + 1] - c0;
        if (nc > NNZ) {  // not the list's row
            if ((threadIdx.x & (32 * WARPS - 1)) == 0) raise(a.err, DEV_COUNT_MISMATCH);
            continue;
        }
        adjoint_row<WARPS>(a, e0, e1, c0, (int)nc, gs[r], cs[r]);
        if constexpr (WARPS == 1) __syncwarp();
        else __syncthreads();
    }
}

// First product of the first staged entry that starts at product t or later
// (the batch's products if none does; pre as stage_entries leaves it).
__device__ __forceinline__ int32_t first_entry_at(const int32_t *pre, int nb, int32_t t) {
    if (nb == 0) return 0;
    const int e = find_entry(pre, nb, t);
    return pre[e] < t ? pre[e + 1] : pre[e];
}

// Rows of more entries: persistent CTAs take rows from a counter, from the
// heaviest bin on.  The row's entries are staged with their B rows' lengths
// and the warps take equal contiguous shares of its products (a warp a row,
// the form before, walked a power-law hub's half a million products alone:
// 3.65 ms on R-MAT 2^14).  Loads, shuffles and barriers set the pace, not the
// FP64 pipe (42%) or L1 (27%): small CTAs, five an SM, and no row alone at
// the end.  With the products kept, 2^14 takes 0.21 ms and 2^16 1.13; 0.30
// and 1.68 with 512 threads, two CTAs an SM and whole rows, 0.26 and 1.37
// with three, 0.33 with 256 threads and whole rows.
// A row of C within kRankWordsMax 32-column words is ranked through a bitmap
// and the words' first positions in shared memory, two shared loads and a bit
// count a lookup; a wider one by binary search.  Four steps of B loads, then
// their four loads of G, are in flight together.
// dA of an entry is summed by the lanes it falls on, in registers while the
// warp stays on it, and stored by the warp it starts in; the parts of an
// entry that warps further on hold are added by one thread, in warp order
// (a fixed order either way).
//
// Rows of at least 2 a.partP products are cut into items (built by
// k_adjoint_split, and taken first): item p of k takes the entries of every
// staged batch whose first products lie in the p-th of k equal shares of it,
// so an entry's sum stays within a CTA.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, kAdjCtaPerSm) k_adjoint_cta(AdjArgs a, int32_t lo, int32_t n, int maxWords) {
    extern __shared__ __align__(16) unsigned char smem[];
    using L = StageLayout<THREADS>;
    constexpr int NW = THREADS / 32;
    __shared__ int32_t sh[NW];
    __shared__ int32_t partEnt[NW];
    __shared__ double partSum[NW];
    __shared__ int32_t next;
    int32_t *pre = reinterpret_cast<int32_t *>(smem + L::pre);
    int32_t *bst = reinterpret_cast<int32_t *>(smem + L::bst);
    double *av = reinterpret_cast<double *>(smem + L::av);
    int32_t *src = reinterpret_cast<int32_t *>(smem + L::bytes);
    uint32_t *bits = reinterpret_cast<uint32_t *>(src + THREADS);
    int32_t *wpre = reinterpret_cast<int32_t *>(bits + maxWords);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int32_t parts = a.items ? (int32_t)min((int64_t)a.ctr[ADJ_PARTS], a.itemCap) : 0;
    if (a.items) n = (int32_t)a.ctr[ADJ_CTA];
    for (;;) {
        if (tid == 0) next = (int32_t)atomicAdd(a.ctr, 1u);
        __syncthreads();
        const int32_t item = next;
        if (item >= parts + n) break;
        AdjItem it{0, 0, 1};
        if (item < parts) it = a.items[item];
        else it.row = a.items ? a.rows[ADJ_CTA][item - parts] : a.order[lo + n - 1 - item];
        const int32_t row = it.row;
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        const int64_t c0 = a.Cp[row], c1 = a.Cp[row + 1];
        const int32_t w0 = c1 > c0 ? a.Ci[c0] >> 5 : 0;
        const int words = c1 > c0 ? max(0, (a.Ci[c1 - 1] >> 5) - w0 + 1) : 0;
        const bool ranked = words <= maxWords;
        if (ranked) {
            for (int i = tid; i < words; i += THREADS) bits[i] = 0u;
            __syncthreads();
            for (int64_t i = c0 + tid; i < c1; i += THREADS) {
                const int32_t c = __ldg(&a.Ci[i]);
                const int32_t before = i > c0 ? __ldg(&a.Ci[i - 1]) : -1;
                const int w = (c >> 5) - w0;
                if ((uint32_t)w >= (uint32_t)words) {  // C's columns do not ascend
                    raise(a.err, DEV_COUNT_MISMATCH);
                    continue;
                }
                atomicOr(&bits[w], 1u << (c & 31));
                if (before < 0 || (before >> 5) != (c >> 5)) wpre[w] = (int32_t)(i - c0);
            }
        }
        // Position of column c in C's row, or -1.
        auto find = [&](int32_t c) -> int64_t {
            if (ranked) {
                const uint32_t w = (uint32_t)((c >> 5) - w0);
                if (w >= (uint32_t)words) return -1;
                const uint32_t word = bits[w], bit = 1u << (c & 31);
                return word & bit ? c0 + wpre[w] + __popc(word & (bit - 1u)) : -1;
            }
            const int64_t q = find_col(a.Ci, c0, c1, c);
            return q < c1 ? q : -1;
        };
        for (int32_t eb = e0; eb < e1; eb += THREADS) {
            int nb;
            const int32_t total = stage_entries<THREADS, true>(a.A, a.B, eb, min(THREADS, e1 - eb), pre, bst, av, &nb,
                                                               sh, false, 0, 0, nullptr, false, src);
            int32_t tb, te;
            if (it.k == 1) {
                warp_share<THREADS>(total, &tb, &te);
            } else {
                const int32_t from = first_entry_at(pre, nb, (int32_t)((int64_t)total * it.p / it.k));
                const int32_t to = first_entry_at(pre, nb, (int32_t)((int64_t)total * (it.p + 1) / it.k));
                warp_share<THREADS>(to - from, &tb, &te);
                tb += from;
                te += from;
            }
            if (lane == 0) partEnt[warp] = -1;
            // The batch's products follow each other in the kept array.
            double *keep = nullptr;
            if (a.prod) {
                const int64_t o = a.off[eb];
                if (o + total <= a.prodCap) keep = a.prod + o;
                else raise(a.err, DEV_COUNT_MISMATCH);  // the patterns are not the forward's
            }
            if (tb < te) {
                RangeWalk walk(pre, bst, nb, tb);
                int cur = walk.e0;              // the entry being summed, in acc over the lanes
                bool later = pre[cur] < tb;     // it starts in an earlier warp
                double acc = 0.0;
                auto flush = [&]() {
                    double s = acc;
#pragma unroll
                    for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(FULL, s, d);
                    if (lane == 0) {
                        if (later) {
                            partEnt[warp] = src[cur];
                            partSum[warp] = s;
                        } else {
                            a.dA[src[cur]] = s;
                        }
                    }
                    later = false;
                };
                constexpr int U = 4;
                for (int32_t g0 = tb; g0 < te; g0 += 32 * U) {
                    int32_t pos[U], col[U];
                    int ent[U];
                    bool val[U];
                    double bv[U], gv[U];
                    walk.template place<U>(pre, bst, nb, g0, te, pos, ent, val);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        col[u] = val[u] ? __ldg(&a.B.idx[pos[u]]) : 0;
                        bv[u] = val[u] ? __ldg(&a.B.val[pos[u]]) : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int64_t q = val[u] ? find(col[u]) : -1;
                        if (val[u] && q < 0) raise(a.err, DEV_COUNT_MISMATCH);
                        gv[u] = q >= 0 ? __ldg(&a.G[q]) : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (val[u] && (a.dB || keep)) {
                            const double x = __dmul_rn(av[ent[u]], gv[u]);
                            if (a.dB) atomicAdd(&a.dB[pos[u]], x);
                            else keep[g0 + 32 * u + lane] = x;
                        }
                        const int e = ent[u];
                        if (val[u] && e == cur) acc = __fma_rn(gv[u], bv[u], acc);
                        const unsigned other = __ballot_sync(FULL, val[u] && e != cur);
                        if (other == 0u) continue;
                        flush();
                        // The valid lanes lead the step and their entries do not
                        // decrease: the last one's entry is summed next, entries
                        // between it and cur lie within this step.
                        const int last = __shfl_sync(FULL, e, 31 - __clz(other));
                        const bool mid = val[u] && e != cur && e != last;
                        if (__any_sync(FULL, mid)) {
                            const int key = mid ? e : -1 - lane;
                            double p = mid ? __dmul_rn(gv[u], bv[u]) : 0.0;
#pragma unroll
                            for (int d = 1; d < 32; d <<= 1) {
                                const int ok = __shfl_down_sync(FULL, key, d);
                                const double op = __shfl_down_sync(FULL, p, d);
                                if (lane + d < 32 && ok == key) p += op;
                            }
                            const int pk = __shfl_up_sync(FULL, key, 1);
                            if (mid && (lane == 0 || pk != key)) a.dA[src[e]] = p;
                        }
                        acc = val[u] && e == last ? __dmul_rn(gv[u], bv[u]) : 0.0;
                        cur = last;
                    }
                }
                flush();
            }
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < NW; ++w)
                    if (partEnt[w] >= 0) a.dA[partEnt[w]] += partSum[w];
            }
            __syncthreads();
        }
        __syncthreads();  // every thread has read `next` before it changes
    }
}

// Tells the rows order[lo, lo + n) apart, the last ones first, a warp a row:
// the parts of those that are cut, and which of the others a CTA, four warps or a
// warp take.
__global__ void __launch_bounds__(256) k_adjoint_split(AdjArgs a, int32_t lo, int32_t n) {
    __shared__ int kinds[8];
    __shared__ uint32_t first[ADJ_COUNTERS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i = (int64_t)blockIdx.x * 8 + w;
    const int32_t row = i < n ? a.order[lo + n - 1 - i] : -1;
    int kind = 0;
    int64_t P = 0;
    if (row >= 0) {
        P = a.rowP[row];
        const int64_t nc = a.Cp[row + 1] - a.Cp[row];
        const int32_t e0 = a.A.ptr[row], e1 = a.A.ptr[row + 1];
        kind = P >= 2 * a.partP ? ADJ_PARTS : ADJ_CTA;
        if (a.rows[ADJ_WARP] && nc <= kAdjWideNnz && e1 - e0 <= 4096) {
            // Steps of the row by one warp, and the longest of them.
            int steps = 0, longest = 0;
            for (int32_t e = e0; e < e1; e += 32) {
                int32_t len = 0;
                if (e + lane < e1) {
                    const int32_t k = __ldg(&a.A.idx[e + lane]);
                    len = __ldg(&a.B.ptr[k + 1]) - __ldg(&a.B.ptr[k]);
                }
                const int L = adjoint_lanes(__reduce_add_sync(FULL, min(len, 1024)), min(32, e1 - e)), per = 32 / L;
                for (int d = 1; d < per; d <<= 1) len = max(len, __shfl_xor_sync(FULL, len, d));
                const int x = (len + 2 * L - 1) / (2 * L);
                if (lane % per == 0) steps += x;
                longest = max(longest, x);
            }
            steps = __reduce_add_sync(FULL, steps);
            longest = __reduce_max_sync(FULL, longest);
            const int batches = (e1 - e0 + kAdjCtaThreads - 1) / kAdjCtaThreads;
            if (steps <= kAdjBase * batches + P / kAdjPer) {
                if (nc <= kAdjWarpNnz && steps <= kAdjWarpSteps) kind = ADJ_WARP;
                else if (max(steps / kAdjWarps, longest) <= kAdjQuadSteps)
                    kind = nc <= kAdjQuadNnz ? ADJ_QUAD : ADJ_WIDE;
            }
        }
    }
    if (lane == 0) kinds[w] = kind;
    __syncthreads();
    if (threadIdx.x < ADJ_COUNTERS) {
        uint32_t k = 0;
        for (int r = 0; r < 8; ++r) k += kinds[r] == (int)threadIdx.x;
        if (threadIdx.x >= ADJ_CTA && k) first[threadIdx.x] = atomicAdd(&a.ctr[threadIdx.x], k);
    }
    __syncthreads();
    if (lane != 0 || kind == 0) return;
    if (kind != ADJ_PARTS) {
        uint32_t at = first[kind];
        for (int r = 0; r < w; ++r) at += kinds[r] == kind;
        a.rows[kind][at] = row;
        return;
    }
    const int k = (int)min((int64_t)kAdjMaxParts, P / a.partP);
    const uint32_t at = atomicAdd(&a.ctr[ADJ_PARTS], (uint32_t)k);
    if ((int64_t)at + k > a.itemCap) raise(a.err, DEV_COUNT_MISMATCH);  // the products are not the forward's
    for (int p = 0; p < k && (int64_t)at + p < a.itemCap; ++p) a.items[at + p] = AdjItem{row, (int16_t)p, (int16_t)k};
}

// Products of every A entry (the length of its B row).
__global__ void __launch_bounds__(256) k_entry_products(CsrDev A, const int32_t *__restrict__ Bp,
                                                        int32_t *__restrict__ len) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < A.nnz; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = A.idx[e];
        len[e] = Bp[k + 1] - Bp[k];
    }
}

// Each A entry's row, and (column, entry) pairs to sort: one warp per row.
__global__ void __launch_bounds__(256) k_entry_rows(CsrDev A, int32_t *rowOf, uint32_t *keys, uint32_t *vals) {
    const int lane = threadIdx.x & 31;
    const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= A.m) return;
    for (int32_t e = A.ptr[r] + lane; e < A.ptr[r + 1]; e += 32) {
        rowOf[e] = (int32_t)r;
        keys[e] = (uint32_t)A.idx[e];
        vals[e] = (uint32_t)e;
    }
}

// Column pointers from the entries sorted by column: column c starts at the
// first entry whose column is >= c.
__global__ void __launch_bounds__(256) k_col_ptr(const uint32_t *__restrict__ cols, int64_t n, int64_t ncols,
                                                 int32_t *__restrict__ colPtr) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t lo = i == 0 ? 0 : (int64_t)cols[i - 1] + 1;
        const int64_t hi = i == n ? ncols : (int64_t)cols[i];
        for (int64_t c = lo; c <= hi; ++c) colPtr[c] = (int32_t)i;
    }
}

// dB = mask_B(A^T G) as its own pass over B's pattern.  Entry (k, j) of B
// sums A(i,k) * G(i,j) down column k of A in row order, each G(i,j) found by
// binary search of C's sorted row i.  The column is cut into segments of
// kAdjSeg entries: one thread per entry of B sums the first segment into
// dB and records how many segments follow; after a scan of those counts,
// k_adjoint_db_tail sums every further segment, one thread each, and
// k_adjoint_db_sum adds them to dB in segment order.  Every sum has a fixed
// order, so dB is identical run to run, and a long column of A (a
// power-law hub) no longer sets the pass's length: no thread sums more
// than kAdjSeg products.
constexpr int kAdjSeg = 32;

// Row of B holding entry f: the k with ptr[k] <= f < ptr[k + 1].
__device__ __forceinline__ int64_t b_row_of(const CsrDev &B, int64_t f) {
    int64_t lo = 0, hi = B.m;
    while (hi - lo > 1) {
        const int64_t mid = lo + ((hi - lo) >> 1);
        if ((int64_t)B.ptr[mid] <= f) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Sum of A(i,k) * G(i,j) over the entries [p, pe) of A's column grouping, in
// order, for entry f = (k,j) of B, the at-th of its row.  With the dA pass's
// products kept (a.prod, entry e's from off[e] on in B's row order) a term is
// one load, next to its neighbours' for the threads of the same row; without,
// a binary search of C's row i, a chain of about 16 dependent loads.  R-MAT
// 2^14 (16.8M products): 126 + 365 us in the two passes that call it with
// the search, 16 + 74 us with the products.
__device__ __forceinline__ double column_sum(const AdjDbArgs &a, int32_t p, int32_t pe, int32_t j, int64_t at) {
    double acc = 0.0;
    if (a.prod) {
        constexpr int U = 8;
        for (; p < pe; p += U) {
            int64_t q[U];
            double x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) q[u] = p + u < pe ? (int64_t)__ldg(&a.perm[p + u]) : -1;
#pragma unroll
            for (int u = 0; u < U; ++u) q[u] = q[u] >= 0 ? __ldg(&a.off[q[u]]) : -1;
#pragma unroll
            for (int u = 0; u < U; ++u) x[u] = q[u] >= 0 && q[u] + at < a.prodCap ? __ldg(&a.prod[q[u] + at]) : 0.0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + u < pe) acc += x[u];
        }
        return acc;
    }
    for (; p < pe; ++p) {
        const uint32_t e = a.perm[p];
        const int32_t i = a.rowOf[e];
        const int64_t c0 = a.Cp[i], c1 = a.Cp[i + 1];
        const int64_t q = find_col(a.Ci, c0, c1, j);
        if (q < c1) acc += __dmul_rn(a.Aval[e], a.G[q]);
        else raise(a.err, DEV_COUNT_MISMATCH);
    }
    return acc;
}

__global__ void __launch_bounds__(256) k_adjoint_db(AdjDbArgs a) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.B.nnz) return;
    const int64_t k = b_row_of(a.B, f);
    const int32_t p0 = a.colPtr[k], p1 = a.colPtr[k + 1];
    const int32_t len = p1 - p0;
    a.dB[f] = column_sum(a, p0, len > kAdjSeg ? p0 + kAdjSeg : p1, a.B.idx[f], f - a.B.ptr[k]);
    a.extra[f] = len > kAdjSeg ? (len - 1) / kAdjSeg : 0;
}

// Segments 1.. of every entry, one thread each (grid-stride over the total,
// which is read on the device), each into its own slot of part.
__global__ void __launch_bounds__(256) k_adjoint_db_tail(AdjDbArgs a) {
    const int64_t total = a.xStart[a.B.nnz];
    if (total > a.partCap) {  // the patterns are not the forward's
        if (blockIdx.x == 0 && threadIdx.x == 0) raise(a.err, DEV_COUNT_MISMATCH);
        return;
    }
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
         g += (int64_t)gridDim.x * blockDim.x) {
        // f: the entry with xStart[f] <= g < xStart[f + 1].
        int64_t lo = 0, hi = a.B.nnz;
        while (hi - lo > 1) {
            const int64_t mid = lo + ((hi - lo) >> 1);
            if (a.xStart[mid] <= g) lo = mid;
            else hi = mid;
        }
        const int64_t f = lo;
        const int64_t k = b_row_of(a.B, f);
        const int32_t p1 = a.colPtr[k + 1];
        const int64_t pb = (int64_t)a.colPtr[k] + (1 + (g - a.xStart[f])) * kAdjSeg;
        a.part[g] = column_sum(a, (int32_t)pb, (int32_t)min((int64_t)p1, pb + kAdjSeg), a.B.idx[f], f - a.B.ptr[k]);
    }
}

__global__ void __launch_bounds__(256) k_adjoint_db_sum(AdjDbArgs a) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.B.nnz || a.xStart[a.B.nnz] > a.partCap) return;
    const int64_t x0 = a.xStart[f], x1 = a.xStart[f + 1];
    if (x1 == x0) return;
    double acc = a.dB[f];
    for (int64_t g = x0; g < x1; ++g) acc += a.part[g];
    a.dB[f] = acc;
}


}  // namespace

void launch_adjoint_transpose(const CsrDev &A, int32_t *rowOf, uint32_t *keys0, uint32_t *vals0, uint32_t *keys1,
                              uint32_t *vals1, void *scratch, int32_t *colPtr, const uint32_t **perm, cudaStream_t s) {
    if (A.m > 0) k_entry_rows<<<(unsigned)ceil_div(A.m, 8), 256, 0, s>>>(A, rowOf, keys0, vals0);
    int bits = 0;
    while (bits < 32 && ((uint64_t)std::max<int64_t>(A.n - 1, 0) >> bits) != 0) ++bits;
    uint32_t *ks = keys0, *vs = vals0;
    launch_stable_sort_u32(keys0, vals0, keys1, vals1, A.nnz, bits, scratch, s, &ks, &vs);
    const int64_t grid = std::min<int64_t>(ceil_div(A.nnz + 1, 256), 65535);
    k_col_ptr<<<(unsigned)std::max<int64_t>(grid, 1), 256, 0, s>>>(ks, A.nnz, A.n, colPtr);
    *perm = vs;
}

void launch_entry_products(const CsrDev &A, const CsrDev &B, int32_t *len, int64_t *scanPart, int64_t *off,
                           cudaStream_t s) {
    if (A.nnz > 0)
        k_entry_products<<<(unsigned)std::min<int64_t>(ceil_div(A.nnz, 256), 65535), 256, 0, s>>>(A, B.ptr, len);
    launch_row_scan(A.nnz, len, scanPart, off, s);
}

int64_t adjoint_db_part_cap(int64_t products) { return products / kAdjSeg + 1; }

void launch_adjoint_db(const AdjDbArgs &a, int64_t *scanPart, int num_sms, cudaStream_t s) {
    if (a.B.nnz <= 0) return;
    const unsigned grid = (unsigned)ceil_div(a.B.nnz, 256);
    k_adjoint_db<<<grid, 256, 0, s>>>(a);
    launch_row_scan(a.B.nnz, a.extra, scanPart, a.xStart, s);
    k_adjoint_db_tail<<<(unsigned)std::max(num_sms, 1) * 8, 256, 0, s>>>(a);
    k_adjoint_db_sum<<<grid, 256, 0, s>>>(a);
}

// Dynamic shared memory of the CTA kernel for bitmaps of `words` words.
static size_t smem_adjoint_cta(int words) {
    return StageLayout<kAdjCtaThreads>::bytes + 4 * (size_t)kAdjCtaThreads + 8 * (size_t)words;
}

void launch_adjoint_warp(const AdjArgs &a, int32_t lo, int32_t hi, cudaStream_t s, int *launches) {
    if (hi <= lo) return;
    k_adjoint_rows<1, kAdjWarpNnz><<<(unsigned)ceil_div(hi - lo, kAdjWarps), 32 * kAdjWarps, 0, s>>>(a, a.order + lo,
                                                                                                   hi - lo, nullptr);
    ++*launches;
}

void launch_adjoint_rows(const AdjArgs &a, int kind, int32_t n, int num_sms, cudaStream_t s, int *launches) {
    // At most 64 CTAs an SM: a short list of many candidates costs little.
    const int rows = kind == ADJ_WARP ? kAdjWarps : 1;
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(n, rows), (int64_t)std::max(num_sms, 1) * 64);
    const auto fn = kind == ADJ_WARP   ? k_adjoint_rows<1, kAdjWarpNnz>
                    : kind == ADJ_QUAD ? k_adjoint_rows<kAdjWarps, kAdjQuadNnz>
                                       : k_adjoint_rows<kAdjWarps, kAdjWideNnz>;
    fn<<<grid, 32 * kAdjWarps, 0, s>>>(a, a.rows[kind], n, a.ctr + kind);
    ++*launches;
}

void launch_adjoint_split(const AdjArgs &a, int32_t lo, int32_t hi, cudaStream_t s, int *launches) {
    if (hi <= lo) return;
    cudaMemsetAsync(a.ctr, 0, ADJ_COUNTERS * sizeof(uint32_t), s);
    if (a.items) {
        k_adjoint_split<<<(unsigned)ceil_div(hi - lo, 8), 256, 0, s>>>(a, lo, hi - lo);
        ++*launches;
    }
}

void launch_adjoint_cta(const AdjArgs &a, int32_t lo, int32_t hi, int num_sms, cudaStream_t s, int *launches) {
    if (hi <= lo) return;
    // A matrix of few columns needs no more bitmap than they take.
    const int words = (int)std::min<int64_t>(kRankWordsMax, a.B.n / 32 + 2);
    const size_t smem = smem_adjoint_cta(words);
    const int per_sm = std::max(1, std::min(kAdjCtaPerSm, (int)((227 * 1024) / (smem + 1024))));
    const int64_t most = (int64_t)(hi - lo) * (a.items ? kAdjMaxParts : 1);
    const int grid = (int)std::min<int64_t>(most, (int64_t)std::max(num_sms, 1) * per_sm);
    k_adjoint_cta<kAdjCtaThreads><<<(unsigned)grid, kAdjCtaThreads, smem, s>>>(a, lo, hi - lo, words);
    ++*launches;
}

void init_adjoint_attributes() {
    cudaFuncSetAttribute(k_adjoint_cta<kAdjCtaThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_adjoint_cta(kRankWordsMax));
}

}  // namespace dbd
