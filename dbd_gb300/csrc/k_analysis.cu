// k_analysis.cu -- work estimate, row categorisation, per-bin row lists and
// the int64 row_ptr scan.
//
// Replaces calculate_UpperBound + get_UpperBound
// (dbd/for_small_datasets/src/preProc.cu:142-179): the reference launches one
// 32-thread CTA per row with a global atomicAdd per A entry, copies the
// counts to the host, scans them sequentially there and copies them back.
// Here eight lanes share a row and reduce with shuffles (no atomics), the
// counts are int64 (the reference's int32 wraps past 2^31 products), and all
// scans stay on the device.
#include "dbd_internal.h"

#include <algorithm>

namespace dbd {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Everything a multiply asks of an operand before it reads through it, in one
// pass: *badPtr <- 1 unless ptr[0] == 0, ptr[m] == nnz and ptr never
// decreases; *badIdx <- 1 if a column lies outside [0, n); the first and last
// column of every row as one pair (INT32_MAX and -1 when empty), which are its
// smallest and largest where the row ascends; and *unsorted += the number of
// entries not above their predecessor in the same row (0: every row ascends).
// badPtr and badIdx may be null.
//
// Bound by the reads of idx and ptr.  Entries are walked flat, so neither
// five-entry rows (a warp each would leave 27 lanes idle) nor power-law hubs
// (one warp walking half a million entries) set its time: the entries below
// their predecessor are counted over the whole array, and the row loop takes
// those at row starts off again, where they are no fault.  It stands for a
// row pointer check, a column check and a warp-per-row minimum and maximum,
// with a host round trip after each.  33M entries in 2^21 power-law rows:
// 1082 us in three launches before, 41 us now (20 us at copy rate); a multiply
// of 2.1M five-point rows takes 251 us less.
// (A row_ptr that fails its check is never read through: no entry is touched
// unless ptr[m] is nnz, which is what says that there are so many, and a row's
// only when both its bounds lie in [0, nnz].)
__global__ void __launch_bounds__(256) k_check_operand(CsrDev M, int2 *__restrict__ range, int *__restrict__ badPtr,
                                                       int *__restrict__ badIdx, int *__restrict__ unsorted) {
    __shared__ int red[8];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nnz = M.ptr[M.m] == M.nnz ? M.nnz : 0;
    int down = 0;
    bool badI = false, badP = false;
    auto entry = [&](int32_t c, int32_t before, bool first) {
        badI |= c < 0 || c >= M.n;
        if (!first && c <= before) ++down;
    };
    // 16 bytes a load from the first aligned entry on, two loads a thread in
    // flight; an entry's predecessor comes from the same load or the lane
    // below, only a warp's first lane loads one.
    const int lane = threadIdx.x & 31;
    const int64_t head = min(nnz, (int64_t)((16 - (reinterpret_cast<uintptr_t>(M.idx) & 15)) & 15) >> 2);
    const int64_t quads = (nnz - head) >> 2;
    const int4 *q4 = reinterpret_cast<const int4 *>(M.idx + head);
    for (int64_t b = t0 - lane; b < quads; b += 2 * stride) {
        int4 c[2];
        int32_t first[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t i = b + u * stride + lane;
            c[u] = i < quads ? __ldg(&q4[i]) : make_int4(0, 0, 0, 0);
            first[u] = lane == 0 && i < quads && head + i > 0 ? M.idx[head + 4 * i - 1] : -1;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t i = b + u * stride + lane;
            const int32_t up = __shfl_up_sync(FULL, c[u].w, 1);
            if (i < quads) {
                entry(c[u].x, lane ? up : first[u], head + i == 0);
                entry(c[u].y, c[u].x, false);
                entry(c[u].z, c[u].y, false);
                entry(c[u].w, c[u].z, false);
            }
        }
    }
    // The unaligned entries before and the remainder behind.
    if (t0 < 8) {
        const int64_t i = t0 < 4 ? t0 : head + 4 * quads + (t0 - 4);
        if (t0 < 4 ? i < head : i < nnz) entry(M.idx[i], i > 0 ? M.idx[i - 1] : -1, i == 0);
    }
    // Four rows a thread in flight.
    for (int64_t b = t0; b <= M.m; b += 4 * stride) {
        int32_t v[4], w[4], lo[4], hi[4], before[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t r = b + u * stride;
            v[u] = r <= M.m ? __ldg(&M.ptr[r]) : 0;
            w[u] = r < M.m ? __ldg(&M.ptr[r + 1]) : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t r = b + u * stride;
            const bool has = r < M.m && v[u] >= 0 && v[u] < w[u] && w[u] <= nnz;
            lo[u] = has ? __ldg(&M.idx[v[u]]) : INT32_MAX;
            hi[u] = has ? __ldg(&M.idx[w[u] - 1]) : -1;
            before[u] = has && v[u] > 0 ? __ldg(&M.idx[v[u] - 1]) : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t r = b + u * stride;
            if (r > M.m) continue;
            badP |= v[u] < 0 || v[u] > M.nnz || (r == 0 && v[u] != 0);
            if (r == M.m) {
                badP |= v[u] != M.nnz;
            } else {
                badP |= w[u] < v[u];
                if (lo[u] <= before[u]) --down;
                range[r] = make_int2(lo[u], hi[u]);
            }
        }
    }
    if (badP && badPtr) atomicExch(badPtr, 1);
    if (badI && badIdx) atomicExch(badIdx, 1);
#pragma unroll
    for (int d = 16; d; d >>= 1) down += __shfl_xor_sync(FULL, down, d);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = down;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) down += red[w];
        if (down) atomicAdd(unsorted, down);
    }
}

// Smallest and largest column of every row of an operand that
// k_check_operand found unsorted (one warp per row); nothing otherwise.  It is
// enqueued before the host has read the checks' results, so an operand whose
// row_ptr failed (*badPtr, where given) is left alone, and no row is read
// outside [0, nnz) whatever its pointers say.
__global__ void k_row_minmax(CsrDev B, int2 *__restrict__ range, const int *__restrict__ badPtr,
                             const int *__restrict__ unsorted) {
    if (*unsorted == 0 || (badPtr && *badPtr != 0)) return;
    const int lane = threadIdx.x & 31;
    int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t stride = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (; row < B.m; row += stride) {
        int32_t lo = INT32_MAX, hi = -1;
        const int32_t s = B.ptr[row], e = B.ptr[row + 1];
        if (s < 0 || e > B.nnz) continue;  // the whole warp
        for (int64_t i = (int64_t)s + lane; i < e; i += 32) {
            const int32_t c = B.idx[i];
            lo = min(lo, c);
            hi = max(hi, c);
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) {
            lo = min(lo, __shfl_xor_sync(FULL, lo, d));
            hi = max(hi, __shfl_xor_sync(FULL, hi, d));
        }
        if (lane == 0) range[row] = make_int2(lo, hi);
    }
}

// Products per row, P_r = sum over k in A_r of |B_k|, and the row's column
// window [lo, hi] from the B rows' first and last columns.  Eight lanes per
// row; rows of more than kLongRow entries (power-law hubs, whose serial walk
// by eight lanes would set the kernel's duration) are left to a second
// stage in which a whole CTA takes each of them.
//
// Where the rows are short (at most kShortMean entries on average) a lane
// takes a row: up to kShortRow entries with all their loads in flight, the
// warp's longer rows four at a time by eight lanes each, and the second stage
// starts at kLongRowShort.  2.1M five-entry rows 105 -> 36 us.  Its longest
// warps are those of a power-law graph's hubs, so it takes kShortRows rows
// and more: means of 2 to 5 entries over 2^20 rows 78 -> 56 us, 2^19 52 ->
// 39, but 2^18 32 -> 37, 2^16 14 -> 21, 2^12 10 -> 14.  The mean's line is on the
// safe side: on rows of Poisson lengths lanes gain up to a mean of 10 (the whole
// work estimate of 2^21 rows, mean 5 217 -> 177 us, 8 278 -> 239, 12 335 -> 331),
// on R-MAT 2^20 up to 12 (6 165 -> 153, 8 176 -> 169, 12 210 -> 202).
constexpr int kLongRow = 256, kLongRowShort = 64;
constexpr int kShortRow = 8;
constexpr int64_t kShortMean = 6, kShortRows = 1 << 19;

__device__ __forceinline__ void row_products_out(const CsrDev &A, int64_t row, int64_t sum, int32_t lo, int32_t hi,
                                                 RowInfo &ri, uint8_t *symBin, int *err, const Tuning &tune) {
    const int32_t n = A.ptr[row + 1] - A.ptr[row];
    ri.rowP[row] = sum;
    ri.lo[row] = lo;
    ri.hi[row] = hi;
    symBin[row] = sym_bin_of(sum, n, span_words(lo, hi), tune);
    if (sum > 0x7fffffffLL) atomicCAS(err, 0, (int)DEV_ROW_TOO_LONG);
}

template <int THREADS, bool SHORT>
__global__ void __launch_bounds__(THREADS) k_row_products(CsrDev A, const int32_t *__restrict__ Bp,
                                                          const int2 *__restrict__ range, RowInfo ri,
                                                          uint8_t *__restrict__ symBin, int *err,
                                                          const int32_t *__restrict__ ctl, Tuning tune) {
    if (ctl && (ctl[CTL_A] | ctl[CTL_A + 1] | ctl[CTL_B] | ctl[CTL_B + 1] | ctl[CTL_PAIR])) {
        for (int64_t r = blockIdx.x * (int64_t)THREADS + threadIdx.x; r < A.m; r += (int64_t)gridDim.x * THREADS) {
            ri.rowP[r] = 0;
            ri.lo[r] = INT32_MAX;
            ri.hi[r] = -1;
            symBin[r] = SB_EMPTY;
        }
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane & 7;
    constexpr int kLong = SHORT ? kLongRowShort : kLongRow;
    const unsigned gmask = 0xffu << (lane & 24);
    if constexpr (SHORT) {
        for (int64_t b = blockIdx.x * (int64_t)THREADS + (tid & ~31); b < A.m; b += (int64_t)gridDim.x * THREADS) {
            const int64_t row = b + lane;
            const int32_t s = row < A.m ? __ldg(&A.ptr[row]) : 0;
            const int32_t e = row < A.m ? __ldg(&A.ptr[row + 1]) : 0;
            int32_t k[kShortRow], len[kShortRow];
            int2 r[kShortRow];
            const bool brief = e - s <= kShortRow;
#pragma unroll
            for (int i = 0; i < kShortRow; ++i) k[i] = brief && s + i < e ? __ldg(&A.idx[s + i]) : -1;
#pragma unroll
            for (int i = 0; i < kShortRow; ++i) {
                r[i] = k[i] >= 0 ? __ldg(&range[k[i]]) : make_int2(INT32_MAX, -1);
                len[i] = k[i] >= 0 ? __ldg(&Bp[k[i] + 1]) - __ldg(&Bp[k[i]]) : 0;
            }
            int64_t sum = 0;
            int32_t lo = INT32_MAX, hi = -1;
#pragma unroll
            for (int i = 0; i < kShortRow; ++i) {
                sum += len[i];
                lo = min(lo, r[i].x);
                hi = max(hi, r[i].y);
            }
            if (row < A.m && brief) row_products_out(A, row, sum, lo, hi, ri, symBin, err, tune);
            // The others up to kLong: four at a time, eight lanes each.
            unsigned more = __ballot_sync(FULL, !brief && e - s <= kLong);
            while (more) {
                int mine = -1;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (more && g == lane >> 3) mine = __ffs(more) - 1;
                    more &= more - 1u;
                }
                const int32_t s8 = __shfl_sync(FULL, s, max(mine, 0)), e8 = __shfl_sync(FULL, e, max(mine, 0));
                sum = 0;
                lo = INT32_MAX;
                hi = -1;
                if (mine >= 0) {
#pragma unroll 4
                    for (int32_t i = s8 + sub; i < e8; i += 8) {
                        const int32_t q = __ldg(&A.idx[i]);
                        const int2 w = __ldg(&range[q]);
                        sum += (int64_t)(__ldg(&Bp[q + 1]) - __ldg(&Bp[q]));
                        lo = min(lo, w.x);
                        hi = max(hi, w.y);
                    }
                }
#pragma unroll
                for (int d = 4; d; d >>= 1) {
                    sum += __shfl_xor_sync(FULL, sum, d);
                    lo = min(lo, __shfl_xor_sync(FULL, lo, d));
                    hi = max(hi, __shfl_xor_sync(FULL, hi, d));
                }
                if (sub == 0 && mine >= 0) row_products_out(A, b + mine, sum, lo, hi, ri, symBin, err, tune);
            }
        }
    } else {
        const int64_t stride = ((int64_t)gridDim.x * THREADS) >> 3;
        // kRowsAhead rows a group in flight: a row is a chain of three dependent
        // loads, which one row at a time leaves the GPU waiting for (2.1M
        // five-entry rows: 155 -> 105 us, with the ranges read as pairs).
        constexpr int kRowsAhead = 4;
        for (int64_t b = (blockIdx.x * (int64_t)THREADS + tid) >> 3; b < A.m; b += kRowsAhead * stride) {
            int32_t s[kRowsAhead], e[kRowsAhead], k[kRowsAhead];
#pragma unroll
            for (int u = 0; u < kRowsAhead; ++u) {
                const int64_t row = b + u * stride;
                s[u] = row < A.m ? __ldg(&A.ptr[row]) : 0;
                e[u] = row < A.m ? __ldg(&A.ptr[row + 1]) : 0;
            }
#pragma unroll
            for (int u = 0; u < kRowsAhead; ++u) k[u] = s[u] + sub < e[u] ? __ldg(&A.idx[s[u] + sub]) : -1;
            int64_t sum[kRowsAhead];
            int32_t lo[kRowsAhead], hi[kRowsAhead];
#pragma unroll
            for (int u = 0; u < kRowsAhead; ++u) {
                const int2 r = k[u] >= 0 ? __ldg(&range[k[u]]) : make_int2(INT32_MAX, -1);
                sum[u] = k[u] >= 0 ? __ldg(&Bp[k[u] + 1]) - __ldg(&Bp[k[u]]) : 0;
                lo[u] = r.x;
                hi[u] = r.y;
            }
#pragma unroll
            for (int u = 0; u < kRowsAhead; ++u) {
                const int64_t row = b + u * stride;
                if (row >= A.m || e[u] - s[u] > kLong) continue;  // the whole group skips together
                for (int32_t i = s[u] + 8 + sub; i < e[u]; i += 8) {
                    const int32_t q = A.idx[i];
                    const int2 r = __ldg(&range[q]);
                    sum[u] += (int64_t)(Bp[q + 1] - Bp[q]);
                    lo[u] = min(lo[u], r.x);
                    hi[u] = max(hi[u], r.y);
                }
#pragma unroll
                for (int d = 4; d; d >>= 1) {
                    sum[u] += __shfl_xor_sync(gmask, sum[u], d, 8);
                    lo[u] = min(lo[u], __shfl_xor_sync(gmask, lo[u], d, 8));
                    hi[u] = max(hi[u], __shfl_xor_sync(gmask, hi[u], d, 8));
                }
                if (sub == 0) row_products_out(A, row, sum[u], lo[u], hi[u], ri, symBin, err, tune);
            }
        }
    }

    // Long rows: CTA b takes the long rows r with r = b (mod gridDim.x), one
    // by one with all its threads.  Hubs sit close together in row order
    // (power-law generators put them at small indices, and at multiples of
    // powers of two), so the modular assignment, by an odd number of CTAs,
    // spreads them over the CTAs.
    __shared__ int32_t longRows[THREADS];
    __shared__ int nLong;
    __shared__ int64_t rs[THREADS / 32];
    __shared__ int32_t rlo[THREADS / 32], rhi[THREADS / 32];
    for (int64_t t0 = 0; t0 < A.m; t0 += (int64_t)gridDim.x * THREADS) {
        if (tid == 0) nLong = 0;
        __syncthreads();
        const int64_t row = t0 + blockIdx.x + (int64_t)gridDim.x * tid;
        if (row < A.m && A.ptr[row + 1] - A.ptr[row] > kLong) longRows[atomicAdd(&nLong, 1)] = (int32_t)row;
        __syncthreads();
        const int nl = nLong;
        for (int j = 0; j < nl; ++j) {
            const int32_t r = longRows[j];
            const int32_t s = A.ptr[r], e = A.ptr[r + 1];
            int64_t sum = 0;
            int32_t lo = INT32_MAX, hi = -1;
            for (int32_t i = s + tid; i < e; i += THREADS) {
                const int32_t k = A.idx[i];
                const int2 kr = __ldg(&range[k]);
                sum += (int64_t)(Bp[k + 1] - Bp[k]);
                lo = min(lo, kr.x);
                hi = max(hi, kr.y);
            }
#pragma unroll
            for (int d = 16; d; d >>= 1) {
                sum += __shfl_xor_sync(FULL, sum, d);
                lo = min(lo, __shfl_xor_sync(FULL, lo, d));
                hi = max(hi, __shfl_xor_sync(FULL, hi, d));
            }
            if (lane == 0) {
                rs[warp] = sum;
                rlo[warp] = lo;
                rhi[warp] = hi;
            }
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < THREADS / 32; ++w) {
                    sum += rs[w];
                    lo = min(lo, rlo[w]);
                    hi = max(hi, rhi[w]);
                }
                row_products_out(A, r, sum, lo, hi, ri, symBin, err, tune);
            }
            __syncthreads();
        }
    }
}

// ---- per-bin row lists ----
//
// Rows are grouped by bin, row order kept, in three launches over tiles of
// kTileRows rows: k_tiles counts every bin's rows per tile (hist[bin][tile])
// and sums a per-row quantity per tile, k_tile_scan turns the counts into
// absolute offsets, k_tile_scatter writes the lists.  The same three launches
// carry what else is needed of the rows on either side of the symbolic pass:
// before it the sums are the rows' products, from which the scan's last CTA
// makes the row blocks' products; after it k_tiles also picks the numeric
// bins, the sums are the rows' entries, which the scan's last CTA scans, and
// the scatter writes C's row pointers.  (Before: five launches ahead of the
// symbolic kernels' and seven behind them, and one CTA scanning all bins one
// after another: all of them 130 and 210 us on 2.1M rows, 40 and 53 us now; on 65k
// rows 14 and 25 us, 7 and 8 us now.)

// What the tiles carry beside the lists: nothing, the products (rowP) of the
// row blocks, or the entries (rowNnz) and numeric bins of the rows.
enum TileMode : int { TILES_PLAIN = 0, TILES_BLOCKS, TILES_NUMERIC };

__global__ void __launch_bounds__(kTileRows) k_tiles(int64_t m, int64_t ntiles, TileMode mode,
                                                     uint8_t *__restrict__ bin, int nbins,
                                                     const int32_t *__restrict__ Ap, RowInfo ri,
                                                     int32_t *__restrict__ rowNnz, Tuning tune,
                                                     int32_t *__restrict__ hist, int64_t *__restrict__ tileSum,
                                                     uint32_t *__restrict__ maxP) {
    __shared__ int32_t wc[kTileRows / 32][kMaxBins];
    __shared__ int64_t ws[kTileRows / 32];
    const int64_t r = (int64_t)blockIdx.x * kTileRows + threadIdx.x;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int b = -1;
    int64_t x = 0;
    if (r < m) {
        if (mode == TILES_NUMERIC) {
            const int32_t nnz = rowNnz[r];
            b = num_bin_of(ri.rowP[r], Ap[r + 1] - Ap[r], nnz, span_words(ri.lo[r], ri.hi[r]), tune);
            bin[r] = (uint8_t)b;
            x = nnz;
        } else {
            b = bin[r];
            if (b == SB_EMPTY) rowNnz[r] = 0;  // no symbolic kernel takes it
            if (mode == TILES_BLOCKS) x = ri.rowP[r];
        }
    }
    for (int q = 0; q < nbins; ++q) {
        const unsigned mk = __ballot_sync(FULL, b == q);
        if (lane == 0) wc[w][q] = __popc(mk);
    }
    if (maxP) {
        // The largest row's products; below 2^31, as the work estimate checks.
        const uint32_t most = __reduce_max_sync(FULL, (uint32_t)min(x, (int64_t)INT32_MAX));
        if (lane == 0 && most > *(volatile uint32_t *)maxP) atomicMax(maxP, most);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) x += __shfl_xor_sync(FULL, x, d);
    if (lane == 0) ws[w] = x;
    __syncthreads();
    if (threadIdx.x < nbins) {
        int32_t s = 0;
        for (int i = 0; i < kTileRows / 32; ++i) s += wc[i][threadIdx.x];
        hist[threadIdx.x * ntiles + blockIdx.x] = s;
    } else if (threadIdx.x == 32 && tileSum) {
        int64_t s = 0;
        for (int i = 0; i < kTileRows / 32; ++i) s += ws[i];
        tileSum[blockIdx.x] = s;
    }
}

constexpr int kScanThreads = 1024;

// Block-wide exclusive scan of one value per thread (blockDim.x ==
// kScanThreads).
template <class T>
__device__ __forceinline__ T block_excl_scan_wide(T v, T *total, T *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = __shfl_up_sync(FULL, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        T t = sh[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T y = __shfl_up_sync(FULL, t, d);
            if (lane >= d) t += y;
        }
        sh[lane] = t;  // inclusive warp totals
    }
    __syncthreads();
    const T base = w ? sh[w - 1] : T(0);
    *total = sh[kScanThreads / 32 - 1];
    __syncthreads();
    return base + x - v;
}

// CTA q < kMaxBins: bin q's start (the rows of all bins below it, from their
// tile counts) and its tiles' absolute offsets, four tiles a thread.  CTA
// kMaxBins: the row blocks' products, or the tiles' entry offsets and C's
// size.
__global__ void __launch_bounds__(kScanThreads) k_tile_scan(int64_t ntiles, TileMode mode, int nbins,
                                                            const int32_t *__restrict__ hist,
                                                            int32_t *__restrict__ tileOff,
                                                            int32_t *__restrict__ binStart,
                                                            int64_t *__restrict__ tileSum, int64_t tilesPerBlock,
                                                            int64_t *__restrict__ out) {
    const int tid = threadIdx.x, q = blockIdx.x;
    if (q < kMaxBins) {
        __shared__ int32_t sh[kScanThreads / 32];
        int32_t below = 0, start;
        const int64_t n = (int64_t)min(q, nbins) * ntiles;
#pragma unroll 8
        for (int64_t i = tid; i < n; i += kScanThreads) below += hist[i];
        block_excl_scan_wide<int32_t>(below, &start, sh);
        int32_t carry = start;
        for (int64_t t0 = 0; t0 < ntiles; t0 += 4 * kScanThreads) {
            const int64_t t = t0 + 4 * tid;
            int32_t v[4];
            int32_t s = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u] = q < nbins && t + u < ntiles ? hist[q * ntiles + t + u] : 0;
                s += v[u];
            }
            int32_t tot;
            int32_t at = carry + block_excl_scan_wide<int32_t>(s, &tot, sh);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (t + u < ntiles) tileOff[(t + u) * kMaxBins + q] = at;
                at += v[u];
            }
            carry += tot;
        }
        if (tid == 0) {
            tileOff[ntiles * kMaxBins + q] = carry;
            binStart[q] = start;
            if (q == kMaxBins - 1) binStart[kMaxBins] = carry;
        }
    } else if (mode == TILES_BLOCKS) {
        // block_Info of divide_Blocks (ZIP:dbd/src/main.cpp:276-296), a warp a block.
        const int64_t blocks = (ntiles + tilesPerBlock - 1) / tilesPerBlock;
        for (int64_t k = tid >> 5; k < blocks; k += kScanThreads / 32) {
            int64_t s = 0;
            for (int64_t t = k * tilesPerBlock + (tid & 31); t < min(ntiles, (k + 1) * tilesPerBlock); t += 32)
                s += tileSum[t];
#pragma unroll
            for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(FULL, s, d);
            if ((tid & 31) == 0) out[k] = s;
        }
    } else if (mode == TILES_NUMERIC) {
        __shared__ int64_t sh[kScanThreads / 32];
        int64_t carry = 0;
        for (int64_t t0 = 0; t0 < ntiles; t0 += 4 * kScanThreads) {
            const int64_t t = t0 + 4 * tid;
            int64_t v[4], s = 0, tot;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u] = t + u < ntiles ? tileSum[t + u] : 0;
                s += v[u];
            }
            int64_t at = carry + block_excl_scan_wide<int64_t>(s, &tot, sh);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (t + u < ntiles) tileSum[t + u] = at;
                at += v[u];
            }
            carry += tot;
        }
        if (tid == 0) *out = carry;
    }
}

// Stable scatter of row ids into their bin's list; with Cp also C's row
// pointers (Cp[m] is the scan's).  The first CTA leaves what the host decides
// the next launches by in its mailbox: pageable copies of the same words cost
// a pass 12 us each.
__global__ void __launch_bounds__(kTileRows) k_tile_scatter(int64_t m, const uint8_t *__restrict__ bin, int nbins,
                                                            const int32_t *__restrict__ tileOff,
                                                            int32_t *__restrict__ list,
                                                            const int32_t *__restrict__ rowNnz,
                                                            const int64_t *__restrict__ tileSum,
                                                            int64_t *__restrict__ Cp, Mail mail) {
    __shared__ int32_t wc[kTileRows / 32][kMaxBins];
    __shared__ int64_t ws[kTileRows / 32];
    const int64_t r = (int64_t)blockIdx.x * kTileRows + threadIdx.x;
    if (mail.to && blockIdx.x == 0) {
        const int t = threadIdx.x;
        if (t < 8) mail.to->flags[t] = mail.ctl[t];
        else if (t < 8 + kMaxBins + 1) mail.to->binStart[t - 8] = mail.binStart[t - 8];
        else if (t == 32) mail.to->err = mail.ctl[CTL_ERR];
        else if (t == 33) mail.to->heavy = mail.ctl[CTL_CTR + CTR_HEAVY];
        else if (t == 35) mail.to->maxP = mail.ctl[CTL_CTR + CTR_MAX_P];
        else if (t == 34 && mail.nnz) mail.to->nnz = *mail.nnz;
    }
    const int b = r < m ? (int)bin[r] : -1;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int rank = 0;
    for (int q = 0; q < nbins; ++q) {
        const unsigned mk = __ballot_sync(FULL, b == q);
        if (b == q) rank = __popc(mk & ((1u << lane) - 1u));
        if (lane == 0) wc[w][q] = __popc(mk);
    }
    const int64_t x = Cp && r < m ? rowNnz[r] : 0;
    int64_t incl = x;
    if (Cp) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t y = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += y;
        }
        if (lane == 31) ws[w] = incl;
    }
    __syncthreads();
    if (b >= 0) {
        int32_t pos = tileOff[(int64_t)blockIdx.x * kMaxBins + b] + rank;
        for (int i = 0; i < w; ++i) pos += wc[i][b];
        list[pos] = (int32_t)r;
    }
    if (Cp && r < m) {
        int64_t at = tileSum[blockIdx.x] + incl - x;
        for (int i = 0; i < w; ++i) at += ws[i];
        Cp[r] = at;
    }
}

// ---- int32 row counts -> int64 exclusive scan (row_ptr of C) ----

__device__ __forceinline__ int64_t block_excl_scan_i64(int64_t v, int64_t *total, int64_t *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int64_t x = v;
    for (int d = 1; d < 32; d <<= 1) {
        const int64_t y = __shfl_up_sync(FULL, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t t = lane < nw ? sh[lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t y = __shfl_up_sync(FULL, t, d);
            if (lane >= d) t += y;
        }
        sh[lane] = t;
    }
    __syncthreads();
    const int64_t base = w ? sh[w - 1] : 0;
    *total = sh[nw - 1];
    __syncthreads();
    return base + x - v;
}

__global__ void k_scan_reduce(int64_t m, const int32_t *__restrict__ cnt, int64_t *__restrict__ part) {
    __shared__ int64_t sh[32];
    const int64_t r0 = (int64_t)blockIdx.x * kScanTile;
    int64_t s = 0;
    for (int i = threadIdx.x; i < kScanTile; i += blockDim.x) {
        const int64_t r = r0 + i;
        if (r < m) s += cnt[r];
    }
    int64_t tot;
    block_excl_scan_i64(s, &tot, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}

__global__ void k_scan_parts(int64_t nparts, int64_t *__restrict__ part) {
    __shared__ int64_t sh[32];
    int64_t carry = 0;
    for (int64_t i0 = 0; i0 < nparts; i0 += blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        const int64_t v = i < nparts ? part[i] : 0;
        int64_t tot;
        const int64_t ex = block_excl_scan_i64(v, &tot, sh);
        if (i < nparts) part[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) part[nparts] = carry;
}

// blockDim.x == kScanTile / 4: four consecutive rows per thread.
__global__ void k_scan_final(int64_t m, const int32_t *__restrict__ cnt,
                             const int64_t *__restrict__ part, int64_t nparts,
                             int64_t *__restrict__ Cp) {
    __shared__ int64_t sh[32];
    const int64_t r0 = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * 4;
    int32_t c[4];
    int64_t s = 0;
    for (int j = 0; j < 4; ++j) {
        c[j] = (r0 + j < m) ? cnt[r0 + j] : 0;
        s += c[j];
    }
    int64_t tot;
    int64_t run = part[blockIdx.x] + block_excl_scan_i64(s, &tot, sh);
    for (int j = 0; j < 4; ++j) {
        if (r0 + j < m) Cp[r0 + j] = run;
        run += c[j];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) Cp[m] = part[nparts];
}

// Widens float32 values (a view with val_fp32) into the FP64 operand copy;
// nothing is read where the operand's row_ptr failed its check.
__global__ void k_f32_to_f64(const float *__restrict__ src, double *__restrict__ dst, int64_t n,
                             const int *__restrict__ badPtr) {
    if (*badPtr != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

}  // namespace

void launch_check_operand(const CsrDev &M, int2 *range, int *badPtr, int *badIdx, int *unsorted, cudaStream_t s,
                          int num_sms) {
    const int64_t work = std::max<int64_t>(M.m + 1, M.nnz);
    const int grid = (int)std::min<int64_t>(ceil_div(work, 256), (int64_t)num_sms * 8);
    k_check_operand<<<grid, 256, 0, s>>>(M, range, badPtr, badIdx, unsorted);
}

void launch_row_minmax(const CsrDev &B, int2 *range, const int *badPtr, const int *unsorted, cudaStream_t s,
                       int num_sms) {
    if (B.m == 0) return;
    const int grid = (int)std::min<int64_t>(ceil_div(B.m * 32, 256), (int64_t)num_sms * 8);
    k_row_minmax<<<grid, 256, 0, s>>>(B, range, badPtr, unsorted);
}

void launch_row_products(const CsrDev &A, const int32_t *Bp, const int2 *range, const RowInfo &ri, uint8_t *symBin,
                         int *err, const int32_t *ctl, const Tuning &t, cudaStream_t s, int num_sms) {
    if (A.m == 0) return;
    constexpr int threads = 256;
    const int64_t fit = (int64_t)num_sms * 8;
    // Odd, for the long rows (262k rows of R-MAT 2^18, 5 entries on average: 58 -> 32 us).
    const auto grid = [&](int64_t need) {
        return (int)(need < fit ? need | 1 : (fit - 1) | 1);
    };
    if (A.m >= kShortRows && A.nnz <= kShortMean * A.m) {
        k_row_products<threads, true><<<grid(ceil_div(A.m, threads)), threads, 0, s>>>(
            A, Bp, range, ri, symBin, err, ctl, t);
    } else {
        k_row_products<threads, false><<<grid(ceil_div(A.m * 8, threads)), threads, 0, s>>>(
            A, Bp, range, ri, symBin, err, ctl, t);
    }
}

void launch_sym_lists(int64_t m, const Binning &b, const RowInfo &ri, int32_t *rowNnz, int64_t *tileSum,
                      int64_t rows_per_block, int64_t *blockP, uint32_t *maxP, const Mail &mail, cudaStream_t s) {
    const int64_t nt = tile_count(m);
    const TileMode mode = blockP ? TILES_BLOCKS : TILES_PLAIN;
    if (nt > 0)
        k_tiles<<<(unsigned)nt, kTileRows, 0, s>>>(m, nt, mode, b.bin, SB_COUNT, nullptr, ri, rowNnz, Tuning{}, b.hist,
                                                   blockP ? tileSum : nullptr, blockP ? maxP : nullptr);
    k_tile_scan<<<kMaxBins + 1, kScanThreads, 0, s>>>(nt, mode, SB_COUNT, b.hist, b.tileOff, b.binStart, tileSum,
                                                      std::max<int64_t>(rows_per_block / kTileRows, 1), blockP);
    if (nt > 0 || mail.to)
        k_tile_scatter<<<(unsigned)std::max<int64_t>(nt, 1), kTileRows, 0, s>>>(m, b.bin, SB_COUNT, b.tileOff, b.list,
                                                                               nullptr, nullptr, nullptr, mail);
}

void launch_num_lists(int64_t m, const Binning &b, const RowInfo &ri, const int32_t *Ap, const int32_t *rowNnz,
                      const Tuning &t, int64_t *tileSum, int64_t *Cp, const Mail &mail, cudaStream_t s) {
    const int64_t nt = tile_count(m);
    if (nt > 0)
        k_tiles<<<(unsigned)nt, kTileRows, 0, s>>>(m, nt, TILES_NUMERIC, b.bin, NB_COUNT, Ap, ri,
                                                   const_cast<int32_t *>(rowNnz), t, b.hist, tileSum, nullptr);
    k_tile_scan<<<kMaxBins + 1, kScanThreads, 0, s>>>(nt, TILES_NUMERIC, NB_COUNT, b.hist, b.tileOff, b.binStart,
                                                      tileSum, 1, Cp + m);
    if (nt > 0 || mail.to)
        k_tile_scatter<<<(unsigned)std::max<int64_t>(nt, 1), kTileRows, 0, s>>>(m, b.bin, NB_COUNT, b.tileOff, b.list,
                                                                               rowNnz, tileSum, Cp, mail);
}

void launch_row_scan(int64_t m, const int32_t *rowNnz, int64_t *part, int64_t *Cp, cudaStream_t s) {
    const int64_t nparts = ceil_div(m, kScanTile);
    if (nparts > 0) k_scan_reduce<<<(unsigned)nparts, 1024, 0, s>>>(m, rowNnz, part);
    k_scan_parts<<<1, 1024, 0, s>>>(nparts, part);
    if (nparts > 0) {
        k_scan_final<<<(unsigned)nparts, kScanTile / 4, 0, s>>>(m, rowNnz, part, nparts, Cp);
    } else {
        cudaMemsetAsync(Cp, 0, sizeof(int64_t), s);
    }
}

void launch_f32_to_f64(const float *src, double *dst, int64_t n, const int *badPtr, cudaStream_t s) {
    if (n <= 0) return;
    k_f32_to_f64<<<(unsigned)std::min<int64_t>(ceil_div(n, 256), 4096), 256, 0, s>>>(src, dst, n, badPtr);
}

// Loads every kernel of this file now (CUDA loads kernels lazily, on first
// launch, by default).  Returns the first error.
cudaError_t preload_analysis_kernels() {
    const void *fns[] = {
        (const void *)k_check_operand, (const void *)k_row_minmax,
        (const void *)k_row_products<256, true>, (const void *)k_row_products<256, false>,
        (const void *)k_tiles, (const void *)k_tile_scan, (const void *)k_tile_scatter,
        (const void *)k_scan_reduce, (const void *)k_scan_parts, (const void *)k_scan_final,
        (const void *)k_f32_to_f64,
    };
    for (const void *f : fns) {
        cudaFuncAttributes fa;
        const cudaError_t e = cudaFuncGetAttributes(&fa, f);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace dbd
