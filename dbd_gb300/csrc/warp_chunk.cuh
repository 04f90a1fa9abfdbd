// Device helpers shared by the multiply and adjoint kernels: the error word
// and the warp-level enumeration of the products of up to 32 consecutive A
// entries (product t, 0 <= t < total, comes from the lane whose inclusive
// length prefix first exceeds t).
#pragma once

#include "dbd_internal.h"

namespace dbd {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// First error wins: a device check records its code once and never traps.
__device__ __forceinline__ void raise(int *err, int code) { atomicCAS(err, 0, code); }

struct Chunk {
    int32_t bs;    // first position of B_k in B.idx
    int32_t len;   // |B_k|
    int32_t incl;  // inclusive prefix of len over lanes
    double a;      // A value of this lane's entry
    int32_t total; // products of the chunk
    bool lead;     // the lanes with products come first
};

__device__ __forceinline__ Chunk load_chunk(const CsrDev &A, const CsrDev &B, int32_t e, int32_t eEnd,
                                            int lane) {
    Chunk c;
    c.bs = 0;
    c.len = 0;
    c.a = 0.0;
    if (e + lane < eEnd) {
        const int32_t k = A.idx[e + lane];
        c.bs = B.ptr[k];
        c.len = B.ptr[k + 1] - c.bs;
        c.a = A.val[e + lane];
    }
    int32_t x = c.len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int32_t y = __shfl_up_sync(FULL, x, d);
        if (lane >= d) x += y;
    }
    c.incl = x;
    c.total = __shfl_sync(FULL, x, 31);
    const unsigned have = __ballot_sync(FULL, c.len > 0);
    c.lead = (have & (have + 1u)) == 0u;
    return c;
}

// Owner lane of this lane's product t = t0 + lane (all 32 lanes must call, t0
// the same on all; t may be out of range).  Where the lanes with products
// come first it is the number of their first products up to t, less one: those
// before the step by a vote, those inside it from a mask of them; otherwise a
// search over the lanes (555k symbolic warp rows of a batch 502 -> 468
// us against the search alone and three shuffles to the position).
__device__ __forceinline__ int chunk_owner(const Chunk &c, int32_t t) {
    if (c.lead) {
        const int lane = threadIdx.x & 31;
        const int32_t at = c.incl - c.len - (t - lane);
        const unsigned before = __ballot_sync(FULL, c.len > 0 && at < 0);
        const uint32_t in = __reduce_or_sync(FULL, c.len > 0 && at >= 0 && at < 32 ? 1u << at : 0u);
        return max(__popc(before) + __popc(in & (FULL >> (31 - lane))) - 1, 0);
    }
    int lo = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const int32_t v = __shfl_sync(FULL, c.incl, lo + step - 1);
        if (v <= t) lo += step;
    }
    return lo;
}

}  // namespace
}  // namespace dbd
