// Enough of CUDA's device language to run a kernel of k_analysis.cu on the
// host, one thread after another: for what a kernel reads and writes, not for
// what its lanes exchange (a shuffle gives a lane its own value, a vote its
// own answer).
#pragma once

#include <algorithm>
#include <climits>
#include <cstdint>

struct Dim {
    int x = 1;
};
static Dim threadIdx, blockIdx, blockDim, gridDim;
struct int2 {
    int x, y;
};
struct int4 {
    int x, y, z, w;
};
inline int2 make_int2(int x, int y) { return {x, y}; }
inline int4 make_int4(int x, int y, int z, int w) { return {x, y, z, w}; }

#define __global__ static
#define __shared__ static
#define __launch_bounds__(...)
#define __syncthreads()
using std::max;
using std::min;

template <class T> T __ldg(const T *p) { return *p; }
template <class T> T __shfl_up_sync(unsigned, T v, int) { return v; }
template <class T> T __shfl_xor_sync(unsigned, T v, int) { return v; }
inline int atomicAdd(int *p, int v) { return *p += v; }
inline int atomicOr(int *p, int v) { return *p |= v; }
inline int atomicExch(int *p, int v) {
    const int old = *p;
    *p = v;
    return old;
}

struct CsrDev {
    int64_t m = 0, n = 0, nnz = 0;
    const int32_t *ptr = nullptr;
    const int32_t *idx = nullptr;
    const double *val = nullptr;
};
constexpr unsigned FULL = 0xffffffffu;

template <class Kernel> void each_thread(int blocks, int threads, Kernel kernel) {
    gridDim.x = blocks;
    blockDim.x = threads;
    for (blockIdx.x = 0; blockIdx.x < blocks; ++blockIdx.x)
        for (threadIdx.x = 0; threadIdx.x < threads; ++threadIdx.x) kernel();
}
