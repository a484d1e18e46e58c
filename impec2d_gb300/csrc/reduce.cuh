// Deterministic block reductions: every block writes its partial, the last block to
// finish (ticket counter) folds the partials in a fixed order.  Reruns are bit-identical
// because the grid size and the per-thread assignment are fixed.
#pragma once
#include <cuda_runtime.h>

namespace impec {

constexpr int RED_THREADS = 256;

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Reduce K values across the block; the results are valid in thread 0.  maxmask bit k selects max.
// An FP64 instruction occupies a quarter of an SM for 64 cycles whether all lanes or some take part, so the
// instruction count on the busiest quarter is what matters.  One value: a shared-memory tree (128, 64,
// 32 pairs) and then one warp's shuffle tree, 8 in a row.  Several values: one warp each, on different
// quarters, 12 in a row (the tree for all of them: 8 K, most in one warp).
// Requires blockDim.x == RED_THREADS.
template <int K>
__device__ __forceinline__ void block_reduce(double (&v)[K], unsigned maxmask) {
    static_assert(K <= RED_THREADS / 32, "one warp per value");
    __shared__ double sh[K][RED_THREADS];
    const int t = threadIdx.x;
#pragma unroll
    for (int k = 0; k < K; ++k) sh[k][t] = v[k];
    __syncthreads();
    if (K == 1) {
#pragma unroll
        for (int s = RED_THREADS / 2; s >= 32; s >>= 1) {
            if (t < s) sh[0][t] = (maxmask & 1) ? fmax(sh[0][t], sh[0][t + s]) : sh[0][t] + sh[0][t + s];
            __syncthreads();
        }
        if (t < 32) v[0] = (maxmask & 1) ? warp_max(sh[0][t]) : warp_sum(sh[0][t]);
        return;
    }
    const int w = t / 32, lane = t & 31;
    if (w < K) {
        const bool mx = (maxmask >> w) & 1;
        double a = sh[w][lane];
#pragma unroll
        for (int s = 32; s < RED_THREADS; s += 32) a = mx ? fmax(a, sh[w][lane + s]) : a + sh[w][lane + s];
        a = mx ? warp_max(a) : warp_sum(a);
        if (lane == 0) sh[w][0] = a;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = sh[k][0];
}

// Blocks for a row-segment walk over an n1 x n2 grid: one block per segment of RED_THREADS
// cells of a row, at most max_blocks (larger grids loop).
static inline int seg_blocks(int n1, int n2, int max_blocks) {
    const long units = (long)n1 * ((n2 + RED_THREADS - 1) / RED_THREADS);
    return (int)(units < max_blocks ? units : max_blocks);
}

// Block limit for the reductions: four blocks per SM, so that each thread folds several cells
// before the FP64 warp sums (five additions per reduced value and thread) are paid.
static inline int red_cap(int num_sms, int max_blocks) { return num_sms * 4 < max_blocks ? num_sms * 4 : max_blocks; }

// Blocks for a flat walk over n values: one value per thread, at most max_blocks.
static inline int flat_blocks(size_t n, int max_blocks) {
    const size_t b = (n + RED_THREADS - 1) / RED_THREADS;
    return (int)(b < (size_t)max_blocks ? (b > 0 ? b : 1) : (size_t)max_blocks);
}

// Row-segment walk (grid of seg_blocks blocks of RED_THREADS): f(i, j, k) for every cell,
// k = i*n2 + j.  A block issues the loads of a whole segment at once and no thread divides
// per cell, which keeps the walk bandwidth- rather than latency-bound.
template <class F>
__device__ __forceinline__ void for_cells(int n1, int n2, F&& f) {
    const int segs = (n2 + RED_THREADS - 1) / RED_THREADS, units = n1 * segs;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int i = u / segs, j = (u - i * segs) * RED_THREADS + (int)threadIdx.x;
        if (j < n2) f(i, j, (size_t)i * n2 + j);
    }
}

// Grid-level reduction with last-block finalisation.  Requires blockDim.x == RED_THREADS,
// 1-D grid with gridDim.x <= max_blocks.  out[k] receives the reduced values.  Returns true in
// every thread of the last block (thread 0 of which wrote out[]).
template <int K>
__device__ bool grid_reduce(double (&v)[K], unsigned maxmask, double* partials, int max_blocks,
                            unsigned* counter, double* out) {
    __shared__ bool last;
    block_reduce<K>(v, maxmask);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) partials[k * max_blocks + blockIdx.x] = v[k];
        __threadfence();
        unsigned ticket = atomicAdd(counter, 1u);
        last = (ticket == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double w[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const bool mx = (maxmask >> k) & 1;
        double a = mx ? -INFINITY : 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
            double p = ((volatile double*)partials)[k * max_blocks + b];
            a = mx ? fmax(a, p) : a + p;
        }
        w[k] = a;
    }
    block_reduce<K>(w, maxmask);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) out[k] = w[k];
        *counter = 0u;
    }
    return true;
}

}  // namespace impec
