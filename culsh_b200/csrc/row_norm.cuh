// Mean L2 norm of the rows of a matrix, from which a p-stable fit takes its default window
// (pstable_lsh.py:191-223), in one launch and one wait.  At the few thousand rows it looks at nothing but
// launches and waits counts: as a conversion to float64, a norm, a mean and a read of the result it
// takes three launches and two temporaries.  A warp takes a whole row, so that a few rows of very many columns
// leave the chip idle; the caller in pstable_lsh.py says which rows come here, with both sides' times.
#pragma once

#include "common.cuh"
#include "index_math.h"

namespace culsh_b200 {

constexpr int RN_THREADS = 256;
constexpr int RN_MAX_BLOCKS = 592;  // four CTAs an SM
constexpr int RN_LOADS = 8;          // of a lane in flight

// A warp per row, sums in float64.  The last CTA to finish adds up the partial sums, in one order, so that
// the result does not depend on which one that is, and leaves the mean in page-locked host memory, and the ticket zero, as it was
// before.  (A word to clear before the kernel and a copy behind it took longer than the kernel: 1,000 x 100, the call 25.3 us, 17.2 now.)
template <typename T>
__global__ void __launch_bounds__(RN_THREADS)
mean_row_norm_kernel(const T* __restrict__ X, int n, int d, double* __restrict__ partial, unsigned* __restrict__ ticket,
                     double* mean) {
    __shared__ double s_sum[RN_THREADS / 32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int WARPS = RN_THREADS / 32;
    double sum = 0.0;
    walk_rows(blockIdx.x * WARPS + warp, gridDim.x * WARPS, n, [&](int row) {
        const T* x = X + (size_t)row * d;
        double s = 0.0;
        auto add = [&](int64_t i, bool whole) {
            T v[RN_LOADS];
#pragma unroll
            for (int j = 0; j < RN_LOADS; ++j) v[j] = whole || i + 32 * j < d ? x[i + 32 * j] : T(0);
#pragma unroll
            for (int j = 0; j < RN_LOADS; ++j) s = fma((double)v[j], (double)v[j], s);
        };
        int64_t i = lane;
        for (; i + 32 * (RN_LOADS - 1) < d; i += 32 * RN_LOADS) add(i, true);
        if (i < d) add(i, false);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        sum += sqrt(s);
    });
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < WARPS; ++w) s += s_sum[w];
        partial[blockIdx.x] = s;
        __threadfence();
        s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last && warp == 0) {
        __threadfence();
        double s = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(partial + b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        if (lane == 0) *mean = s / n;
    }
}

template <typename T>
inline double mean_row_norm(const CtxPtr& c, const T* X, int n, int d) {
    const int blocks = (int)std::min<size_t>(ceil_div(n, RN_THREADS / 32), RN_MAX_BLOCKS);
    Scratch<double> partial(c, SL_MISC2, RN_MAX_BLOCKS);
    double* const mean = reinterpret_cast<double*>(c->pinned + HS_NORM);
    mean_row_norm_kernel<T><<<blocks, RN_THREADS, 0, c->stream>>>(X, n, d, partial.p, c->d_ticket, mean);
    KERNEL_CHECK();
    CU_CHECK(cudaStreamSynchronize(c->stream));
    return *mean;
}

}  // namespace culsh_b200
