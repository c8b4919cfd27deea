// chol.cuh -- log det R from its Cholesky factor (Cholesky_logdet_lower_packed,
// pixelgrid.cpp:17201-17210; F's is k_final's), for the FP64 factor of the plain path and the
// FP32 one of the mixed path; the sum of logarithms is FP64 in both.
#pragma once
#include "qlpix_internal.h"

namespace qlpix {

template <typename T>
__global__ void __launch_bounds__(1024) k_logdet_t(const T* __restrict__ A, int ld, const GridState* __restrict__ gs,
                                                   EvalOut* out)
{
    __shared__ double red[32];
    const int M = gs->M;
    double acc = 0;
    for (int i = threadIdx.x; i < M; i += blockDim.x) acc += log(fabs((double)A[(size_t)i * ld + i]));
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += red[k];
        out->logdet_R = 2 * t;
    }
}

}  // namespace qlpix
