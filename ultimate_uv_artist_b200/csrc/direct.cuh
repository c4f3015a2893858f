// Interface of the direct island solver (direct.cu) to the batch entry points
// (solve.cu).
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

constexpr int kDirectMaxN = 16384;   // vertices of an island (band positions fit 14 bits)
// counters in uva_batch.work beside the CG path's four
constexpr int kWorkNext = 4, kWorkLeft = 5, kWorkCg = 6;

// uva_batch.band: position of every solver row (n), first block column of
// every block row (n / 16 + nc), then 4 ints per island: a factor is possible
// (bit 0) and the coarse operators of CG are built (bit 1), blocks, widest
// row, solved by the last launch.
__host__ __device__ __forceinline__ int32_t* band_first(const uva_batch& b, int v0, int isl) {
    return b.band + b.n + v0 / 16 + isl;
}
__host__ __device__ __forceinline__ int32_t* band_info(const uva_batch& b, int isl) {
    return b.band + b.n + b.n / 16 + b.nc + 4 * static_cast<int64_t>(isl);
}

cudaError_t uva_direct_attributes();
int uva_direct_order(const uva_batch* b, cudaStream_t s);                       // after the set-up's rows and pins
int uva_direct_launch(const uva_batch* b, const uva_solve_params* prm, bool lscm, cudaStream_t s);
