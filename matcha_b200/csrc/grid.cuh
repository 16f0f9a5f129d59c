// The SO(3) grid kernel for oversampling 2 (grid.cu), called by the search front end (search.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// The complex multiply-add steps re += x tx - y ty, im += x ty + y tx of both grid kernels' transforms,
// with the roundings written out: one product of each pair is fused, the sum is not.
__device__ __forceinline__ float re_mac(float a, float x, float y, float tx, float ty) {
  return __fadd_rn(a, __fmaf_rn(x, tx, -__fmul_rn(y, ty)));
}
__device__ __forceinline__ float im_mac(float a, float x, float y, float tx, float ty) {
  return __fadd_rn(a, __fmaf_rn(y, tx, __fmul_rn(x, ty)));
}

// Whether grid_columns_launch covers a grid: oversampling 2, 3 <= L0 <= 16.
bool grid_columns_cover(int L0, int K);

// Grid search of B subtomograms (n = 4 L0 points per axis) with the C <= 32 best points of each
// as angles, in order; grid (B, n, n, n) receives every value unless null.
int grid_columns_launch(const float2* sigma, int64_t stride, int B, const float* dtab, int L0, int C, float* alpha,
                        float* beta, float* gamma, float* grid, cudaStream_t st);
