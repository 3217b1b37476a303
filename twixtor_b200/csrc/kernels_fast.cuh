// The fast mode's variants of the solver kernels: fused.cu, solver.cu and coarse.cu compiled a second
// time with TW_FAST_VARIANT (FMA contraction, approximate division and square root, denormals
// flushed to zero). Same signatures as the strict kernels in kernels.cuh; namespace tw::fast.
#pragma once
#include "kernels.cuh"

namespace tw {
namespace fast {

__global__ void k_range_any(const float2* __restrict__ f, int w, int h, int* __restrict__ any_in_range);
__global__ void k_bm_rows(const float* __restrict__ A, const float* __restrict__ B, const float2* __restrict__ f, int w,
                          int h, float2* __restrict__ ft, float z);
__global__ void k_bm_cols(const float* __restrict__ AT, const float* __restrict__ BT, const float2* __restrict__ ft, int w,
                          int h, float2* f, float z, int* any);
__global__ void k_transpose2(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ at,
                             float* __restrict__ bt, int w, int h);
__global__ void k_pyramid_step_16(const __grid_constant__ PyramidStep P);
__global__ void k_pyramid_step_32(const __grid_constant__ PyramidStep P);
__global__ void k_pyramid_tail(const __grid_constant__ PyramidTail P);
__global__ void k_level_init_16x16(const __grid_constant__ LevelInitArgs P);
__global__ void k_level_init_32x32(const __grid_constant__ LevelInitArgs P);
__global__ void k_level_iter_16x16(const __grid_constant__ LevelIterArgs P);
__global__ void k_level_iter_32x32(const __grid_constant__ LevelIterArgs P);
__global__ void k_level_iter_32x64(const __grid_constant__ LevelIterArgs P);
__global__ void k_level_iter_64x32(const __grid_constant__ LevelIterArgs P);
__global__ void k_level_iter_64x64(const __grid_constant__ LevelIterArgs P);
__global__ void k_calc_b_pitched(const float* __restrict__ i1, const float* __restrict__ i0,
                                 const float2* __restrict__ grad, const float2* __restrict__ f, int w, int h,
                                 const float* __restrict__ mask_y, float2* __restrict__ b_out, int bp);
__global__ void k_apply_upsample(const float2* __restrict__ src, int sw, int sh, UpsampleScale up,
                                 const int* __restrict__ any, int l, int start, bool damp_now, float damp,
                                 float2* __restrict__ dst, int dw, int dh);
__global__ void k_apply_negate(const float2* __restrict__ f, long n, const int* __restrict__ any, int start,
                               bool damp_now, float damp, float2* __restrict__ out, int* __restrict__ nan_flag);
__global__ void k_solve_coarse(const __grid_constant__ CoarseJob job);

}  // namespace fast
}  // namespace tw
