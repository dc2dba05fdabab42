// The end of an FP8 GEMM whose output rows are finished one warp at a time (decode kernel, 128-row pair kernel).
#pragma once

#include "sm100.cuh"

namespace llmmm {

// One finished row of one 128-column output group, four columns per lane of one warp: fp32 as it is, or the
// row's absmax (the bit pattern of a non-negative float orders like the float: one warp-wide integer max), the
// two divisions of the quantisation rule, four e4m3 bytes per lane and the scale.
template<bool OUT_F32>
__device__ __forceinline__ void store_group_row(float4 s, int m, int nb, void* __restrict__ C_out, float* __restrict__ C_s,
                                                int M, int N, int lane)
{
  if constexpr (OUT_F32) {
    reinterpret_cast<float4*>(reinterpret_cast<float*>(C_out) + (size_t)m * N + (size_t)nb * 128)[lane] = s;
  }
  else {
    const float    mine = fmaxf(fmaxf(fabsf(s.x), fabsf(s.y)), fmaxf(fabsf(s.z), fabsf(s.w)));
    const float    amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mine)));
    const float    inv  = amax > 0.0f ? __fdiv_rn(448.0f, amax) : 0.0f;
    const uint32_t q    = pack_e4m3x4(s.x * inv, s.y * inv, s.z * inv, s.w * inv);
    reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(C_out) + (size_t)m * N + (size_t)nb * 128)[lane] = q;
    if (lane == 0) {
      C_s[(size_t)nb * M + m] = __fdiv_rn(amax, 448.0f);
    }
  }
}

// Several such rows of one warp at once: lane j does the two divisions of row j for everybody (one after the other
// they took half of the time).  Rows whose group is not below n_groups are left out.  The maximum starts from zero and
// passes NaN over, as in the kernels whose threads hold whole rows: the finite values of a group keep their scale and codes.
template<bool OUT_F32, int ROWS>
__device__ __forceinline__ void store_group_rows(const float4 (&s)[ROWS], const int (&m)[ROWS], const int (&nb)[ROWS], int n_groups,
                                                 void* __restrict__ C_out, float* __restrict__ C_s, int M, int N, int lane)
{
  if constexpr (OUT_F32) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (nb[j] < n_groups) {
        store_group_row<true>(s[j], m[j], nb[j], C_out, C_s, M, N, lane);
      }
    }
  }
  else {
    float amax  = 0.0f;
    int   row   = 0, group = n_groups;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const float mine = fmaxf(fmaxf(fmaxf(0.0f, fabsf(s[j].x)), fabsf(s[j].y)), fmaxf(fmaxf(0.0f, fabsf(s[j].z)), fabsf(s[j].w)));
      const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mine)));
      if (lane == j) {
        amax  = most;
        row   = m[j];
        group = nb[j];
      }
    }
    const float inv = amax > 0.0f ? __fdiv_rn(448.0f, amax) : 0.0f;
    if (group < n_groups) {
      C_s[(size_t)group * M + row] = __fdiv_rn(amax, 448.0f);
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const float f = __shfl_sync(0xffffffffu, inv, j);
      if (nb[j] < n_groups) {
        reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(C_out) + (size_t)m[j] * N + (size_t)nb[j] * 128)[lane] =
          pack_e4m3x4(s[j].x * f, s[j].y * f, s[j].z * f, s[j].w * f);
      }
    }
  }
}

}  // namespace llmmm
