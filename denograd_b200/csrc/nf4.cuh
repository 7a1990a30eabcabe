// The 16 code values of NF4 weights (NF4Linear, jsgrad/models/llama3.ts:79-117); rounded to fp16 before a block's scale meets them (:81).
// Selected, not looked up: a module with a table in constant memory pays for it at each of its launches (gemm_tc.cu with one beside it:
// 0.2 to 0.7 us more, a step of 32 rows 3.57 -> 3.61 ms).
#pragma once
#include "common.cuh"

#ifdef __CUDACC__
__device__ __forceinline__ float nf4_code(int i) {
  float v = -1.0f;
  v = i == 1 ? -0.6961928009986877f : v;
  v = i == 2 ? -0.5250730514526367f : v;
  v = i == 3 ? -0.39491748809814453f : v;
  v = i == 4 ? -0.28444138169288635f : v;
  v = i == 5 ? -0.18477343022823334f : v;
  v = i == 6 ? -0.09105003625154495f : v;
  v = i == 7 ? 0.0f : v;
  v = i == 8 ? 0.07958029955625534f : v;
  v = i == 9 ? 0.16093020141124725f : v;
  v = i == 10 ? 0.24611230194568634f : v;
  v = i == 11 ? 0.33791524171829224f : v;
  v = i == 12 ? 0.44070982933044434f : v;
  v = i == 13 ? 0.5626170039176941f : v;
  v = i == 14 ? 0.7229568362236023f : v;
  return i == 15 ? 1.0f : v;
}
// The pair of codes of byte b (high nibble first), which all lanes of a warp ask for; lane_code = nf4_code(lane % 16).
__device__ __forceinline__ __half2 nf4_pair(float lane_code, int b) {
  return __halves2half2(__float2half_rn(__shfl_sync(0xffffffffu, lane_code, b >> 4)), __float2half_rn(__shfl_sync(0xffffffffu, lane_code, b & 15)));
}
#endif
