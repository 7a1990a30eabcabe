// Quantised weights as the projections see them: int8 (Int8Linear, jsgrad/models/llama3.ts:27-35) and NF4 (NF4Linear, :79-117).
#pragma once
#include "common.cuh"

#ifdef __CUDACC__
// the 16 code values; rounded to fp16 before a block's scale meets them (jsgrad/models/llama3.ts:81)
static __constant__ float c_nf4[16] = {-1.0f, -0.6961928009986877f, -0.5250730514526367f, -0.39491748809814453f, -0.28444138169288635f, -0.18477343022823334f,
                                       -0.09105003625154495f, 0.0f, 0.07958029955625534f, 0.16093020141124725f, 0.24611230194568634f, 0.33791524171829224f,
                                       0.44070982933044434f, 0.5626170039176941f, 0.7229568362236023f, 1.0f};

// int8 x16 -> sixteen halves of half(q) * s (eight half2 registers in k order), each product rounded once.  Bytes become halves exactly
// through the exponent of 1024 (0x6400).
__device__ __forceinline__ void w8_to_half2(const uint4& raw, __half2 s2, uint32_t (&out)[8]) {
  const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
  const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);  // 1024 + 128
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t v = words[i] ^ 0x80808080u;          // signed -> offset-binary
    uint32_t lo = __byte_perm(v, 0x64646464u, 0x4140);  // bytes 0,1 -> halves 1024 + b
    uint32_t hi = __byte_perm(v, 0x64646464u, 0x4342);  // bytes 2,3
    const __half2 a = __hmul2_rn(__hsub2(*reinterpret_cast<__half2*>(&lo), bias), s2);
    const __half2 b = __hmul2_rn(__hsub2(*reinterpret_cast<__half2*>(&hi), bias), s2);
    out[2 * i] = *reinterpret_cast<const uint32_t*>(&a);
    out[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&b);
  }
}
#endif
