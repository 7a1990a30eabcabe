// int8 weights as the projections see them (Int8Linear, jsgrad/models/llama3.ts:27-35).
#pragma once
#include "common.cuh"

#ifdef __CUDACC__
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
