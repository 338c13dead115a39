// int8 codes -> 16-bit floats, exact for all 256 codes, four at a time (one word -> two words of two
// values, in order).  Integer-to-float conversions run at a fraction of the rate of what is used here:
//   fp16: 0x6400 | u is the half 1024 + u with u = q + 128; subtract 1152.
//   bf16: 0x4300 | (q & 0x7F) is 128 + (q mod 128), and 0x4300 | (q & 0x80) is 128 for q >= 0 and
//         256 for q < 0: their difference is q.  Two permutes, four logic operations and two
//         packed subtractions (through fp32, 2^23 + u, it took six permutes and one more
//         instruction in all: the permutes and logic share the ALU pipe, which bounds the
//         decode kernels).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200q {
namespace {

template <typename T>
__device__ __forceinline__ uint2 expand4(uint32_t w);
template <>
__device__ __forceinline__ uint2 expand4<__half>(uint32_t w) {
  const uint32_t t = w ^ 0x80808080u;
  uint32_t lo = __byte_perm(t, 0x64646464u, 0x4140);
  uint32_t hi = __byte_perm(t, 0x64646464u, 0x4342);
  const __half2 bias = __floats2half2_rn(1152.f, 1152.f);
  const __half2 l = __hsub2(*reinterpret_cast<__half2*>(&lo), bias);
  const __half2 h = __hsub2(*reinterpret_cast<__half2*>(&hi), bias);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&l), *reinterpret_cast<const uint32_t*>(&h));
}
template <>
__device__ __forceinline__ uint2 expand4<__nv_bfloat16>(uint32_t w) {
  const uint32_t lo = __byte_perm(w, 0x43434343u, 0x4140), hi = __byte_perm(w, 0x43434343u, 0x4342);
  const uint32_t al = lo & 0xFF7FFF7Fu, bl = lo & 0xFF80FF80u;
  const uint32_t ah = hi & 0xFF7FFF7Fu, bh = hi & 0xFF80FF80u;
  const __nv_bfloat162 l = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&al),
                                   *reinterpret_cast<const __nv_bfloat162*>(&bl));
  const __nv_bfloat162 h = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&ah),
                                   *reinterpret_cast<const __nv_bfloat162*>(&bh));
  return make_uint2(*reinterpret_cast<const uint32_t*>(&l), *reinterpret_cast<const uint32_t*>(&h));
}

}  // namespace
}  // namespace b200q
