// int8 codes -> 16-bit floats, exact for all 256 codes, four at a time (one word -> two words of two
// values, in order).  Integer-to-float conversions run at a fraction of the rate of what is used here.
// With u = q + 128:
//   fp16: 0x6400 | u is the half 1024 + u; subtract 1152.
//   bf16: 0x00uu is u * 2^-133 for EVERY u below 256: at u = 128 the subnormals end and the exponent
//         field becomes 1, where the spacing is still the same.  One fused multiply-add by 2^127, the
//         largest power of two there is, and minus 2 makes it (u - 128) / 64 = q / 64, exactly.
// Either way one logic operation, two permutes and two packed operations per four codes: 64 codes per clock
// and SM.  (bf16 as 0x4300 | q took four more logic operations: 36 codes.  The permutes and logic share the
// ALU pipe, which bounded the decode kernels: HBM delivers 24 codes per clock and SM.)
// The factor 1 / 64 goes into the fp32 scale of the channel (kCodeUnit): a power of two, so no sum rounds
// differently unless it falls below 2^-126, with activations below 2^-120.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200q {
namespace {

// expand4_scaled<T> gives q / kCodeUnit<T>
template <typename T>
constexpr float kCodeUnit = 1.f;
template <>
constexpr float kCodeUnit<__nv_bfloat16> = 64.f;

template <typename T>
__device__ __forceinline__ uint2 expand4_scaled(uint32_t w);
template <>
__device__ __forceinline__ uint2 expand4_scaled<__half>(uint32_t w) {
  const uint32_t t = w ^ 0x80808080u;
  uint32_t lo = __byte_perm(t, 0x64646464u, 0x4140);
  uint32_t hi = __byte_perm(t, 0x64646464u, 0x4342);
  const __half2 bias = __floats2half2_rn(1152.f, 1152.f);
  const __half2 l = __hsub2(*reinterpret_cast<__half2*>(&lo), bias);
  const __half2 h = __hsub2(*reinterpret_cast<__half2*>(&hi), bias);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&l), *reinterpret_cast<const uint32_t*>(&h));
}
template <>
__device__ __forceinline__ uint2 expand4_scaled<__nv_bfloat16>(uint32_t w) {
  const uint32_t t = w ^ 0x80808080u;
  const uint32_t lo = __byte_perm(t, 0u, 0x4140), hi = __byte_perm(t, 0u, 0x4342);
  uint2 r;   // 0x7F00 = 2^127, 0xC000 = -2
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r.x) : "r"(lo), "r"(0x7F007F00u), "r"(0xC000C000u));
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r.y) : "r"(hi), "r"(0x7F007F00u), "r"(0xC000C000u));
  return r;
}

// the codes themselves
template <typename T>
__device__ __forceinline__ uint2 expand4(uint32_t w) {
  return expand4_scaled<T>(w);
}
template <>
__device__ __forceinline__ uint2 expand4<__nv_bfloat16>(uint32_t w) {
  // 0x4300 | (q & 0x7F) is 128 + (q mod 128), 0x4300 | (q & 0x80) is 128 or, for q < 0, 256
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
