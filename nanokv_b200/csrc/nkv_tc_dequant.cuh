// INT4 code words -> bf16 latents, shared by the kernels that expand packed codes.
#pragma once

#include "nkv_tc.cuh"

namespace nkv {
namespace tc {

__device__ __forceinline__ float scale_to_float(uint16_t bits, int dtype) {
  return dtype == NKV_BF16 ? bf16_bits_to_float(bits) : __half2float(__ushort_as_half(bits));
}

// 4 code bytes (8 nibbles, even element in the low nibble) -> 8 bf16 latents
__device__ __forceinline__ uint4 dequant8(uint32_t word, float scale) {
  uint4 r;
  uint32_t* o = &r.x;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    uint32_t byte = (word >> (8 * b)) & 0xFFu;
    float lo = static_cast<float>(static_cast<int>(byte & 15u) - 7) * scale;
    float hi = static_cast<float>(static_cast<int>(byte >> 4) - 7) * scale;
    o[b] = pack_bf16x2(lo, hi);
  }
  return r;
}

// Same result with bf16 pair arithmetic and no int->float conversions, for bf16 scales:
// the bit pattern 0x4300 | n is the bf16 number 128 + n; (128 + n) - 135 = n - 7 exactly, and the
// bf16 product of two bf16 numbers is the exact product rounded once, as the reference computes it.
__device__ __forceinline__ uint4 dequant8_bf16(uint32_t word, __nv_bfloat162 scale2) {
  const uint32_t lo = word & 0x0F0F0F0Fu, hi = (word >> 4) & 0x0F0F0F0Fu;
  const uint32_t t[4] = {__byte_perm(lo, hi, 0x4400), __byte_perm(lo, hi, 0x5511),
                         __byte_perm(lo, hi, 0x6622), __byte_perm(lo, hi, 0x7733)};
  const uint32_t bias_bits = 0x43074307u;   // bf16 pair (135, 135)
  const __nv_bfloat162 bias2 = *reinterpret_cast<const __nv_bfloat162*>(&bias_bits);
  uint4 r;
  uint32_t* o = &r.x;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t bits = (t[i] & 0x00FF00FFu) | 0x43004300u;
    const __nv_bfloat162 v = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&bits), bias2), scale2);
    o[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
  return r;
}

// Kernel-order variants: the decoder rows were prepared (tc_prepare_decoder) so that within every
// group of 8 latent columns the order is e0 e2 e4 e6 e1 e3 e5 e7.  The even elements are the low
// nibbles of a code word and the odd ones its high nibbles, so a byte permute against the constant
// 0x43 builds each bf16 pair directly (4 PRMT per 8 elements instead of 4 PRMT + 4 LOP3: the
// integer pipe is what bounds the expansion).
__device__ __forceinline__ uint4 dequant8_bf16_perm(uint32_t word, __nv_bfloat162 scale2) {
  const uint32_t lo = word & 0x0F0F0F0Fu, hi = (word >> 4) & 0x0F0F0F0Fu, magic = 0x43434343u;
  const uint32_t t[4] = {__byte_perm(lo, magic, 0x4140), __byte_perm(lo, magic, 0x4342),
                         __byte_perm(hi, magic, 0x4140), __byte_perm(hi, magic, 0x4342)};
  const uint32_t bias_bits = 0x43074307u;   // bf16 pair (135, 135)
  const __nv_bfloat162 bias2 = *reinterpret_cast<const __nv_bfloat162*>(&bias_bits);
  uint4 r;
  uint32_t* o = &r.x;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 v = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&t[i]), bias2), scale2);
    o[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
  return r;
}

__device__ __forceinline__ uint4 dequant8_perm(uint32_t word, float scale) {
  float e[8];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const uint32_t byte = (word >> (8 * b)) & 0xFFu;
    e[2 * b] = static_cast<float>(static_cast<int>(byte & 15u) - 7) * scale;
    e[2 * b + 1] = static_cast<float>(static_cast<int>(byte >> 4) - 7) * scale;
  }
  return make_uint4(pack_bf16x2(e[0], e[2]), pack_bf16x2(e[4], e[6]), pack_bf16x2(e[1], e[3]),
                    pack_bf16x2(e[5], e[7]));
}

}  // namespace tc
}  // namespace nkv
