// Shared host/device helpers of the nanokv_b200 kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nanokv_b200.h"

namespace nkv {

// ---- host-side status plumbing -------------------------------------------
int fail(int status, const char* fmt, ...);  // records the message, returns status

#define NKV_REQUIRE(cond, status, ...)                       \
  do {                                                       \
    if (!(cond)) return ::nkv::fail((status), __VA_ARGS__);  \
  } while (0)

#define NKV_CUDA(expr)                                                          \
  do {                                                                          \
    cudaError_t err__ = (expr);                                                 \
    if (err__ != cudaSuccess)                                                   \
      return ::nkv::fail(NKV_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(err__)); \
  } while (0)

#define NKV_LAUNCH_CHECK(name)                                                  \
  do {                                                                          \
    cudaError_t err__ = cudaGetLastError();                                     \
    if (err__ != cudaSuccess)                                                   \
      return ::nkv::fail(NKV_ERR_CUDA, "launch of %s: %s", name, cudaGetErrorString(err__)); \
  } while (0)

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline size_t dtype_bytes(int dtype) { return dtype == NKV_F32 ? 4 : 2; }

// test / triage hook: route bf16 work through the fp32 CUDA-core kernels.
bool simt_forced();

// ---- device helpers ---------------------------------------------------------
__device__ __forceinline__ float bf16_bits_to_float(uint16_t bits) {
  return __uint_as_float(static_cast<uint32_t>(bits) << 16);
}

__device__ __forceinline__ float round_to_bf16(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}

__device__ __forceinline__ uint16_t float_to_bf16_bits(float v) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// two fp32 values in one 64-bit register pair: the packed operations issue once for both
__device__ __forceinline__ uint64_t pair_bits(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pair_f32(float lo, float hi) {
  return pair_bits(__float_as_uint(lo), __float_as_uint(hi));
}
__device__ __forceinline__ void split_f32(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// INT4 code (0..14, i.e. the signed code plus 7) of coefficient z for a group scale, with the
// reference's rounding points.  IN_BF16: the quotient is rounded to bf16 before rint (LingBot's
// form).  Otherwise rint(z / scale) in fp32, taken through the reciprocal: z * inv is within 2 ulp
// of the IEEE quotient, so the two can only round to different integers when z * inv lies within
// ~1e-6 of a half; exactly those values take the IEEE division.
template <bool IN_BF16>
__device__ __forceinline__ int quant_code(float z, float scale, float inv) {
  float q;
  if (IN_BF16) {
    q = round_to_bf16(__fdiv_rn(z, scale));
  } else {
    q = z * inv;
    if (fabsf(q - rintf(q)) > 0.49999f && fabsf(q) < 8.5f) q = __fdiv_rn(z, scale);
  }
  return static_cast<int>(fminf(fmaxf(rintf(q), -7.f), 7.f)) + 7;
}

// The listed values of a word redone with the IEEE division, lane by lane: a warp takes as many rounds as its
// lane with the most of them, not one per value that any of its lanes lists.
template <bool IN_BF16>
__device__ __forceinline__ uint32_t quant_word_exact(const uint32_t (&w)[4], float scale, float inv, uint32_t hits, uint32_t out) {
  for (; hits != 0; hits &= hits - 1) {
    const int e = __ffs(hits) - 1;
    const uint32_t word = (e & 4) ? ((e & 2) ? w[3] : w[2]) : ((e & 2) ? w[1] : w[0]);
    const float z = __uint_as_float((e & 1) ? (word & 0xFFFF0000u) : (word << 16));
    out = (out & ~(0xFu << (4 * e))) | (static_cast<uint32_t>(quant_code<IN_BF16>(z, scale, inv)) << (4 * e));
  }
  return out;
}

// Codes of eight bf16 coefficients (two per word, the even one in the low half) as one 32-bit word, without a
// conversion instruction per value.
template <bool IN_BF16>
__device__ __forceinline__ uint32_t quant_word(const uint32_t (&w)[4], float scale, float inv) {
  uint32_t out = 0;
  if (IN_BF16) {
    // The quotient is rounded to bf16 before rint.  z * inv is within 2 ulp of the IEEE quotient,
    // so both round to the same bf16 number unless the product's low 16 bits lie within 4 of the
    // rounding boundary 0x8000; only such values take the division (an exact boundary case cannot
    // occur: a ratio of two 8-bit mantissas is never a 9-bit midpoint).  rint of the bf16 quotient
    // is again the addition of 1.5 * 2^23 (exact on a bf16 number, ties to even as rint has them).
    constexpr float MAGIC = 12582912.0f;
    constexpr uint32_t MAGIC_BITS = 0x4B400000u;
    constexpr uint32_t PACK_BIAS = (MAGIC_BITS - 7u) * 0x11111111u;
    bool ambiguous = false;
    uint32_t acc = 0;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      const float q1 = __uint_as_float(w[k] & 0xFFFF0000u) * inv;
      const float q0 = __uint_as_float(w[k] << 16) * inv;
      ambiguous |= ((__float_as_uint(q1) + 0x8004u) & 0xFFFFu) <= 8u;
      ambiguous |= ((__float_as_uint(q0) + 0x8004u) & 0xFFFFu) <= 8u;
      const __nv_bfloat162 rounded = __floats2bfloat162_rn(q0, q1);
      const uint32_t both = *reinterpret_cast<const uint32_t*>(&rounded);
      const float t1 = __uint_as_float(both & 0xFFFF0000u) + MAGIC;
      const float t0 = __uint_as_float(both << 16) + MAGIC;
      acc = (acc << 4) + __float_as_uint(t1);
      acc = (acc << 4) + __float_as_uint(t0);
    }
    out = acc - PACK_BIAS;
    if (ambiguous) {
      uint32_t hits = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float z = __uint_as_float((e & 1) ? (w[e >> 1] & 0xFFFF0000u) : (w[e >> 1] << 16));
        if (((__float_as_uint(z * inv) + 0x8004u) & 0xFFFFu) <= 8u) hits |= 1u << e;
      }
      out = quant_word_exact<true>(w, scale, inv, hits, out);
    }
  } else {
    // whole piece through the reciprocal; a piece holding a value whose scaled form lies within
    // 1e-5 of a half-integer (where the reciprocal and the IEEE quotient could round apart) is
    // redone value by value with the exact rule.  Rounding to the nearest-even integer is the
    // fp32 addition of 1.5 * 2^23 (the integer then sits in the low mantissa bits), which keeps
    // the whole loop on the full-rate floating-point and integer pipes: no conversion
    // instruction per value.  No clamp is needed here: |z| <= the group's maximum and
    // scale = max(that, eps) / 7 bound |z * inv| by 7 (1 + 2^-22) for every finite row, and a row
    // with a non-finite value has no defined codes in the reference either (the 32-bit word of
    // such a piece may then hold arbitrary bits; nothing outside that word is touched).
    constexpr float MAGIC = 12582912.0f;
    constexpr uint32_t MAGIC_BITS = 0x4B400000u;
    // the float bits of (q + MAGIC) are MAGIC_BITS + rint(q): eight of them, each shifted four
    // bits further, add up (mod 2^32) to the packed word plus a constant
    constexpr uint32_t PACK_BIAS = (MAGIC_BITS - 7u) * 0x11111111u;
    float worst = 0.f;
    uint32_t acc = 0;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      const float q1 = __uint_as_float(w[k] & 0xFFFF0000u) * inv;
      const float q0 = __uint_as_float(w[k] << 16) * inv;
      const float t1 = q1 + MAGIC, t0 = q0 + MAGIC;
      worst = fmaxf(worst, fabsf(q1 - (t1 - MAGIC)));
      worst = fmaxf(worst, fabsf(q0 - (t0 - MAGIC)));
      acc = (acc << 4) + __float_as_uint(t1);
      acc = (acc << 4) + __float_as_uint(t0);
    }
    out = acc - PACK_BIAS;
    const bool near_half = worst > 0.49999f;
    if (near_half) {
      // exact ties are not rare (a row whose maximum has a mantissa divisible by 7 holds many),
      // so only the values that are near a half take the IEEE division; their nibble is replaced
      uint32_t hits = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float z = __uint_as_float((e & 1) ? (w[e >> 1] & 0xFFFF0000u) : (w[e >> 1] << 16));
        const float q = z * inv;
        if (fabsf(q - ((q + MAGIC) - MAGIC)) > 0.49999f) hits |= 1u << e;
      }
      out = quant_word_exact<false>(w, scale, inv, hits, out);
    }
  }
  return out;
}

// element i of an array of the given element type, as float (exact)
__device__ __forceinline__ float load_float(const void* base, int dtype, size_t i) {
  if (dtype == NKV_F32) return static_cast<const float*>(base)[i];
  uint16_t bits = static_cast<const uint16_t*>(base)[i];
  if (dtype == NKV_BF16) return bf16_bits_to_float(bits);
  return __half2float(__ushort_as_half(bits));
}

__device__ __forceinline__ void store_float(void* base, int dtype, size_t i, float v) {
  if (dtype == NKV_F32) {
    static_cast<float*>(base)[i] = v;
  } else if (dtype == NKV_BF16) {
    static_cast<uint16_t*>(base)[i] = float_to_bf16_bits(v);
  } else {
    static_cast<uint16_t*>(base)[i] = __half_as_ushort(__float2half_rn(v));
  }
}

__device__ __forceinline__ int load_id(const void* ids, int id_bytes, size_t t) {
  return id_bytes == 1 ? static_cast<const uint8_t*>(ids)[t]
                       : static_cast<const uint16_t*>(ids)[t];
}

// Segment of token t: largest s with seg_start[s] <= t (binary search).
__device__ __forceinline__ int find_segment(const int32_t* seg_start, int segments, int t) {
  int lo = 0, hi = segments - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (seg_start[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Row of the stacked centre table that token t was assigned to.
__device__ __forceinline__ int center_row_of(const nkv_history& h, int t) {
  int s = find_segment(h.seg_start, h.segments, t);
  return h.seg_center_row[s] + load_id(h.ids, h.id_bytes, t);
}

// latent coefficient j of token t: code * stored scale (exact in fp32).
__device__ __forceinline__ float latent_value(const nkv_history& h, int t, int j) {
  uint8_t byte = h.codes[static_cast<size_t>(t) * (h.rank >> 1) + (j >> 1)];
  int nibble = (j & 1) ? (byte >> 4) : (byte & 15);
  float scale = load_float(h.scales, h.scale_dtype,
                           static_cast<size_t>(t) * (h.rank / h.group) + j / h.group);
  return static_cast<float>(nibble - 7) * scale;
}

}  // namespace nkv
