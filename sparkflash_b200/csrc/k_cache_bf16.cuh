// Cache codes to bf16, shared by the two attention kernels over the quantised caches (k_attn.cu, k_attn_tc.cu).
#pragma once
#include "k_common.cuh"

namespace sfb {

// ---- cache codes -> bf16 by bit placement ----------------------------------------------------------------------
// An E4M3 byte shifted into a bf16 (sign to bit 15, the seven exponent|mantissa bits to bits 4..10) is the code's value
// times 2^-120, subnormal codes included (they land on bf16 subnormals).  Two exact bf16 multiplications by powers of two, 2^120 and
// the block scale, make it the entry: first the code's value, then the product, so that any scale gives what the entry is - beyond
// bf16's range an infinity.  An E2M1 nibble is looked up and multiplied by its E4M3 scale: two significant bits times four.  Every
// intermediate is representable, so the result is the exact product.
__device__ __forceinline__ uint32_t e4m3x2_to_bf16x2_raw(uint32_t two_bytes_in_high_halves) {
  // input: byte a in bits 8..15, byte b in bits 24..31
  const uint32_t t = two_bytes_in_high_halves;
  return (t & 0x80008000u) | ((t >> 4) & 0x07f007f0u);
}
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf16x2_splat(float f) {
  __nv_bfloat162 r = __float2bfloat162_rn(f);
  return *reinterpret_cast<uint32_t*>(&r);
}
// a UE8M0 scale, 2^(code - 127), in both halves of a word: the code is the exponent field, and 0 is a subnormal
__device__ __forceinline__ uint32_t ue8m0_splat(uint8_t code) { return code ? (uint32_t)code * 0x00800080u : 0x00400040u; }
// 16 E4M3 codes (one uint4) with one splatted power-of-two scale -> two uint4 of bf16
__device__ __forceinline__ void fp8x16_to_bf16(const uint4& v, uint32_t scale, uint4& o0, uint4& o1) {
  constexpr uint32_t M120 = 0x7b807b80u;      // 2^120, twice
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t r[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lo = __byte_perm(w[i], 0u, 0x1404);   // bytes: [0, b0, 0, b1] -> b0 in bits 8..15, b1 in bits 24..31
    const uint32_t hi = __byte_perm(w[i], 0u, 0x3424);   // b2, b3
    r[2 * i] = bf16x2_mul(bf16x2_mul(e4m3x2_to_bf16x2_raw(lo), M120), scale);
    r[2 * i + 1] = bf16x2_mul(bf16x2_mul(e4m3x2_to_bf16x2_raw(hi), M120), scale);
  }
  o0 = make_uint4(r[0], r[1], r[2], r[3]);
  o1 = make_uint4(r[4], r[5], r[6], r[7]);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// 8 E2M1 codes (one 32-bit word, element i in nibble i) times one splatted bf16 scale -> one uint4 of bf16.  The codes are the selectors of
// byte permutations: their low three bits look up the two bytes of the magnitude's bf16 form, and the sign bit, which as a selector's top
// bit asks for the sign of the byte looked up, turns 0x80 into 0xff.
__device__ __forceinline__ uint4 fp4x8_to_bf16(uint32_t w, uint32_t scale) {
  const uint32_t m = w & 0x77777777u;
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t sel = m >> (16 * i);
    const uint32_t sign = (prmt(0x80808080u, 0x80808080u, w >> (16 * i)) << 1) & 0x80808080u;
    const uint32_t hi = prmt(0x3f3f3f00u, 0x40404040u, sel) | sign, lo = prmt(0xc0800000u, 0xc0804000u, sel);
    r[2 * i] = bf16x2_mul(prmt(lo, hi, 0x5140u), scale);
    r[2 * i + 1] = bf16x2_mul(prmt(lo, hi, 0x7362u), scale);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}
// two E4M3 scales (exact in bf16), each in both halves of a word
__device__ __forceinline__ void e4m3x2_splat(uint16_t two, uint32_t& s0, uint32_t& s1) {
  const float2 f = cvt_e4m3x2(two);
  s0 = bf16x2_splat(f.x);
  s1 = bf16x2_splat(f.y);
}

}  // namespace sfb
