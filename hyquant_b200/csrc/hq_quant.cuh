// Warp-level per-token quantiser (8 / 4 / 2 bits) shared by the flush kernel and the cache
// reorganisation kernel.  Bit-exact contract (reference
// src/ops/decode_d_stage.py:50-77, 104-135), q_max = 2^(bits-1) - 1:
//   absmax = max(max|x|, 1e-5);  scale = half_rn(absmax / q_max)   [IEEE fp32 divide]
//   q = clamp(rint(x / float(scale)), -q_max - 1, q_max)            [IEEE divide, half-to-even]
//   8 bits: one byte per channel;  4 bits: byte = (q[2i] & 0xF) | ((q[2i+1] & 0xF) << 4);
//   2 bits: byte = (q[4i] & 3) | (q[4i+1] & 3) << 2 | (q[4i+2] & 3) << 4 | (q[4i+3] & 3) << 6
// This translation unit must not be built with --use_fast_math.
#pragma once
#include "hq_common.cuh"

namespace hq {

// Work split: EIGHT lanes per token row, sixteen channels per lane, so a warp works on four rows at a time and the
// per-row overhead (row arithmetic, the maximum's shuffles, the scale) is paid once per four rows.  (With a whole warp
// on one row the kernels were bound by instruction issue at a fifth of the memory bandwidth.)
__device__ __forceinline__ void unpack16(const uint4& a, const uint4& b, float (&v)[16]) {      // sixteen bf16
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
}
__device__ __forceinline__ void load16(const __nv_bfloat16* p, float (&v)[16]) {
  unpack16(*reinterpret_cast<const uint4*>(p), *reinterpret_cast<const uint4*>(p + 8), v);
}
__device__ __forceinline__ void load16(const __half* p, float (&v)[16]) {
  const uint4 a = *reinterpret_cast<const uint4*>(p), b = *reinterpret_cast<const uint4*>(p + 8);
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w[i]);
    v[2 * i] = __low2float(h); v[2 * i + 1] = __high2float(h);
  }
}
__device__ __forceinline__ void load16(const float* p, float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 f = *reinterpret_cast<const float4*>(p + 4 * i);
    v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
  }
}

// Called by all 32 lanes; lanes 8 g .. 8 g + 7 hold one 128-channel token (lane l: channels 16 (l & 7) .. + 15).
// Returns the row's fp16 scale (the same on the row's eight lanes) and this lane's 16 codes packed in channel order
// into `code` (BITS / 2 words: 16 bytes at 8 bits, 8 at 4, 4 at 2); a token row is 16 * BITS bytes and lane l owns
// bytes [2 BITS (l & 7), 2 BITS ((l & 7) + 1)).
// q = rint(x / sf), the IEEE quotient rounded half to even and clamped.  Infinities and NaNs: x / inf = 0; 0 / 0 cannot happen
// (the scale is >= half(1e-5 / q_max) > 0); a NaN, inf / inf too, becomes the lowest code in the clamp.
template <int BITS>
__device__ __forceinline__ void quant_row16_exact(const float (&v)[16], float sf, uint32_t (&code)[BITS / 2]) {
  constexpr float qmax = (float)((1 << (BITS - 1)) - 1), qmin = -(float)(1 << (BITS - 1));
  constexpr int kPerWord = 32 / BITS;
#pragma unroll
  for (int w = 0; w < BITS / 2; ++w) {
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < kPerWord; ++i) {
      const float q = fminf(fmaxf(rintf(__fdiv_rn(v[w * kPerWord + i], sf)), qmin), qmax);
      c |= ((uint32_t)(__float2int_rn(q)) & ((1u << BITS) - 1u)) << (BITS * i);
    }
    code[w] = c;
  }
}

// The common row costs no division, conversion, clamp or mask, and the same whatever its values.  The product with the rounded
// reciprocal, corrected once by its remainder (Markstein, IBM J. Res. Dev. 34, 1990), is on the same side of every half-integer
// h as the IEEE quotient, and h where that is: h sf (19 bits at most) and the remainder are exact, so the quotient is h or at
// least 2^-24 h away from it, at least 2^-43 h outside what rounds to h, and the corrected product is within 2^-46 h of it before its own
// rounding.  Adding 1.5 * 2^23 rounds to the integer (ties to even, as rintf) and leaves it in the low bits; shifted and added up,
// the sixteen codes plus 2^(BITS-1) each are digits without borrows, and flipping their top bits makes them two's complement.
// The exact form takes lanes that hold a NaN, and rows whose scale is infinite or whose largest quotient rounds past q_max
// (subnormal scales only: a normal one is within 2^-11 of amax / q_max); it stands inline, because an array handed to a
// function is kept in local memory on the common path too (19 -> 31 us below).
// 8 x 32K rows of bf16 that lie in L2, codes of 2 / 4 / 8 bits: 19 / 19 / 22 us, zero rows and half-integers the same.  With a
// division instead wherever a product lies near a half-integer (bf16 rows often do in 2 bits) 31 / 25 / 22, half-integers
// 42 / 38 / 55; the reorganisation of 32K tokens of eight kv-heads 57 us, now 44 (HBM floor 26).
template <int BITS>
__device__ __forceinline__ __half quant_row16(const float (&v)[16], int scale_mode, uint32_t (&code)[BITS / 2]) {
  constexpr float qmax = (float)((1 << (BITS - 1)) - 1);
  float top = 0.f;
#pragma unroll
  for (int i = 0; i < 16; i += 2) top = fmax3_abs_nan(top, v[i], v[i + 1]);
  bool exact = top != top;
  if (exact) {                                 // a NaN does not count for the scale
    top = 0.f;
#pragma unroll
    for (int i = 0; i < 16; i += 2) top = fmax3_abs(top, v[i], v[i + 1]);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  const float amax = fmaxf(top, 1e-5f);
  const float s32 = scale_mode == 0 ? __fdiv_rn(amax, qmax) : __fmul_rn(amax, __fdiv_rn(1.0f, qmax));
  const __half sh = __float2half_rn(s32);
  const float sf = __half2float(sh);
  const float rcp = __frcp_rn(sf);
  constexpr int kPerWord = 32 / BITS;
  constexpr uint32_t kOnes = BITS == 8 ? 0x01010101u : BITS == 4 ? 0x11111111u : 0x55555555u;     // a one in every digit
  constexpr uint32_t kTop = kOnes << (BITS - 1);
  constexpr uint32_t kMagic = 0x4B400000u;                       // 1.5 * 2^23
  const float2 rcp2 = make_float2(rcp, rcp), nsf2 = make_float2(-sf, -sf), magic2 = make_float2(12582912.f, 12582912.f);
#pragma unroll
  for (int w = 0; w < BITS / 2; ++w) {
    uint32_t c = kTop - kMagic * kOnes;
#pragma unroll
    for (int i = 0; i < kPerWord; i += 2) {
      const float2 x = make_float2(v[w * kPerWord + i], v[w * kPerWord + i + 1]);
      const float2 t = fmul2(x, rcp2);
      const float2 r = fadd2(ffma2(ffma2(t, nsf2, x), rcp2, t), magic2);
      c += __float_as_uint(r.x) << (BITS * i);
      c += __float_as_uint(r.y) << (BITS * (i + 1));
    }
    code[w] = c ^ kTop;
  }
  exact |= !(rcp > 0.f && top * rcp < qmax + 0.499f);
  if (__builtin_expect(exact, 0)) quant_row16_exact<BITS>(v, sf, code);
  return sh;
}

// store the lane's codes of a token row that starts at `prow` (sub = lane & 7)
template <int BITS>
__device__ __forceinline__ void store_codes16(uint8_t* prow, int sub, const uint32_t (&code)[BITS / 2]) {
  if (BITS == 8) reinterpret_cast<uint4*>(prow)[sub] = make_uint4(code[0], code[1], code[2], code[3]);
  else if (BITS == 4) reinterpret_cast<uint2*>(prow)[sub] = make_uint2(code[0], code[BITS == 4 ? 1 : 0]);
  else reinterpret_cast<uint32_t*>(prow)[sub] = code[0];
}

// quantise one token row (eight lanes) with a run-time bit width and store its codes if `store`; returns the scale
__device__ __forceinline__ __half quant_store_row16(int bits, const float (&v)[16], int scale_mode, uint8_t* prow, int sub, bool store) {
  __half s;
  if (bits == 8) { uint32_t c[4]; s = quant_row16<8>(v, scale_mode, c); if (store) store_codes16<8>(prow, sub, c); }
  else if (bits == 4) { uint32_t c[2]; s = quant_row16<4>(v, scale_mode, c); if (store) store_codes16<4>(prow, sub, c); }
  else { uint32_t c[1]; s = quant_row16<2>(v, scale_mode, c); if (store) store_codes16<2>(prow, sub, c); }
  return s;
}

}  // namespace hq
