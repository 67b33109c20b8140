// Operand preparation for the hybrid prefill kernel (one pass over Q and K):
//   * K smoothing: k_sm = k - mean_n(k) per (batch, kv-head, channel), formed in bf16
//     like the reference (src/ops/sage_unified.py:565-568);
//   * INT8 of k_sm and of q * sm_scale * log2(e) with scale = max|x| / 127 and
//     round-half-away-from-zero — the arithmetic of the reference's block quantiser
//     (src/ops/vendor/sageattention/triton/quant_per_block.py:21-47) applied with one scale
//     per token row instead of one per 64-key / 128-query block: an outlier row then costs
//     no precision in its neighbours, and the scales are applied to the fp32 score for free;
//   * a contiguous BF16 copy of the query for the BF16 tiles (unscaled: the kernel applies
//     sm_scale * log2(e) to the fp32 score, so no rounding is added to the query).
// HBM-bound: reads Q and K once, writes the INT8 and BF16 copies.
#include "hq_common.cuh"

namespace hq {

constexpr int kMeanChunks = 32;

// partial[bh][chunk][128] = sum over the chunk's rows.  Sixteen threads own a row (16 bytes each), so a block has sixteen
// rows in flight per load instruction and the rows of a trip are independent (two-byte loads, two rows at a time, took
// 16 us for 8 heads x 8192 rows, 16 MB).
__global__ void __launch_bounds__(256)
kmean_partial_kernel(const __nv_bfloat16* __restrict__ k, int64_t sb, int64_t sh, int64_t sn, int H, int N,
                     float* __restrict__ partial) {
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H, chunk = blockIdx.x;
  const int grp = threadIdx.x >> 4, c = (threadIdx.x & 15) * 8;
  const int rows_per = (N + kMeanChunks - 1) / kMeanChunks;
  const int r0 = chunk * rows_per, r1 = min(N, r0 + rows_per);
  const __nv_bfloat16* base = k + b * sb + h * sh + c;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
  for (int r = r0 + grp; r < r1; r += 16) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(base + (int64_t)r * sn));
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[2 * j] += __uint_as_float(w[j] << 16); acc[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u); }
  }
  __shared__ float s[16][128];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[grp][c + j] = acc[j];
  __syncthreads();
  if (threadIdx.x < 128) {
    float t = 0.f;
#pragma unroll
    for (int g = 0; g < 16; ++g) t += s[g][threadIdx.x];
    partial[((int64_t)bh * kMeanChunks + chunk) * 128 + threadIdx.x] = t;
  }
}

__global__ void kmean_final_kernel(const float* __restrict__ partial, int N, int smooth, __nv_bfloat16* __restrict__ mean) {
  const int bh = blockIdx.x, d = threadIdx.x;
  float acc = 0.f;
#pragma unroll
  for (int c = 0; c < kMeanChunks; ++c) acc += partial[((int64_t)bh * kMeanChunks + c) * 128 + d];
  mean[(int64_t)bh * 128 + d] = __float2bfloat16_rn(smooth ? acc / (float)N : 0.f);
}

// kIsK: subtract the bf16 mean (rounding the difference to bf16) and write it as the BF16 copy; else multiply by `mul`
// in fp32 and quantise the fp32 product (the BF16 query copy is the row itself; xbf == nullptr: the caller reads x).
// One INT8 scale per ROW (token): scale = max|x| / 127, code = x / scale rounded half away from zero; rows N ..
// scale_pitch - 1 get scale 0.
//
// Eight lanes per row, sixteen channels each, 32 rows per CTA.  Bound by instruction issue before HBM, so the work per
// element is kept small: the row maximum on pairs of bf16 bit patterns, everything else on magnitudes, two to an
// instruction, the sign put back on four packed bytes at a time.  Rounding half away from zero is |y| + 0.5 cut off, and
// y has to be the correctly rounded quotient (a bf16 value over a 127th of another lies exactly on a tie often enough
// that falling back near ties meant falling back in most warps): Markstein's division (IBM J. Res. Dev. 34, 1990),
// the product with the rounded reciprocal corrected once by its exact remainder.  Rows that hold a
// NaN, and rows whose maximum is infinite or out of that method's range, take the divide instruction element by element:
// x / inf = 0; NaN (inf / inf too) becomes the lowest code in the clamp.
__device__ __noinline__ void row_codes_exact(const float (&v)[16], float sc, uint32_t (&code)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t c = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float y = __fdiv_rn(v[4 * i + e], sc);
      y += y >= 0.f ? 0.5f : -0.5f;
      c |= ((uint32_t)(int)fminf(fmaxf(truncf(y), -128.f), 127.f) & 0xFFu) << (8 * e);
    }
    code[i] = c;
  }
}

template <bool kIsK>
__global__ void __launch_bounds__(256, 5)
row_quant_kernel(const __nv_bfloat16* __restrict__ x, int64_t sb, int64_t sh, int64_t sn, int H, int N,
                 const __nv_bfloat16* __restrict__ mean, float mul,
                 int8_t* __restrict__ xi8, __nv_bfloat16* __restrict__ xbf, float* __restrict__ scale, int scale_pitch) {
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
  const int tid = threadIdx.x;
  const int row = blockIdx.x * 32 + (tid >> 3), c = (tid & 7) * 16;
  const bool ok = row < N;
  uint4 raw[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  if (ok) {
    const uint4* src = reinterpret_cast<const uint4*>(x + b * sb + h * sh + (int64_t)row * sn + c);
    raw[0] = __ldg(src); raw[1] = __ldg(src + 1);
  }
  uint32_t w[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
  if (kIsK) {
    uint32_t mw[8];
    const __nv_bfloat16* mp = mean + (int64_t)bh * 128 + c;
    if ((reinterpret_cast<uintptr_t>(mp) & 15) == 0) {
      const uint4 m0 = __ldg(reinterpret_cast<const uint4*>(mp)), m1 = __ldg(reinterpret_cast<const uint4*>(mp) + 1);
      mw[0] = m0.x; mw[1] = m0.y; mw[2] = m0.z; mw[3] = m0.w; mw[4] = m1.x; mw[5] = m1.y; mw[6] = m1.z; mw[7] = m1.w;
    } else {
      const uint16_t* e = reinterpret_cast<const uint16_t*>(mp);
#pragma unroll
      for (int j = 0; j < 8; ++j) mw[j] = (uint32_t)__ldg(e + 2 * j) | ((uint32_t)__ldg(e + 2 * j + 1) << 16);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __nv_bfloat162 d = __floats2bfloat162_rn(__uint_as_float(w[j] << 16) - __uint_as_float(mw[j] << 16),
                                                     __uint_as_float(w[j] & 0xFFFF0000u) - __uint_as_float(mw[j] & 0xFFFF0000u));
      w[j] = *reinterpret_cast<const uint32_t*>(&d);
    }
  }
  // max|x| over the row: magnitudes of bf16 values order like their bit patterns, NaN above infinity
  uint32_t pm = 0u;
#pragma unroll
  for (int j = 0; j < 8; ++j) pm = __vmaxu2(pm, w[j] & 0x7FFF7FFFu);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) pm = __vmaxu2(pm, __shfl_xor_sync(0xffffffffu, pm, o));
  const uint32_t top = max(pm & 0xFFFFu, pm >> 16);
  if (!ok) {
    if ((tid & 7) == 0 && row < scale_pitch) scale[(int64_t)bh * scale_pitch + row] = 0.f;
    return;
  }
  if (kIsK || xbf != nullptr) {
    uint4* dst = reinterpret_cast<uint4*>(xbf + ((int64_t)bh * N + row) * 128 + c);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
  float amax = __uint_as_float(top << 16) * (kIsK ? 1.0f : fabsf(mul));
  if (top > 0x7F80u) {                                  // a NaN in the row does not count for its maximum
    amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(w[j] << 16) * (kIsK ? 1.0f : mul)), fabsf(__uint_as_float(w[j] & 0xFFFF0000u) * (kIsK ? 1.0f : mul))));
    const uint32_t lanes = 0xFFu << (tid & 24);         // the row's eight lanes are here together
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(lanes, amax, o));
  }
  const float sc = __fdiv_rn(fmaxf(amax, 1e-30f), 127.f);     // an all-zero row keeps codes 0 instead of NaN
  if ((tid & 7) == 0) scale[(int64_t)bh * scale_pitch + row] = sc;
  const float rcp = __frcp_rn(sc);
  const float2 rcp2 = make_float2(rcp, rcp), nsc2 = make_float2(-sc, -sc), half2 = make_float2(0.5f, 0.5f);
  const float2 big2 = make_float2(8388608.f, 8388608.f), mul2 = make_float2(fabsf(mul), fabsf(mul));
  const uint32_t turn = !kIsK && mul < 0.f ? 0xFFFFFFFFu : 0u;
  // two magnitudes of a word -> floor(quotient + 0.5) in the low mantissa bits
  auto two = [&](uint32_t word) -> float2 {
    const uint32_t m = word & 0x7FFF7FFFu;
    float2 v = make_float2(__uint_as_float(m << 16), __uint_as_float(m & 0xFFFF0000u));
    if (!kIsK) v = fmul2(v, mul2);
    const float2 q = fmul2(v, rcp2);
    const float2 y = ffma2(ffma2(q, nsc2, v), rcp2, q);
    return fadd2_rz(fadd2(y, half2), big2);
  };
  uint32_t code[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 r0 = two(w[2 * i]), r1 = two(w[2 * i + 1]);
    const uint32_t n = prmt(prmt(__float_as_uint(r0.x), __float_as_uint(r0.y), 0x0040), prmt(__float_as_uint(r1.x), __float_as_uint(r1.y), 0x0040), 0x5410);
    const uint32_t neg = prmt(w[2 * i], w[2 * i + 1], 0xFDB9) ^ turn;       // 0xFF in the bytes of negative elements
    const uint32_t flipped = n ^ neg;                                       // n <= 127: minus n is its complement plus one
    code[i] = ((flipped & 0x7F7F7F7Fu) + (neg & 0x01010101u)) ^ (flipped & 0x80808080u);
  }
  if (top > 0x7F80u || !(amax >= 1e-25f && amax <= 1e30f)) {
    float v[16];                        // arrays of their own: what goes to the call by address must not be the common path's
    uint32_t exact[4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[2 * j] = __uint_as_float(w[j] << 16); v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
      if (!kIsK) { v[2 * j] *= mul; v[2 * j + 1] *= mul; }
    }
    row_codes_exact(v, sc, exact);
#pragma unroll
    for (int j = 0; j < 4; ++j) code[j] = exact[j];
  }
  int8_t* out = xi8 + ((int64_t)bh * N + row) * 128 + c;       // 8-byte aligned at least
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    *reinterpret_cast<uint4*>(out) = make_uint4(code[0], code[1], code[2], code[3]);
  } else {
    reinterpret_cast<uint2*>(out)[0] = make_uint2(code[0], code[1]);
    reinterpret_cast<uint2*>(out)[1] = make_uint2(code[2], code[3]);
  }
}


// ---- the reference's block quantiser, bit for bit --------------------------------------------------------
// quant_per_block_int8_kernel (src/ops/vendor/sageattention/triton/quant_per_block.py:21-47): one scale per
// block of `blk` token rows x 128 channels, scale = max|x * mul| / 127, code = trunc(x * mul / scale + 0.5 sign).
// Triton lowers both fp32 divisions to div.full.f32 (not IEEE), so this kernel issues the same instruction;
// an all-zero block gives scale 0 and 0 / 0 = NaN, which the float -> int conversion turns into code 0.
__device__ __forceinline__ float div_full(float a, float b) {
  float r;
  asm("div.full.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// One CTA per (block, head): 256 threads, 16 threads per row, 8 channels each, rows in steps of 16.
// `mean` (bf16 [BH,128], may be null): subtracted first and the difference rounded to bf16, as k - km is
// formed in the input dtype before the kernel (quant_per_block.py:53-54).
// scale_rows (may be null) receives the block's scale once per token row ([BH, row_pitch]), the layout the
// attention kernel reads; scale_blocks (may be null) is the reference's [BH, ceil(L / blk)].
__global__ void __launch_bounds__(256)
block_quant_kernel(const __nv_bfloat16* __restrict__ x, int64_t sb, int64_t sh, int64_t sn, int H, int L, int blk,
                   const __nv_bfloat16* __restrict__ mean, float mul, int8_t* __restrict__ xi8, int64_t ob, int64_t oh,
                   int64_t on, __nv_bfloat16* __restrict__ xbf, float* __restrict__ scale_blocks, int nblk,
                   float* __restrict__ scale_rows, int row_pitch) {
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H, r0 = blockIdx.x * blk;
  const int tid = threadIdx.x, c = (tid & 15) * 8;
  const __nv_bfloat16* src = x + b * sb + h * sh;
  float m[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) m[j] = mean ? __bfloat162float(mean[(int64_t)bh * 128 + c + j]) : 0.f;
  auto load_row = [&](int row, float (&v)[8]) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)row * sn + c));
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float f0 = __uint_as_float(w[j] << 16), f1 = __uint_as_float(w[j] & 0xFFFF0000u);
      if (mean) {
        f0 = __bfloat162float(__float2bfloat16_rn(f0 - m[2 * j]));
        f1 = __bfloat162float(__float2bfloat16_rn(f1 - m[2 * j + 1]));
      }
      v[2 * j] = f0; v[2 * j + 1] = f1;
    }
  };
  float amax = 0.f;
  for (int row = r0 + (tid >> 4); row < min(L, r0 + blk); row += 16) {
    float v[8];
    load_row(row, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j] * mul));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  __shared__ float s_max[8];
  if ((tid & 31) == 0) s_max[tid >> 5] = amax;
  __syncthreads();
  amax = s_max[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) amax = fmaxf(amax, s_max[w]);
  const float sc = div_full(amax, 127.f);
  if (tid == 0 && scale_blocks) scale_blocks[(int64_t)bh * nblk + blockIdx.x] = sc;
  for (int row = r0 + (tid >> 4); row < min(L, r0 + blk); row += 16) {
    float v[8];
    load_row(row, v);
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float y = div_full(v[j] * mul, sc);
      y += y >= 0.f ? 0.5f : -0.5f;
      const int q = (y != y) ? 0 : (int)y;                      // truncation towards zero; NaN -> 0
      (j < 4 ? lo : hi) |= ((uint32_t)(uint8_t)(int8_t)q) << (8 * (j & 3));
    }
    *reinterpret_cast<uint2*>(xi8 + b * ob + h * oh + (int64_t)row * on + c) = make_uint2(lo, hi);
    if (xbf) {
      uint4 o4;
      uint32_t* ow = reinterpret_cast<uint32_t*>(&o4);
      if (mean) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { __nv_bfloat162 pk = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]); ow[j] = *reinterpret_cast<uint32_t*>(&pk); }
      } else {
        o4 = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)row * sn + c));
      }
      *reinterpret_cast<uint4*>(xbf + ((int64_t)bh * L + row) * 128 + c) = o4;
    }
    if (scale_rows && (tid & 15) == 0) scale_rows[(int64_t)bh * row_pitch + row] = fmaxf(sc, 1e-30f);
  }
}

}  // namespace hq

extern "C" int hq_prefill_quant_workspace_bytes(int B, int H_KV, int64_t* bytes) {
  using namespace hq;
  HQ_REQUIRE(bytes && B > 0 && H_KV > 0, HQ_ERR_INVALID, "hq_prefill_quant_workspace_bytes: bad sizes");
  *bytes = (int64_t)B * H_KV * kMeanChunks * 128 * 4;
  return HQ_OK;
}

extern "C" int hq_prefill_quant(const void* q, int64_t q_sb, int64_t q_sh, int64_t q_sn,
                                const void* k, int64_t k_sb, int64_t k_sh, int64_t k_sn,
                                int B, int H_Q, int H_KV, int N, float sm_scale, int smooth_k,
                                void* q_i8, void* q_bf, float* q_scale,
                                void* k_i8, void* k_bf, float* k_scale, void* k_mean,
                                void* workspace, int64_t workspace_bytes, void* stream) {
  using namespace hq;
  HQ_REQUIRE(B > 0 && H_Q > 0 && H_KV > 0 && N > 0, HQ_ERR_INVALID, "hq_prefill_quant: bad sizes");
  HQ_REQUIRE(q && k && q_i8 && q_bf && q_scale && k_i8 && k_bf && k_scale && k_mean && workspace, HQ_ERR_INVALID,
             "hq_prefill_quant: null pointer");
  int64_t need = 0;
  hq_prefill_quant_workspace_bytes(B, H_KV, &need);
  HQ_REQUIRE(workspace_bytes >= need, HQ_ERR_WORKSPACE, "hq_prefill_quant: workspace of %lld bytes needed", (long long)need);
  HQ_REQUIRE(aligned16(q) && aligned16(k) && q_sb % 8 == 0 && q_sh % 8 == 0 && q_sn % 8 == 0 && k_sb % 8 == 0 &&
                 k_sh % 8 == 0 && k_sn % 8 == 0,
             HQ_ERR_ALIGNMENT, "hq_prefill_quant: q/k rows must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const __nv_bfloat16* kk = (const __nv_bfloat16*)k;
  const int nrb = ((N + 63) / 64 * 64) / 32;                      // the padding rows' scales are written too
  // q_bf may be q itself when q is contiguous (a dimension of one row has no stride): the copy is then left out
  const bool same_q = q_bf == q && (N == 1 || q_sn == 128) && (H_Q == 1 || q_sh == (int64_t)N * 128) &&
                      (B == 1 || q_sb == (int64_t)H_Q * N * 128);
  HQ_REQUIRE(q_bf != q || same_q, HQ_ERR_INVALID, "hq_prefill_quant: q_bf may be q only if q is contiguous");
  kmean_partial_kernel<<<dim3(kMeanChunks, B * H_KV), 256, 0, st>>>(kk, k_sb, k_sh, k_sn, H_KV, N, (float*)workspace);
  kmean_final_kernel<<<B * H_KV, 128, 0, st>>>((const float*)workspace, N, smooth_k, (__nv_bfloat16*)k_mean);
  row_quant_kernel<true><<<dim3(nrb, B * H_KV), 256, 0, st>>>(kk, k_sb, k_sh, k_sn, H_KV, N, (const __nv_bfloat16*)k_mean, 1.0f,
                                                             (int8_t*)k_i8, (__nv_bfloat16*)k_bf, k_scale, (N + 63) / 64 * 64);
  row_quant_kernel<false><<<dim3(nrb, B * H_Q), 256, 0, st>>>((const __nv_bfloat16*)q, q_sb, q_sh, q_sn, H_Q, N, nullptr,
                                                             sm_scale * 1.44269504f, (int8_t*)q_i8,
                                                             same_q ? nullptr : (__nv_bfloat16*)q_bf, q_scale, (N + 63) / 64 * 64);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

extern "C" int hq_per_block_int8(const void* x, int64_t x_sb, int64_t x_sh, int64_t x_sn, int B, int H, int L, int blk,
                                 float mul, const void* mean, void* x_i8, int64_t o_sb, int64_t o_sh, int64_t o_sn,
                                 float* scale, void* stream) {
  using namespace hq;
  HQ_REQUIRE(x && x_i8 && scale && B > 0 && H > 0 && L > 0 && blk > 0, HQ_ERR_INVALID, "hq_per_block_int8: bad arguments");
  HQ_REQUIRE(aligned16(x) && x_sb % 8 == 0 && x_sh % 8 == 0 && x_sn % 8 == 0 && ((uintptr_t)x_i8 & 7) == 0 && o_sb % 8 == 0 &&
                 o_sh % 8 == 0 && o_sn % 8 == 0, HQ_ERR_ALIGNMENT, "hq_per_block_int8: rows must be 16-byte (input) / 8-byte (codes) aligned");
  const int nblk = (L + blk - 1) / blk;
  block_quant_kernel<<<dim3(nblk, B * H), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, x_sb, x_sh, x_sn, H, L, blk, (const __nv_bfloat16*)mean, mul, (int8_t*)x_i8, o_sb, o_sh, o_sn,
      nullptr, scale, nblk, nullptr, 0);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

extern "C" int hq_prefill_quant_blocks(const void* q, int64_t q_sb, int64_t q_sh, int64_t q_sn,
                                       const void* k, int64_t k_sb, int64_t k_sh, int64_t k_sn,
                                       int B, int H_Q, int H_KV, int N, float sm_scale, int smooth_k,
                                       void* q_i8, void* q_bf, float* q_scale,
                                       void* k_i8, void* k_bf, float* k_scale, void* k_mean,
                                       void* workspace, int64_t workspace_bytes, void* stream) {
  using namespace hq;
  HQ_REQUIRE(B > 0 && H_Q > 0 && H_KV > 0 && N > 0, HQ_ERR_INVALID, "hq_prefill_quant_blocks: bad sizes");
  HQ_REQUIRE(q && k && q_i8 && q_bf && q_scale && k_i8 && k_bf && k_scale && k_mean && workspace, HQ_ERR_INVALID,
             "hq_prefill_quant_blocks: null pointer");
  int64_t need = 0;
  hq_prefill_quant_workspace_bytes(B, H_KV, &need);
  HQ_REQUIRE(workspace_bytes >= need, HQ_ERR_WORKSPACE, "hq_prefill_quant_blocks: workspace of %lld bytes needed", (long long)need);
  HQ_REQUIRE(aligned16(q) && aligned16(k) && q_sb % 8 == 0 && q_sh % 8 == 0 && q_sn % 8 == 0 && k_sb % 8 == 0 &&
                 k_sh % 8 == 0 && k_sn % 8 == 0,
             HQ_ERR_ALIGNMENT, "hq_prefill_quant_blocks: q/k rows must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const __nv_bfloat16* kk = (const __nv_bfloat16*)k;
  kmean_partial_kernel<<<dim3(kMeanChunks, B * H_KV), 256, 0, st>>>(kk, k_sb, k_sh, k_sn, H_KV, N, (float*)workspace);
  kmean_final_kernel<<<B * H_KV, 128, 0, st>>>((const float*)workspace, N, smooth_k, (__nv_bfloat16*)k_mean);
  const int pitch = (N + 63) / 64 * 64;
  block_quant_kernel<<<dim3((N + 63) / 64, B * H_KV), 256, 0, st>>>(
      kk, k_sb, k_sh, k_sn, H_KV, N, 64, smooth_k ? (const __nv_bfloat16*)k_mean : nullptr, 1.0f, (int8_t*)k_i8,
      (int64_t)H_KV * N * 128, (int64_t)N * 128, 128, (__nv_bfloat16*)k_bf, nullptr, 0, k_scale, pitch);
  block_quant_kernel<<<dim3((N + 127) / 128, B * H_Q), 256, 0, st>>>(
      (const __nv_bfloat16*)q, q_sb, q_sh, q_sn, H_Q, N, 128, nullptr, sm_scale * 1.44269504f, (int8_t*)q_i8,
      (int64_t)H_Q * N * 128, (int64_t)N * 128, 128, (__nv_bfloat16*)q_bf, nullptr, 0, q_scale, pitch);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}
