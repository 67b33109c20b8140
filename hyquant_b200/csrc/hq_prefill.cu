// Hybrid-precision causal prefill attention, GQA-native: entry points and vertical-line bookkeeping.
//
// For the 128-query block starting at s of query head h (kv head h / R):
//   keys j <  wla(s)          : INT8 QK^T (one scale per query row and per key row, smoothed K)
//                               unless j is a vertical line of head h -> masked there and taken
//                               from the gathered BF16 vertical tiles instead;
//   vertical lines < wla(s)   : BF16 QK^T on the gathered rows (ascending position);
//   keys in [wla(s), s + 128) : BF16 QK^T with the causal mask (local window + diagonal);
// with wla(s) = floor(max(0, s - (W - 1)) / 64) * 64 — the block rule of the reference kernel
// (src/ops/sage_unified.py:483-485, 538-544).  All tiles share one online softmax in base 2 and one
// fp32 accumulator; P V runs in BF16.  Unlike the reference nothing is expanded to query heads or
// physically reordered: K / V stay at kv-head granularity and a per (query head, key) additive
// term of the INT8 score conversion, -inf on the head's vertical lines, removes those columns from
// the INT8 pass.
//
// Tensor-bound.  FLOPs per call: 4 * B * H_Q * 128 * N (N + 1) / 2.  The attention kernel itself
// (tcgen05 / tensor memory / TMA) lives in hq_prefill_tc.cu.
#include <cstddef>
#include "hq_common.cuh"

namespace hq {

// Vertical-line bookkeeping: for every (batch, query head) the ascending index list gives
//   k_bias[key]  = -12582912 * k_scale[key], or -inf if the key is a vertical line of this head: the
//                  INT8 pass turns an s32 score i into float as bits(i + 0x4B400000) = 12582912 + i and
//                  applies the key scale and this term in one fused multiply-add;
//   nv_valid[qb] = number of vertical lines below wla(128 qb)
// (the role of the reference's reorder_kv_for_vertical counts, src/ops/sage_unified.py:537-544)
// One block per 1024 keys of a (batch, query head): the block finds its piece of the index list (one CTA per head walked
// the whole row of biases: 19 us for 32 heads x 8192 keys on 32 SMs).
constexpr int kMetaKeys = 1024;
__device__ __forceinline__ int count_below(const int* a, int n, int v) {
  int lo = 0, hi = n;
  while (lo < hi) { const int mid = (lo + hi) >> 1; if (__ldg(a + mid) < v) lo = mid + 1; else hi = mid; }
  return lo;
}
__global__ void __launch_bounds__(256)
vertical_meta_kernel(const int* __restrict__ vasc, int T, int N, int Npad, int W, int nqb, int R,
                     const float* __restrict__ k_scale, float* __restrict__ k_bias, int* __restrict__ nv_valid) {
  const int64_t bh = blockIdx.y;
  const int x0 = blockIdx.x * kMetaKeys, x1 = min(Npad, x0 + kMetaKeys), tid = threadIdx.x;
  const float* ks = k_scale + (bh / R) * Npad;           // (b, hq) -> (b, hq / R): heads of a batch are contiguous
  float* kb = k_bias + bh * Npad;
  for (int x = x0 + tid; x < x1; x += 256) kb[x] = -12582912.0f * ks[x];
  if (T == 0) return;
  const int* a = vasc + bh * T;
  // query blocks whose number falls to this block (the last block takes what is left)
  const int per = (nqb + gridDim.x - 1) / gridDim.x;
  for (int qb = blockIdx.x * per + tid; qb < min(nqb, (int)(blockIdx.x + 1) * per); qb += 256) {
    const int s0 = qb * 128;
    nv_valid[bh * nqb + qb] = count_below(a, T, W > 0 ? (max(0, s0 - (W - 1)) / 64) * 64 : s0);
  }
  __syncthreads();                                         // the biases are written: the lines may overwrite them
  const int lo = count_below(a, T, x0), hi = count_below(a, T, min(x1, N));
  for (int i = lo + tid; i < hi; i += 256) kb[a[i]] = -INFINITY;
}

// idx int64 [rows, T] in any order -> asc int32 [rows, T]: clamped to [0, last], ascending (a position given twice
// stays twice).  Latency-bound, one CTA per row: a bitmap of the positions in shared memory and a scan over its words'
// counts; each thread then writes the positions of its words out in order.  Where a position is repeated (the clamp
// makes that of lists with positions out of range), the entries are counted per distinct position instead, and every
// entry takes the next place of its position: linear in T however often one is repeated (moving each position up by a
// walk over a side list of the repeated entries was quadratic: 16384 entries over 100 positions 4225 us, now 38; distinct ones 44 and 45).
// Takes the place of a clamp, a library sort with its index arrays and two conversions (40 us for 32 rows x 400).
constexpr int kSortThreads = 1024;
constexpr int kSortMaxT = 16384, kSortMaxLast = 1 << 20;

// exclusive prefix of v over the block's 1024 threads
__device__ __forceinline__ int sort_block_scan(int v, int* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += n;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int ws = warp_sums[lane];
    const int own = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += n;
    }
    warp_sums[lane] = ws - own;
  }
  __syncthreads();
  return warp_sums[warp] + inc - v;
}

__global__ void __launch_bounds__(kSortThreads)
vertical_sort_kernel(const int64_t* __restrict__ idx, int T, int last, int32_t* __restrict__ asc) {
  extern __shared__ uint32_t s_bits[];                     // [words], then an entry count per distinct position [T]
  const int words = last / 32 + 1;
  int* places = reinterpret_cast<int*>(s_bits + words);
  __shared__ int first_rank[kSortThreads];                 // distinct positions below each thread's words
  __shared__ int warp_sums[32];
  const int tid = threadIdx.x;
  const int64_t* src = idx + (int64_t)blockIdx.x * T;
  int32_t* dst = asc + (int64_t)blockIdx.x * T;
  auto position = [&](int i) {
    const int64_t raw = __ldg(src + i);
    return raw < 0 ? 0 : raw > last ? last : (int)raw;
  };
  for (int i = tid; i < words; i += kSortThreads) s_bits[i] = 0u;
  __syncthreads();
  int repeated = 0;
#pragma unroll 4
  for (int i = tid; i < T; i += kSortThreads) {
    const int v = position(i);
    const uint32_t bit = 1u << (v & 31);
    repeated |= (atomicOr(&s_bits[v >> 5], bit) & bit) != 0u;
  }
  repeated = __syncthreads_or(repeated);
  const int per = (words + kSortThreads - 1) / kSortThreads, w0 = min(words, tid * per), w1 = min(words, w0 + per);
  int count = 0;
  for (int w = w0; w < w1; ++w) count += __popc(s_bits[w]);
  int pos = sort_block_scan(count, warp_sums);
  if (!repeated) {
    for (int w = w0; w < w1; ++w)
      for (uint32_t m = s_bits[w]; m != 0u; m &= m - 1u) dst[pos++] = w * 32 + __ffs(m) - 1;
    return;
  }
  first_rank[tid] = pos;
  for (int i = tid; i < T; i += kSortThreads) places[i] = 0;
  __syncthreads();
  auto rank = [&](int v) {                                 // distinct positions below v
    const int word = v >> 5, owner = word / per;
    int r = first_rank[owner] + __popc(s_bits[word] & ((1u << (v & 31)) - 1u));
    for (int w = owner * per; w < word; ++w) r += __popc(s_bits[w]);
    return r;
  };
  for (int i = tid; i < T; i += kSortThreads) atomicAdd(&places[rank(position(i))], 1);
  __syncthreads();
  const int tper = (T + kSortThreads - 1) / kSortThreads, t0 = min(T, tid * tper), t1 = min(T, t0 + tper);
  int entries = 0;
  for (int i = t0; i < t1; ++i) entries += places[i];
  int base = sort_block_scan(entries, warp_sums);
  for (int i = t0; i < t1; ++i) { const int n = places[i]; places[i] = base; base += n; }
  __syncthreads();
  for (int i = tid; i < T; i += kSortThreads) {
    const int v = position(i);
    dst[atomicAdd(&places[rank(v)], 1)] = v;               // equal entries: any order is the same list
  }
}

}  // namespace hq

namespace hq {
int prefill_tc_launch(const hq_prefill_args* a, bool v_rows, cudaStream_t st);
int prefill_tc_prepare_v(const void* v, int64_t sb, int64_t sh, int64_t sn, int B, int H_KV, int N, void* v_t, cudaStream_t st);
int prefill_tc_prepare_vertical(bool rows, const int32_t* vasc, int B, int H_Q, int H_KV, int N, int T, const void* k_bf, const void* v,
                                int64_t v_sb, int64_t v_sh, int64_t v_sn, void* xk, void* xvt, cudaStream_t st);
int prefill_tc_prepare_v_fp8(const void* v, int64_t sb, int64_t sh, int64_t sn, int B, int H_KV, int N, void* v_t8, float* v_scale,
                             void* amax_scratch, cudaStream_t st);
int prefill_tc_gather_v_fp8(const int32_t* vasc, int B, int H_Q, int H_KV, int N, int T, const void* v, int64_t v_sb, int64_t v_sh,
                            int64_t v_sn, const float* v_scale, void* xvt8, cudaStream_t st);
}

extern "C" int hq_prefill_vertical_gather_v_fp8(const int32_t* vidx_asc, int B, int H_Q, int H_KV, int N, int T, const void* v,
                                                int64_t v_sb, int64_t v_sh, int64_t v_sn, const float* v_scale, void* vert_vt8,
                                                void* stream) {
  using namespace hq;
  HQ_REQUIRE(vidx_asc && v && v_scale && vert_vt8 && B > 0 && H_Q > 0 && H_KV > 0 && N > 0 && T > 0 && H_Q % H_KV == 0, HQ_ERR_INVALID,
             "hq_prefill_vertical_gather_v_fp8: bad arguments");
  HQ_REQUIRE(aligned16(v) && aligned16(vert_vt8) && v_sb % 8 == 0 && v_sh % 8 == 0 && v_sn % 8 == 0, HQ_ERR_ALIGNMENT,
             "hq_prefill_vertical_gather_v_fp8: rows must be 16-byte aligned");
  return prefill_tc_gather_v_fp8(vidx_asc, B, H_Q, H_KV, N, T, v, v_sb, v_sh, v_sn, v_scale, vert_vt8, (cudaStream_t)stream);
}

extern "C" int hq_prefill_quant_v_fp8(const void* v, int64_t v_sb, int64_t v_sh, int64_t v_sn, int B, int H_KV, int N,
                                      void* v_t8, float* v_scale, void* amax_scratch, void* stream) {
  using namespace hq;
  HQ_REQUIRE(v && v_t8 && v_scale && amax_scratch && B > 0 && H_KV > 0 && N > 0, HQ_ERR_INVALID, "hq_prefill_quant_v_fp8: bad arguments");
  HQ_REQUIRE(aligned16(v) && aligned16(v_t8) && v_sb % 8 == 0 && v_sh % 8 == 0 && v_sn % 8 == 0, HQ_ERR_ALIGNMENT,
             "hq_prefill_quant_v_fp8: rows must be 16-byte aligned");
  return prefill_tc_prepare_v_fp8(v, v_sb, v_sh, v_sn, B, H_KV, N, v_t8, v_scale, amax_scratch, (cudaStream_t)stream);
}

extern "C" int hq_prefill_transpose_v(const void* v, int64_t v_sb, int64_t v_sh, int64_t v_sn, int B, int H_KV, int N,
                                      void* v_t, void* stream) {
  using namespace hq;
  HQ_REQUIRE(v && v_t && B > 0 && H_KV > 0 && N > 0, HQ_ERR_INVALID, "hq_prefill_transpose_v: bad arguments");
  HQ_REQUIRE(aligned16(v) && aligned16(v_t) && v_sb % 8 == 0 && v_sh % 8 == 0 && v_sn % 8 == 0, HQ_ERR_ALIGNMENT,
             "hq_prefill_transpose_v: rows must be 16-byte aligned");
  return prefill_tc_prepare_v(v, v_sb, v_sh, v_sn, B, H_KV, N, v_t, (cudaStream_t)stream);
}

extern "C" int hq_prefill_vertical_sort(const int64_t* vidx, int rows, int T, int last, int32_t* vidx_asc, void* stream) {
  using namespace hq;
  HQ_REQUIRE(rows >= 0 && T >= 0 && last >= 0, HQ_ERR_INVALID, "hq_prefill_vertical_sort: bad sizes");
  HQ_REQUIRE(T <= kSortMaxT && last < kSortMaxLast, HQ_ERR_UNSUPPORTED, "hq_prefill_vertical_sort: T %d > %d or position %d >= %d",
             T, kSortMaxT, last, kSortMaxLast);
  if (rows == 0 || T == 0) return HQ_OK;
  HQ_REQUIRE(vidx && vidx_asc, HQ_ERR_INVALID, "hq_prefill_vertical_sort: null pointer");
  static thread_local int attr_dev = -1;
  int dev = 0;
  HQ_CUDA(cudaGetDevice(&dev));
  if (attr_dev != dev) {
    HQ_CUDA(cudaFuncSetAttribute(vertical_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSortMaxLast / 8 + kSortMaxT * 4));
    attr_dev = dev;
  }
  const size_t smem = (size_t)(last / 32 + 1) * 4 + (size_t)T * 4;
  vertical_sort_kernel<<<rows, kSortThreads, smem, (cudaStream_t)stream>>>(vidx, T, last, vidx_asc);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

static int vertical_prepare(bool rows, const int32_t* vidx_asc, int B, int H_Q, int H_KV, int N, int window, int T,
                            const void* k_bf, const void* v, int64_t v_sb, int64_t v_sh, int64_t v_sn,
                            const float* k_scale, void* vert_k, void* vert_vt, float* k_bias,
                            int32_t* nv_valid, void* stream) {
  using namespace hq;
  HQ_REQUIRE(B > 0 && H_Q > 0 && H_KV > 0 && N > 0 && T >= 0 && window >= 0 && H_Q % H_KV == 0, HQ_ERR_INVALID,
             "hq_prefill_vertical_prepare: bad sizes");
  HQ_REQUIRE(k_scale && k_bias, HQ_ERR_INVALID, "hq_prefill_vertical_prepare: k_scale / k_bias missing");
  HQ_REQUIRE(T == 0 || (vidx_asc && k_bf && v && vert_k && vert_vt && nv_valid), HQ_ERR_INVALID,
             "hq_prefill_vertical_prepare: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const int nqb = (N + 127) / 128, Npad = (N + 63) / 64 * 64;
  // (b, hq) -> (b, hq / R) as one division of the flat index needs R to divide H_Q, checked above
  vertical_meta_kernel<<<dim3((Npad + kMetaKeys - 1) / kMetaKeys, B * H_Q), 256, 0, st>>>(vidx_asc, T, N, Npad, window, nqb, H_Q / H_KV, k_scale, k_bias, nv_valid);
  HQ_CUDA(cudaGetLastError());
  if (T == 0) return HQ_OK;
  HQ_REQUIRE(aligned16(v) && aligned16(k_bf) && aligned16(vert_k) && aligned16(vert_vt) && v_sb % 8 == 0 &&
                 v_sh % 8 == 0 && v_sn % 8 == 0, HQ_ERR_ALIGNMENT, "hq_prefill_vertical_prepare: rows must be 16-byte aligned");
  return prefill_tc_prepare_vertical(rows, vidx_asc, B, H_Q, H_KV, N, T, k_bf, v, v_sb, v_sh, v_sn, vert_k, vert_vt, st);
}

extern "C" int hq_prefill_vertical_prepare(const int32_t* vidx_asc, int B, int H_Q, int H_KV, int N, int window, int T,
                                           const void* k_bf, const void* v, int64_t v_sb, int64_t v_sh, int64_t v_sn,
                                           const float* k_scale, void* vert_k, void* vert_vt, float* k_bias,
                                           int32_t* nv_valid, void* stream) {
  return vertical_prepare(false, vidx_asc, B, H_Q, H_KV, N, window, T, k_bf, v, v_sb, v_sh, v_sn, k_scale, vert_k, vert_vt, k_bias,
                          nv_valid, stream);
}

extern "C" int hq_prefill_vertical_prepare_rows(const int32_t* vidx_asc, int B, int H_Q, int H_KV, int N, int window, int T,
                                           const void* k_bf, const void* v, int64_t v_sb, int64_t v_sh, int64_t v_sn,
                                           const float* k_scale, void* vert_k, void* vert_v, float* k_bias,
                                           int32_t* nv_valid, void* stream) {
  return vertical_prepare(true, vidx_asc, B, H_Q, H_KV, N, window, T, k_bf, v, v_sb, v_sh, v_sn, k_scale, vert_k, vert_v, k_bias,
                          nv_valid, stream);
}

extern "C" int hq_prefill_hybrid(const hq_prefill_args* a, void* stream) {
  using namespace hq;
  HQ_REQUIRE(a != nullptr, HQ_ERR_INVALID, "hq_prefill_hybrid: null args");
  // the struct as it was before V's strides is taken too (its flag word was reserved and is not read)
  const bool short_args = a->struct_bytes == (int32_t)offsetof(hq_prefill_args, v_sb);
  HQ_REQUIRE(short_args || a->struct_bytes == (int32_t)sizeof(hq_prefill_args), HQ_ERR_INVALID, "hq_prefill_hybrid: struct_bytes %d != %d",
             a->struct_bytes, (int)sizeof(hq_prefill_args));
  const bool v_rows = !short_args && a->v_rows != 0 && !a->pv_fp8;
  HQ_REQUIRE(a->head_dim == 128, HQ_ERR_UNSUPPORTED, "hq_prefill_hybrid: head_dim %d (only 128 is built)", a->head_dim);
  HQ_REQUIRE(a->B > 0 && a->H_Q > 0 && a->H_KV > 0 && a->N > 0 && a->H_Q % a->H_KV == 0 && a->window >= 0 && a->T >= 0,
             HQ_ERR_INVALID, "hq_prefill_hybrid: bad sizes");
  HQ_REQUIRE(a->q_i8 && a->q_bf && a->q_scale && a->k_i8 && a->k_bf && a->k_scale && a->k_bias && a->out && a->status,
             HQ_ERR_INVALID, "hq_prefill_hybrid: null pointer");
  if (a->pv_fp8) {
    HQ_REQUIRE(a->v_t8 && a->v_scale8 && aligned16(a->v_t8), HQ_ERR_INVALID, "hq_prefill_hybrid: FP8 P V needs v_t8 (16-byte aligned) and v_scale8");
    HQ_REQUIRE(a->T == 0 || (a->vert_vt8 && aligned16(a->vert_vt8)), HQ_ERR_INVALID, "hq_prefill_hybrid: FP8 P V with vertical lines needs vert_vt8");
  } else {
    HQ_REQUIRE(a->v_t != nullptr, HQ_ERR_INVALID, "hq_prefill_hybrid: v_t is null");
  }
  HQ_REQUIRE(a->T == 0 || (a->vert_k && (a->vert_vt || a->pv_fp8) && a->nv_valid), HQ_ERR_INVALID,
             "hq_prefill_hybrid: vertical arguments missing");
  HQ_REQUIRE(aligned16(a->q_i8) && aligned16(a->q_bf) && aligned16(a->k_i8) && aligned16(a->k_bf) && (a->pv_fp8 || aligned16(a->v_t)) &&
                 aligned16(a->k_scale) && aligned16(a->k_bias) && aligned16(a->out) && a->o_sn % 8 == 0 && a->o_sh % 8 == 0 && a->o_sb % 8 == 0,
             HQ_ERR_ALIGNMENT, "hq_prefill_hybrid: operand rows must be 16-byte aligned");
  HQ_REQUIRE(a->out_dtype == HQ_BF16 || a->out_dtype == HQ_F16 || a->out_dtype == HQ_F32, HQ_ERR_UNSUPPORTED,
             "hq_prefill_hybrid: out_dtype %d", a->out_dtype);
  if (v_rows) {
    HQ_REQUIRE(a->v_sb > 0 && a->v_sh > 0 && a->v_sn > 0 && a->v_sb % 8 == 0 && a->v_sh % 8 == 0 && a->v_sn % 8 == 0, HQ_ERR_ALIGNMENT,
               "hq_prefill_hybrid: rows of v must be 16-byte aligned");
    HQ_REQUIRE(a->T == 0 || aligned16(a->vert_vt), HQ_ERR_ALIGNMENT, "hq_prefill_hybrid: vert_vt must be 16-byte aligned");
  }
  return prefill_tc_launch(a, v_rows, (cudaStream_t)stream);
}
