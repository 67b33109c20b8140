// Vertical-line identification: pooled-query scores over the candidate keys and
// an exact, deterministic top-k.
//
// Scores kernel — HBM-bound (one read of the candidate keys, 256 B per token per
// kv-head; 4 B per (token, query head) written).  scores^T[token, head] =
// K[token, :] . qbar[head, :] is computed with mma.sync bf16 (tokens on the M
// axis, the kv-group's query heads on the N axis), the pooled query being split
// into a bf16 high and low part so that an unrounded fp32 mean keeps ~16 bits.
// K fragments come straight from global memory as 16-byte loads; the channel
// axis is permuted consistently on both operands so that no shuffle is needed.
//
// Top-k kernels — latency-bound: a row's keys are read once, eight loads a thread in flight, and kept in shared memory
// where they fit; three-pass radix select of the k-th largest key with a scan over the bins, order-preserving
// compaction (ties go to the lower index; it is also the ascending list), bitonic sort of the selected (key, ~index)
// pairs, the short distances inside warps.  topk_kernel: one CTA per row.  topk_cluster_kernel: a cluster of four or
// eight CTAs per row, for long rows of calls that leave SMs idle otherwise (the rule is in hq_topk_form.h).
#include <cooperative_groups.h>
#include "hq_common.cuh"
#include "hq_topk_form.h"

namespace hq {

// ------------------------------------------------------------------ pooling
// `group` > 1: output head h is the mean of the input heads h group .. h group + group - 1, taken per token and rounded
// to the input dtype (what a 16-bit mean over the head axis gives) before the tokens are pooled.
//
// Latency-bound: a few hundred KB in all.  One block per (output head, 16 channels): 256 threads fetch 128 tokens of
// all the group's heads at once, 16 bytes a load where the rows are aligned, and leave the per-token means in shared
// memory, where one thread per channel adds them up in token order (the order of the sum decides ties of the
// selection, so it stays).  One thread per channel with a dependent load per token and head took 93 us for 8 kv-heads
// x 4 heads x 128 tokens.
constexpr int kPoolRows = 128;    // tokens per trip
constexpr int kPoolCh = 16;       // channels per block
constexpr int kPoolThreads = kPoolRows * kPoolCh / 8;

template <typename T>
__device__ __forceinline__ void load8(const T* p, bool vec, float (&v)[8]) {
  if (vec) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(p));
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = load_as_float<T>(e + j);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = load_as_float<T>(p + j);
  }
}

template <typename T>
__global__ void __launch_bounds__(kPoolThreads)
pool_query_kernel(const T* __restrict__ q, int64_t sb, int64_t sh, int64_t sn, int H_Q, int n_q,
                  int tail_len, int round_mode /*-1 none, else dtype*/, int group, int group_dtype,
                  int vec /* rows are 16-byte aligned */, float* __restrict__ pooled) {
  __shared__ float s_mean[kPoolRows][kPoolCh + 1];
  const int bh = blockIdx.x, b = bh / H_Q, h = bh - b * H_Q, d0 = blockIdx.y * kPoolCh;
  const int tid = threadIdx.x, r0 = tid >> 1, c = (tid & 1) * 8;
  const T* base = q + b * sb + (int64_t)h * group * sh + (int64_t)(n_q - tail_len) * sn + d0 + c;
  float acc = 0.f;
  for (int i0 = 0; i0 < tail_len; i0 += kPoolRows) {
    const int i = i0 + r0;
    if (i < tail_len) {
      float m[8];
      if (group <= 1) {
        load8<T>(base + (int64_t)i * sn, vec, m);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) m[j] = 0.f;
#pragma unroll 4
        for (int r = 0; r < group; ++r) {
          float v[8];
          load8<T>(base + r * sh + (int64_t)i * sn, vec, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) m[j] += v[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) m[j] = out_round(m[j] / (float)group, group_dtype);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s_mean[r0][c + j] = m[j];
    }
    __syncthreads();
    if (tid < kPoolCh) {
      const int rows = min(kPoolRows, tail_len - i0);
#pragma unroll 8
      for (int r = 0; r < rows; ++r) acc += s_mean[r][tid];
    }
    __syncthreads();
  }
  if (tid < kPoolCh) {
    float m = acc / (float)tail_len;
    if (round_mode >= 0) m = out_round(m, round_mode);
    pooled[(int64_t)bh * 128 + d0 + tid] = m;
  }
}

// ------------------------------------------------------------------ scores
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if (kBf16) { __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi); return *reinterpret_cast<uint32_t*>(&h); }
  __half2 h = __floats2half2_rn(lo, hi); return *reinterpret_cast<uint32_t*>(&h);
}
template <bool kBf16>
__device__ __forceinline__ float round16(float v) {
  return kBf16 ? __bfloat162float(__float2bfloat16_rn(v)) : __half2float(__float2half_rn(v));
}

constexpr int kScoreWarps = 8;

// grid (chunks, B*H_KV).  K rows 128 elements wide, 16-bit dtype.
template <bool kBf16, int NT>
__global__ void __launch_bounds__(kScoreWarps * 32)
vertical_scores_kernel(const uint16_t* __restrict__ k, int64_t ksb, int64_t ksh, int64_t ksn, int H_KV, int R, int n_cand,
                       const float* __restrict__ pooled, int round_scores, float* __restrict__ scores) {
  const int bhk = blockIdx.y, b = bhk / H_KV, hk = bhk - b * H_KV;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  // B fragments of qbar (hi and lo parts).  16-byte chunk j = 4 w + t of a key row
  // holds channels 8 j .. 8 j + 7; MMA chunk 2 w takes channels (0,1 | 2,3) of it,
  // chunk 2 w + 1 takes (4,5 | 6,7).
  uint32_t qh[NT][8][2], ql[NT][8][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int hd = nt * 8 + g;
    const float* qrow = pooled + ((int64_t)(b * H_KV + hk) * R + hd) * 128;
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int ch = 8 * (4 * (c >> 1) + t) + 4 * (c & 1) + 2 * r;
        float x0 = 0.f, x1 = 0.f;
        if (hd < R) { x0 = qrow[ch]; x1 = qrow[ch + 1]; }
        const float h0 = round16<kBf16>(x0), h1 = round16<kBf16>(x1);
        qh[nt][c][r] = pack2<kBf16>(h0, h1);
        ql[nt][c][r] = pack2<kBf16>(x0 - h0, x1 - h1);
      }
  }
  const uint16_t* kbase = k + b * ksb + hk * ksh;
  const int tiles = (n_cand + 15) / 16;
  const int tile_stride = gridDim.x * kScoreWarps;
  for (int tile = blockIdx.x * kScoreWarps + warp; tile < tiles; tile += tile_stride) {
    const int tokA = tile * 16 + g, tokB = tokA + 8;
    const bool okA = tokA < n_cand, okB = tokB < n_cand;
    uint4 ka[4], kb[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      ka[w] = okA ? __ldg(reinterpret_cast<const uint4*>(kbase + (int64_t)tokA * ksn + (4 * w + t) * 8)) : make_uint4(0, 0, 0, 0);
      kb[w] = okB ? __ldg(reinterpret_cast<const uint4*>(kbase + (int64_t)tokB * ksn + (4 * w + t) * 8)) : make_uint4(0, 0, 0, 0);
    }
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if (kBf16) {
          mma_bf16(s[nt], ka[w].x, kb[w].x, ka[w].y, kb[w].y, ql[nt][2 * w][0], ql[nt][2 * w][1]);
          mma_bf16(s[nt], ka[w].z, kb[w].z, ka[w].w, kb[w].w, ql[nt][2 * w + 1][0], ql[nt][2 * w + 1][1]);
          mma_bf16(s[nt], ka[w].x, kb[w].x, ka[w].y, kb[w].y, qh[nt][2 * w][0], qh[nt][2 * w][1]);
          mma_bf16(s[nt], ka[w].z, kb[w].z, ka[w].w, kb[w].w, qh[nt][2 * w + 1][0], qh[nt][2 * w + 1][1]);
        } else {
          mma_f16(s[nt], ka[w].x, kb[w].x, ka[w].y, kb[w].y, ql[nt][2 * w][0], ql[nt][2 * w][1]);
          mma_f16(s[nt], ka[w].z, kb[w].z, ka[w].w, kb[w].w, ql[nt][2 * w + 1][0], ql[nt][2 * w + 1][1]);
          mma_f16(s[nt], ka[w].x, kb[w].x, ka[w].y, kb[w].y, qh[nt][2 * w][0], qh[nt][2 * w][1]);
          mma_f16(s[nt], ka[w].z, kb[w].z, ka[w].w, kb[w].w, qh[nt][2 * w + 1][0], qh[nt][2 * w + 1][1]);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int hd = nt * 8 + 2 * t + j;
        if (hd < R) {
          float* srow = scores + ((int64_t)(b * H_KV + hk) * R + hd) * n_cand;
          float vA = s[nt][j], vB = s[nt][2 + j];
          if (round_scores) { vA = round16<kBf16>(vA); vB = round16<kBf16>(vB); }
          if (okA) srow[tokA] = vA;
          if (okB) srow[tokB] = vB;
        }
      }
    }
  }
}

// ------------------------------------------------------------------- top-k
__device__ __forceinline__ uint32_t orderable(float f) {
  uint32_t u = (f == 0.0f) ? 0u : __float_as_uint(f);   // -0.0 and +0.0 compare equal, as in torch.topk
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int kTopkThreads = 1024;

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
  // 1024 threads; returns exclusive prefix of v over the block, total in `total`
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += n;
  }
  __syncthreads();               // protect warp_sums reuse
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int ws = warp_sums[lane];
    int winc = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += n;
    }
    warp_sums[lane] = winc - ws;          // exclusive prefix of warp totals
    if (lane == 31) warp_sums[32] = winc;   // block total
  }
  __syncthreads();
  total = warp_sums[32];
  return warp_sums[warp] + inc - v;
}

// 64 entries per warp (lane l: base + l and base + 32 + l): the compare-exchange steps of a bitonic stage `size` whose
// distance is at most `first` (32 or less), without leaving registers
__device__ __forceinline__ void bitonic_in_warp(unsigned long long& a, unsigned long long& c, int base, int lane, int size, int first) {
  if (first >= 32) {
    const bool desc = ((base + lane) & size) == 0;
    if ((a < c) == desc) { const unsigned long long x = a; a = c; c = x; }
    first = 16;
  }
  const bool da = ((base + lane) & size) == 0, dc = ((base + 32 + lane) & size) == 0;
  for (int strd = first; strd > 0; strd >>= 1) {
    const unsigned long long pa = __shfl_xor_sync(0xffffffffu, a, strd), pc = __shfl_xor_sync(0xffffffffu, c, strd);
    const bool lower = (lane & strd) == 0;
    a = ((a > pa) == (lower == da)) ? a : pa;
    c = ((c > pc) == (lower == dc)) ? c : pc;
  }
}

// kCached: the row's keys stay in shared memory after the first pass (with the list of kpad entries they have to fit 224 KB:
// 55 thousand candidates with a list of 64, 22 thousand with 16384); longer rows read them again from L2.
template <bool kCached>
__global__ void __launch_bounds__(kTopkThreads)
topk_kernel(const float* __restrict__ scores, int64_t stride, int n, int k, int kpad,
            int64_t* __restrict__ idx_desc, int32_t* __restrict__ idx_asc) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  unsigned long long* sel = reinterpret_cast<unsigned long long*>(smem_raw);   // [kpad]
  int* hist = reinterpret_cast<int*>(sel + kpad);                              // [kTopkBins]
  uint32_t* keys = reinterpret_cast<uint32_t*>(hist + kTopkBins);              // [n] if kCached
  __shared__ int warp_sums[33];
  __shared__ uint32_t s_bin;
  __shared__ int s_remaining;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* row = scores + (int64_t)blockIdx.x * stride;
  auto key_at = [&](int i) -> uint32_t { return kCached ? keys[i] : orderable(__ldg(row + i)); };

  // ---- radix select: find key T of the k-th largest element (digits of 11, 11 and 10 bits)
  uint32_t prefix = 0, mask = 0;
  int remaining = k;   // rank (1-based from the top) within the current candidate set
#pragma unroll 1
  for (int pass = 0; pass < 3; ++pass) {
    const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
    const uint32_t digits = pass == 2 ? 1023u : 2047u;
    for (int x = tid; x < kTopkBins; x += kTopkThreads) hist[x] = 0;
    __syncthreads();
    for (int i0 = tid; i0 < n; i0 += 8 * kTopkThreads) {
      uint32_t key[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j * kTopkThreads;
        key[j] = i < n ? ((kCached && pass > 0) ? keys[i] : orderable(__ldg(row + i))) : 0u;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j * kTopkThreads;
        if (i < n) {
          if (kCached && pass == 0) keys[i] = key[j];
          if ((key[j] & mask) == prefix) atomicAdd(&hist[(key[j] >> shift) & digits], 1);
        }
      }
    }
    __syncthreads();
    // the digit that holds the wanted rank: thread t has the bins kTopkBins - 1 - 2 t and the one below it
    const int h0 = hist[kTopkBins - 1 - 2 * tid], h1 = hist[kTopkBins - 2 - 2 * tid];
    int total;
    const int above = block_exclusive_scan(h0 + h1, warp_sums, total);
    if (above < remaining && remaining <= above + h0 + h1) {
      const bool first = remaining <= above + h0;
      s_bin = (uint32_t)(kTopkBins - 1 - 2 * tid - (first ? 0 : 1));
      s_remaining = remaining - above - (first ? 0 : h0);
    }
    __syncthreads();
    prefix |= s_bin << shift;
    remaining = s_remaining;
    mask |= digits << shift;
  }
  const uint32_t T = prefix;        // threshold key
  const int need_eq = remaining;    // how many elements equal to T to take (lowest indices first)

  // ---- order-preserving compaction into sel[]: warp w owns one contiguous range of the row, counts what it has and
  // writes once the warps before it are known; the order of the list is the ascending index list
  const int seg = ((n + 31) / 32 + 31) & ~31;
  const int s0 = min(warp * seg, n), s1 = min(s0 + seg, n);
  int gt = 0, eq = 0;
  for (int i = s0 + lane; i < s1; i += 32) {
    const uint32_t key = key_at(i);
    gt += key > T;
    eq += key == T;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gt += __shfl_xor_sync(0xffffffffu, gt, o);
    eq += __shfl_xor_sync(0xffffffffu, eq, o);
  }
  int total;
  const int eq_scan = block_exclusive_scan(lane == 0 ? eq : 0, warp_sums, total);
  int eq_seen = __shfl_sync(0xffffffffu, eq_scan, 0);           // == T elements of the warps before
  const int mine = gt + max(0, min(eq, need_eq - eq_seen));
  const int out_scan = block_exclusive_scan(lane == 0 ? mine : 0, warp_sums, total);
  int out_pos = __shfl_sync(0xffffffffu, out_scan, 0);
  if (mine > 0) {
    const uint32_t lt = (1u << lane) - 1u;
    for (int i0 = s0; i0 < s1; i0 += 32) {
      const int i = i0 + lane;
      const uint32_t key = i < s1 ? key_at(i) : 0u;
      const bool is_eq = i < s1 && key == T;
      const uint32_t eqs = __ballot_sync(0xffffffffu, is_eq);
      const bool take = i < s1 && (key > T || (is_eq && eq_seen + __popc(eqs & lt) < need_eq));
      const uint32_t takes = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int pos = out_pos + __popc(takes & lt);
        sel[pos] = ((unsigned long long)key << 32) | (uint32_t)(~(uint32_t)i);
        if (idx_asc) idx_asc[(int64_t)blockIdx.x * k + pos] = i;
      }
      eq_seen += __popc(eqs);
      out_pos += __popc(takes);
    }
  }
  for (int i = k + tid; i < kpad; i += kTopkThreads) sel[i] = 0ull;   // smaller than any real entry
  __syncthreads();

  // ---- bitonic sort, descending: distances of 64 and more through shared memory, the rest inside warps
  for (int base = warp * 64; base < kpad; base += (kTopkThreads / 32) * 64) {
    unsigned long long a = sel[base + lane], c = sel[base + 32 + lane];
    for (int size = 2; size <= 64; size <<= 1) bitonic_in_warp(a, c, base, lane, size, size >> 1);
    sel[base + lane] = a; sel[base + 32 + lane] = c;
  }
  __syncthreads();
  for (int size = 128; size <= kpad; size <<= 1) {
    for (int strd = size >> 1; strd >= 64; strd >>= 1) {
      for (int x = tid; x < (kpad >> 1); x += kTopkThreads) {
        const int lo = 2 * x - (x & (strd - 1));
        const int hi = lo + strd;
        const bool desc = ((lo & size) == 0);
        const unsigned long long a = sel[lo], b2 = sel[hi];
        if ((a < b2) == desc) { sel[lo] = b2; sel[hi] = a; }
      }
      __syncthreads();
    }
    for (int base = warp * 64; base < kpad; base += (kTopkThreads / 32) * 64) {
      unsigned long long a = sel[base + lane], c = sel[base + 32 + lane];
      bitonic_in_warp(a, c, base, lane, size, 32);
      sel[base + lane] = a; sel[base + 32 + lane] = c;
    }
    __syncthreads();
  }
  for (int i = tid; i < k; i += kTopkThreads)
    idx_desc[(int64_t)blockIdx.x * k + i] = (int64_t)(~(uint32_t)(sel[i] & 0xFFFFFFFFull));
}

// ---- the same for long rows
constexpr int kSliceThreads = 512, kSliceWarps = kSliceThreads / 32;

__device__ __forceinline__ int warp_inclusive_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

__device__ __forceinline__ int slice_exclusive_scan(int v, int* warp_sums) {
  // kSliceThreads threads; returns the exclusive prefix of v over the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int inc = warp_inclusive_scan(v);
  __syncthreads();               // protect warp_sums reuse
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  int before = lane < warp ? warp_sums[lane] : 0;               // kSliceWarps <= 32
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  return before + inc - v;
}

// A row is taken by a cluster of blocks, each with a contiguous slice of it.  Radix select: every block counts its slice's
// digits, adds up the cluster's counters over distributed shared memory and finds the same digit; then it keeps what it has
// above the threshold (and its share of what equals it) in index order, sorts that, and an entry's place in the whole list
// is its own plus, for every other block, the entries above it there (a binary search).  8 rows of 32K candidates: 36 us
// with a block each (counting 20 K clocks, compaction 14 K, the sort 18 K of 74 K), 19 us this way.
// kCached: the slice's keys stay in shared memory after the first pass, where seg keys, selcap entries and the counters fit 224 KB
// (53 thousand keys with a list of 64, 36 thousand with 8192, 20 thousand with 16384); longer slices are read again.
template <bool kCached>
__global__ void __launch_bounds__(kSliceThreads)
topk_cluster_kernel(const float* __restrict__ scores, int64_t stride, int n, int k, int seg, int selcap,
            int64_t* __restrict__ idx_desc, int32_t* __restrict__ idx_asc) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  unsigned long long* sel = reinterpret_cast<unsigned long long*>(smem_raw);   // [selcap]
  int* hist = reinterpret_cast<int*>(sel + selcap);                            // [2][kTopkBins]
  uint32_t* keys = reinterpret_cast<uint32_t*>(hist + 2 * kTopkBins);          // [seg] if kCached
  __shared__ int warp_sums[kSliceWarps];
  __shared__ __align__(8) int s_sums[2][kTopkBins / 32];
  __shared__ uint32_t s_bin;
  __shared__ int s_remaining;
  __shared__ int s_count[2];                                                   // above T, equal to T
  __shared__ int s_off[kTopkCluster + 1];                                      // where the blocks' entries begin in the ascending list
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int blocks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r = blockIdx.x / blocks;
  const int first = min(rank * seg, n), m = min(first + seg, n) - first;       // the slice: first .. first + m
  const float* row = scores + r * stride + first;
  auto key_at = [&](int i) -> uint32_t { return kCached ? keys[i] : orderable(__ldg(row + i)); };

  // ---- radix select: find key T of the k-th largest element (digits of 11, 11 and 10 bits)
  uint32_t prefix = 0, mask = 0;
  int remaining = k;   // rank (1-based from the top) within the current candidate set
#pragma unroll 1
  for (int pass = 0; pass < 3; ++pass) {
    const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
    const uint32_t digits = pass == 2 ? 1023u : 2047u;
    // the counters of two passes ago: the cluster has met since their last reader
    int* h = hist + (pass & 1) * kTopkBins;
    *reinterpret_cast<int4*>(h + 4 * tid) = make_int4(0, 0, 0, 0);
    __syncthreads();
    for (int i0 = tid; i0 < m; i0 += 8 * kSliceThreads) {
      uint32_t key[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j * kSliceThreads;
        key[j] = i < m ? ((kCached && pass > 0) ? keys[i] : orderable(__ldg(row + i))) : 0u;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j * kSliceThreads;
        if (i < m) {
          if (kCached && pass == 0) keys[i] = key[j];
          if ((key[j] & mask) == prefix) atomicAdd(&h[(key[j] >> shift) & digits], 1);
        }
      }
    }
    __syncthreads();
    // sums of 32 counters, so that the cluster's are first added up 64 sums and then 32 counters at a time (all 2048 of
    // every block: 4400 clocks a pass at 8 blocks, now 1700)
    int* sums = s_sums[pass & 1];
    for (int x = warp; x < kTopkBins / 32; x += kSliceWarps) {
      const int v = __reduce_add_sync(0xffffffffu, h[32 * x + lane]);
      if (lane == 0) sums[x] = v;
    }
    cluster.sync();
    // the digit that holds the wanted rank: the group of bins (lane l has groups 63 - 2 l and 62 - 2 l), then the bin
    if (warp == 0) {
      int2 c = make_int2(0, 0);
#pragma unroll
      for (int b = 0; b < kTopkCluster; ++b) {                   // all loads in flight together
        if (b < blocks) {
          const int2 x = *reinterpret_cast<const int2*>(cluster.map_shared_rank(sums, b) + 62 - 2 * lane);
          c.x += x.x; c.y += x.y;
        }
      }
      int upto = warp_inclusive_scan(c.x + c.y);
      int above = upto - c.x - c.y;
      const int at = __ffs(__ballot_sync(0xffffffffu, above < remaining && remaining <= upto)) - 1;
      const bool high = remaining <= above + c.y;
      const int group = __shfl_sync(0xffffffffu, high ? 63 - 2 * lane : 62 - 2 * lane, at);
      const int left = remaining - __shfl_sync(0xffffffffu, high ? above : above + c.y, at);
      int n_bin = 0;
#pragma unroll
      for (int b = 0; b < kTopkCluster; ++b)
        if (b < blocks) n_bin += cluster.map_shared_rank(h, b)[32 * group + 31 - lane];
      upto = warp_inclusive_scan(n_bin);
      if (upto - n_bin < left && left <= upto) {
        s_bin = (uint32_t)(32 * group + 31 - lane);
        s_remaining = left - (upto - n_bin);
      }
    }
    __syncthreads();
    prefix |= s_bin << shift;
    remaining = s_remaining;
    mask |= digits << shift;
  }
  const uint32_t T = prefix;        // threshold key
  const int need_eq = remaining;    // how many elements equal to T to take (lowest indices first)

  // ---- order-preserving compaction into sel[]: warp w owns one contiguous range of the slice, counts what it has and
  // writes once the warps and blocks before it are known; the order of the list is the ascending index list
  const int wseg = ((seg + kSliceWarps - 1) / kSliceWarps + 31) & ~31;
  const int s0 = min(warp * wseg, m), s1 = min(s0 + wseg, m);
  int gt = 0, eq = 0;
  for (int i = s0 + lane; i < s1; i += 32) {
    const uint32_t key = key_at(i);
    gt += key > T;
    eq += key == T;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gt += __shfl_xor_sync(0xffffffffu, gt, o);
    eq += __shfl_xor_sync(0xffffffffu, eq, o);
  }
  const int eq_scan = slice_exclusive_scan(lane == 0 ? eq : 0, warp_sums);
  const int gt_scan = slice_exclusive_scan(lane == 0 ? gt : 0, warp_sums);
  if (tid == kSliceThreads - 32) { s_count[0] = gt_scan + gt; s_count[1] = eq_scan + eq; }
  cluster.sync();
  // lane b: block b's counts, and what the blocks before it have of either and keep
  int b_gt = 0, b_eq = 0;
  if (lane < blocks) {
    const int* c = cluster.map_shared_rank(s_count, lane);
    b_gt = c[0];
    b_eq = c[1];
  }
  int gt_upto = b_gt, eq_upto = b_eq;
#pragma unroll
  for (int o = 1; o < kTopkCluster; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, gt_upto, o), y = __shfl_up_sync(0xffffffffu, eq_upto, o);
    if (lane >= o) { gt_upto += x; eq_upto += y; }
  }
  const int b_end = gt_upto + min(eq_upto, need_eq);
  if (warp == 0 && lane < blocks) s_off[lane + 1] = b_end;
  if (tid == 0) s_off[0] = 0;
  const int gt_before = __shfl_sync(0xffffffffu, gt_upto - b_gt, rank), eq_before = __shfl_sync(0xffffffffu, eq_upto - b_eq, rank);
  const int out0 = gt_before + min(eq_before, need_eq);         // the block's place in the ascending list
  int eq_seen = eq_before + __shfl_sync(0xffffffffu, eq_scan, 0);            // == T elements of the blocks and warps before
  int out_pos = gt_before + __shfl_sync(0xffffffffu, gt_scan, 0) + min(eq_seen, need_eq) - out0;
  const int kept = __shfl_sync(0xffffffffu, b_end, rank) - out0;
  if (gt + max(0, min(eq, need_eq - eq_seen)) > 0) {
    const uint32_t lt = (1u << lane) - 1u;
    for (int i0 = s0; i0 < s1; i0 += 32) {
      const int i = i0 + lane;
      const uint32_t key = i < s1 ? key_at(i) : 0u;
      const bool is_eq = i < s1 && key == T;
      const uint32_t eqs = __ballot_sync(0xffffffffu, is_eq);
      const bool take = i < s1 && (key > T || (is_eq && eq_seen + __popc(eqs & lt) < need_eq));
      const uint32_t takes = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int pos = out_pos + __popc(takes & lt);
        sel[pos] = ((unsigned long long)key << 32) | (uint32_t)(~(uint32_t)(first + i));
        if (idx_asc) idx_asc[r * k + out0 + pos] = first + i;
      }
      eq_seen += __popc(eqs);
      out_pos += __popc(takes);
    }
  }
  int kpad = 64;
  while (kpad < kept) kpad <<= 1;                               // <= selcap
  for (int i = kept + tid; i < kpad; i += kSliceThreads) sel[i] = 0ull;   // smaller than any real entry
  __syncthreads();

  // ---- bitonic sort, descending: distances of 64 and more through shared memory, the rest inside warps
  for (int base = warp * 64; base < kpad; base += kSliceWarps * 64) {
    unsigned long long a = sel[base + lane], c = sel[base + 32 + lane];
    for (int size = 2; size <= 64; size <<= 1) bitonic_in_warp(a, c, base, lane, size, size >> 1);
    sel[base + lane] = a; sel[base + 32 + lane] = c;
  }
  __syncthreads();
  for (int size = 128; size <= kpad; size <<= 1) {
    for (int strd = size >> 1; strd >= 64; strd >>= 1) {
      for (int x = tid; x < (kpad >> 1); x += kSliceThreads) {
        const int lo = 2 * x - (x & (strd - 1));
        const int hi = lo + strd;
        const bool desc = ((lo & size) == 0);
        const unsigned long long a = sel[lo], b2 = sel[hi];
        if ((a < b2) == desc) { sel[lo] = b2; sel[hi] = a; }
      }
      __syncthreads();
    }
    for (int base = warp * 64; base < kpad; base += kSliceWarps * 64) {
      unsigned long long a = sel[base + lane], c = sel[base + 32 + lane];
      bitonic_in_warp(a, c, base, lane, size, 32);
      sel[base + lane] = a; sel[base + 32 + lane] = c;
    }
    __syncthreads();
  }

  // ---- places: entries are distinct (the index is part of them), so the lists of the blocks interleave without ties.  All
  // lists are brought over where the counters and keys, which are done with, leave room for them (k up to 2048, and half a
  // slice besides where its keys were kept), and the searches of an entry run side by side.
  cluster.sync();
  if (blocks > 1 && (size_t)k * 8 <= 2 * kTopkBins * sizeof(int) + (kCached ? (size_t)seg * 4 : 0)) {
    unsigned long long* all = reinterpret_cast<unsigned long long*>(hist);
    int longest = 0;
#pragma unroll
    for (int b = 0; b < kTopkCluster; ++b)
      if (b < blocks) longest = max(longest, s_off[b + 1] - s_off[b]);
#pragma unroll 4
    for (int x = tid; x < k; x += kSliceThreads) {
      int b = 0;
#pragma unroll
      for (int c = 1; c < kTopkCluster; ++c) b += c < blocks && x >= s_off[c];
      all[x] = cluster.map_shared_rank(sel, b)[x - s_off[b]];
    }
    __syncthreads();
    int top = 1;
    while (2 * top <= longest) top <<= 1;
    for (int i = tid; i < kept; i += kSliceThreads) {
      const unsigned long long e = sel[i];
      int pos[kTopkCluster] = {};                                // entries above e in the block's list
      for (int step = top; step > 0; step >>= 1) {
#pragma unroll
        for (int b = 0; b < kTopkCluster; ++b)
          if (b < blocks) {
            const int at = s_off[b] + pos[b] + step;
            if (at <= s_off[b + 1] && all[at - 1] > e) pos[b] += step;
          }
      }
      int place = 0;
#pragma unroll
      for (int b = 0; b < kTopkCluster; ++b) place += pos[b];
      idx_desc[r * k + place] = (int64_t)(~(uint32_t)(e & 0xFFFFFFFFull));
    }
  } else {
    for (int i = tid; i < kept; i += kSliceThreads) {
      const unsigned long long e = sel[i];
      int place = i;
      for (int d = 1; d < blocks; ++d) {
        const int b = (rank + d) % blocks;
        const unsigned long long* other = cluster.map_shared_rank(sel, b);
        int lo = 0, hi = s_off[b + 1] - s_off[b];
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (other[mid] > e) lo = mid + 1; else hi = mid;
        }
        place += lo;
      }
      idx_desc[r * k + place] = (int64_t)(~(uint32_t)(e & 0xFFFFFFFFull));
    }
  }
  cluster.sync();                   // a block's lists stay until the others have read them
}

}  // namespace hq

namespace hq {
static int vertical_scores_impl(const void* q, int io_dtype, int64_t q_stride_b, int64_t q_stride_h, int64_t q_stride_n,
                                int B, int H_Q, int n_q, int tail_len, int group,
                                const void* k, int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_n,
                                int H_KV, int n_cand, int round_mean, int round_scores,
                                float* pooled, float* scores, void* stream) {
  HQ_REQUIRE(B >= 0 && H_Q > 0 && H_KV > 0 && n_q > 0 && n_cand >= 0, HQ_ERR_INVALID, "hq_vertical_scores: bad sizes");
  HQ_REQUIRE(H_Q % H_KV == 0, HQ_ERR_INVALID, "hq_vertical_scores: H_Q %d not a multiple of H_KV %d", H_Q, H_KV);
  const int R = H_Q / H_KV;
  HQ_REQUIRE(R <= 16, HQ_ERR_UNSUPPORTED, "hq_vertical_scores: kv_repeat %d > 16", R);
  HQ_REQUIRE(tail_len >= 1 && tail_len <= n_q, HQ_ERR_INVALID, "hq_vertical_scores: tail_len %d outside 1..%d", tail_len, n_q);
  HQ_REQUIRE(io_dtype == HQ_BF16 || io_dtype == HQ_F16, HQ_ERR_UNSUPPORTED,
             "hq_vertical_scores: keys must be bf16 or fp16 on the device path");
  if (B == 0 || n_cand == 0) return HQ_OK;
  HQ_REQUIRE(q && k && pooled && scores, HQ_ERR_INVALID, "hq_vertical_scores: null pointer");
  HQ_REQUIRE(aligned16(k) && k_stride_b % 8 == 0 && k_stride_h % 8 == 0 && k_stride_n % 8 == 0, HQ_ERR_ALIGNMENT,
             "hq_vertical_scores: key rows must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const int rm = round_mean ? io_dtype : -1;
  const int vec = aligned16(q) && q_stride_b % 8 == 0 && q_stride_h % 8 == 0 && q_stride_n % 8 == 0;
  const dim3 pgrid((unsigned)(B * H_Q), 128 / kPoolCh);
  if (io_dtype == HQ_BF16)
    pool_query_kernel<__nv_bfloat16><<<pgrid, kPoolThreads, 0, st>>>((const __nv_bfloat16*)q, q_stride_b, q_stride_h, q_stride_n, H_Q,
                                                                     n_q, tail_len, rm, group, io_dtype, vec, pooled);
  else
    pool_query_kernel<__half><<<pgrid, kPoolThreads, 0, st>>>((const __half*)q, q_stride_b, q_stride_h, q_stride_n, H_Q, n_q,
                                                              tail_len, rm, group, io_dtype, vec, pooled);
  HQ_CUDA(cudaGetLastError());
  const int tiles = (n_cand + 15) / 16;
  int chunks = (2 * sm_count() + B * H_KV - 1) / (B * H_KV);
  const int max_chunks = (tiles + kScoreWarps - 1) / kScoreWarps;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  dim3 grid((unsigned)chunks, (unsigned)(B * H_KV)), block(kScoreWarps * 32);
  const uint16_t* kk = (const uint16_t*)k;
  const bool bf = io_dtype == HQ_BF16;
  if (R <= 8) {
    if (bf) vertical_scores_kernel<true, 1><<<grid, block, 0, st>>>(kk, k_stride_b, k_stride_h, k_stride_n, H_KV, R, n_cand, pooled, round_scores, scores);
    else vertical_scores_kernel<false, 1><<<grid, block, 0, st>>>(kk, k_stride_b, k_stride_h, k_stride_n, H_KV, R, n_cand, pooled, round_scores, scores);
  } else {
    if (bf) vertical_scores_kernel<true, 2><<<grid, block, 0, st>>>(kk, k_stride_b, k_stride_h, k_stride_n, H_KV, R, n_cand, pooled, round_scores, scores);
    else vertical_scores_kernel<false, 2><<<grid, block, 0, st>>>(kk, k_stride_b, k_stride_h, k_stride_n, H_KV, R, n_cand, pooled, round_scores, scores);
  }
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}
}  // namespace hq

extern "C" int hq_vertical_scores(const void* q, int io_dtype, int64_t q_stride_b, int64_t q_stride_h, int64_t q_stride_n,
                                  int B, int H_Q, int n_q, int tail_len,
                                  const void* k, int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_n,
                                  int H_KV, int n_cand, int round_mean, int round_scores,
                                  float* pooled, float* scores, void* stream) {
  return hq::vertical_scores_impl(q, io_dtype, q_stride_b, q_stride_h, q_stride_n, B, H_Q, n_q, tail_len, 1, k, k_stride_b,
                                  k_stride_h, k_stride_n, H_KV, n_cand, round_mean, round_scores, pooled, scores, stream);
}

// The selection of the cache's freeze: the saved queries of the `group` query heads of a kv-head are averaged first
// (per token, rounded to io_dtype), then pooled and scored per KV head.  q is [B, H_KV * group, n_q, 128].
extern "C" int hq_vertical_scores_grouped(const void* q, int io_dtype, int64_t q_stride_b, int64_t q_stride_h, int64_t q_stride_n,
                                          int B, int H_KV, int group, int n_q, int tail_len,
                                          const void* k, int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_n,
                                          int n_cand, int round_mean, int round_scores,
                                          float* pooled, float* scores, void* stream) {
  using namespace hq;
  HQ_REQUIRE(group >= 1 && group <= 64, HQ_ERR_INVALID, "hq_vertical_scores_grouped: group %d outside 1..64", group);
  return vertical_scores_impl(q, io_dtype, q_stride_b, q_stride_h, q_stride_n, B, H_KV, n_q, tail_len, group, k, k_stride_b,
                              k_stride_h, k_stride_n, H_KV, n_cand, round_mean, round_scores, pooled, scores, stream);
}

extern "C" int hq_topk(const float* scores, int64_t scores_stride, int rows, int n, int k,
                       int64_t* idx_desc, int32_t* idx_asc, void* stream) {
  using namespace hq;
  HQ_REQUIRE(rows >= 0 && n >= 0 && k >= 0, HQ_ERR_INVALID, "hq_topk: negative size");
  if (rows == 0 || k == 0) return HQ_OK;
  HQ_REQUIRE(k <= n, HQ_ERR_INVALID, "hq_topk: k %d > n %d", k, n);
  HQ_REQUIRE(k <= kTopkMaxK, HQ_ERR_UNSUPPORTED, "hq_topk: k %d > %d", k, kTopkMaxK);
  HQ_REQUIRE(scores && idx_desc, HQ_ERR_INVALID, "hq_topk: null pointer");
  static thread_local int attr_dev = -1;
  int dev = 0;
  HQ_CUDA(cudaGetDevice(&dev));
  if (attr_dev != dev) {
    HQ_CUDA(cudaFuncSetAttribute(topk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopkSmem));
    HQ_CUDA(cudaFuncSetAttribute(topk_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopkSmem));
    HQ_CUDA(cudaFuncSetAttribute(topk_cluster_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopkSmem));
    HQ_CUDA(cudaFuncSetAttribute(topk_cluster_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopkSmem));
    attr_dev = dev;
  }
  const TopkForm f = topk_form(rows, n, k, sm_count());
  if (f.blocks > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows * f.blocks);
    cfg.blockDim = dim3(kSliceThreads);
    cfg.dynamicSmemBytes = f.smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)f.blocks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const auto kernel = f.kept ? topk_cluster_kernel<true> : topk_cluster_kernel<false>;
    HQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, scores, scores_stride, n, k, f.seg, f.list, idx_desc, idx_asc));
    return HQ_OK;
  }
  const auto kernel = f.kept ? topk_kernel<true> : topk_kernel<false>;
  kernel<<<rows, kTopkThreads, f.smem, (cudaStream_t)stream>>>(scores, scores_stride, n, k, f.list, idx_desc, idx_asc);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}
