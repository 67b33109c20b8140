// Hybrid-precision causal prefill attention on the Blackwell tensor path.
//
// Tile semantics as stated in hq_prefill.cu's header: for the 128-query
// block at s of query head h, keys below wla(s) are INT8 unless they are vertical lines of h
// (masked here, served from gathered BF16 tiles), keys in [wla(s), s + 128) are BF16 + causal mask.
//
// One CTA works on the same 128 queries of TWO query heads of one KV group (A and B), so every INT8 and
// window K / V tile that reaches shared memory feeds two score tiles, and the two heads' softmax chains
// interleave on the SM: while one head's threads are in their exponentials the tensor core runs the other
// head's products.  11 warps:
//   warp 8 (one lane)  producer: TMA tensor-map loads (128-byte swizzle) of both heads' Q once, then K tiles
//                      and V tiles into two rings of three and four slots (a K slot is free again
//                      after the heads' Q K^T, a V slot after their P V).  INT8 and window items serve both heads;
//                      the gathered vertical-line tiles are per head.
//   warps 9, 10        (an elected lane each) issue tcgen05.mma for head A / B: S = Q K^T (kind::i8 with s32
//                      accumulators, or kind::f16 on bf16) into one of the head's two S buffers in tensor
//                      memory, two tiles ahead of O += P V (kind::f16, P read from tensor memory, V from
//                      shared memory); completion is signalled with tcgen05.commit.
//   warps 0-3 / 4-7    softmax of head A / B, one thread per query row: tcgen05.ld of the 64 scores,
//                      scales / masks, online softmax in base 2 with a lazily updated maximum (the O
//                      accumulator is rescaled in tensor memory only when the maximum grows by more than
//                      2^8), P as bf16 pairs written back over the first 32 columns of the same S buffer,
//                      final O / l from tensor memory.
// Tensor memory (512 columns): S_A0 | S_A1 | S_B0 | S_B1 (64 each) | O_A | O_B (128 each).
// Shared-memory operands are K-major, but for V of 16-bit P V where the caller gives it as it lies (v_rows): a tile is then two
// boxes of 64 keys x 64 channels, an MN-major operand, and nothing is transposed or padded (keys past N load as zero).
// With V transposed first, a call took 8 us more at 8K and 5 to 8 us of 105 at 2 x 1973; a plan that is kept for later and
// FP8 P V (V is quantised anyway) still take V^T.
// Every wait is bounded and abortable; a failed wait raises bit 1 of the status word, and the rows of the block and of
// those after it are NaN.
#include "hq_tc05.cuh"

namespace hq {

struct PrefillTcParams {
  const float* q_scale; const float* k_scale;      // [B,H_Q,Npad], [B,H_KV,Npad]
  const float* v_scale;                            // FP8 P V: [B,H_KV,128], one per channel
  const int* nv_valid;
  void* out; int out_dtype; int64_t o_sb, o_sh, o_sn;
  int B, H_Q, H_KV, N, Npad, W, T, Tpad, nqb, nkb;
  int group;                                       // head pairs whose blocks are launched together
  int v_rows;                                      // V tiles are rows of keys (mVt 4-D, mXv 2-D) instead of V^T
  float sml;
  int* status;
};

constexpr int kTcThreads = 352;            // 2 x 4 softmax warps + producer warp + one MMA warp per head
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColS = 0, kColO = 256; // S buffer of head h, parity s: kColS + 128 h + 64 s; O of head h: kColO + 128 h

constexpr int kKStages = 3;    // depth of the K ring: Q K^T runs two tiles ahead of P V and frees its slot at once
constexpr int kVStages = 4;    // depth of the V ring
constexpr int kNearRun = 2;    // a head waits for a K item before a due P V across at most this many items of the other head
constexpr uint32_t kDrainPolls = 400000;   // limit of the waits at the end of a block
constexpr int kKsSlots = 6;    // ring of key-scale rows: a row is dead once P V of its item + 2 has been issued
constexpr int kKsBytes = 768;  // 64 key scales | 64 bias terms of head A | 64 bias terms of head B
struct TcSmem {              // offsets from a 1024-aligned base
  static constexpr int Qi = 0;                             // 2 x 16 KB  [head][128 rows][128 B] int8
  static constexpr int Qb = 32768;                         // 2 x 32 KB  [head][2 halves][128 rows][128 B] bf16
  static constexpr int K = 98304;                          // kKStages x 16 KB: int8 tile, or two bf16 halves
  static constexpr int V = K + kKStages * 16384;           // kVStages x 16 KB: V^T [128 d rows][128 B], or V [2 halves of d][64 key rows][128 B]
  static constexpr int Ks = V + kVStages * 16384;          // kKsSlots x kKsBytes
  static constexpr int Bar = Ks + kKsSlots * kKsBytes;     // barriers + scratch
  static constexpr int Total = Bar + 256;
};

// A converged warp's wait.  The first poll (which the hardware holds for a while) is inline and nearly always enough; the
// poll loop is out of line, so that a wait is straight-line code.  A poll takes 40 clocks, but with the poll loop inline a
// wait for a barrier that had long flipped took 300 to 450 in these loops: softmax and issuing warps fetch different
// code through one instruction cache, and every taken branch of a wait, of the ring walk and of the two kinds of tiles went
// somewhere cold.  With the waits straight, the INT8 tiles in loops of their own (softmax and issuing warps), and the three
// waits of an issuing warp asked together: hybrid 8K 708 -> 667 us, 32K 9.01 -> 8.53 ms, FP8 16K 2.93 -> 2.81 ms, 16-bit
// 2 x 1973 112 -> 107 us per call.
static __device__ __noinline__ bool mbar_wait_rest(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return (bool)__all_sync(0xffffffffu, tc::mbar_wait_abortable(bar, parity, abort_flag));
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (__builtin_expect(__all_sync(0xffffffffu, mbar_try_wait(bar, parity)), 1)) return true;
  return mbar_wait_rest(bar, parity, abort_flag);
}
// three at once: one vote where all are there
__device__ __forceinline__ bool mbar_wait_warp3(uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1, uint64_t* b2, uint32_t p2,
                                                volatile int* abort_flag) {
  const bool r0 = mbar_try_wait(b0, p0), r1 = mbar_try_wait(b1, p1), r2 = mbar_try_wait(b2, p2);
  if (__builtin_expect(__all_sync(0xffffffffu, r0 && r1 && r2), 1)) return true;
  return mbar_wait_rest(b0, p0, abort_flag) && mbar_wait_rest(b1, p1, abort_flag) && mbar_wait_rest(b2, p2, abort_flag);
}

struct TcPlan {
  int n_rest, n_win, nvert0, nvert1, nheads;
  __device__ __forceinline__ int nvert(int h) const { return h ? nvert1 : nvert0; }
  __device__ __forceinline__ int n_ops() const { return nheads * (n_rest + n_win) + nvert0 + nvert1; }
  __device__ __forceinline__ int n_tiles(int h) const { return h < nheads ? n_rest + nvert(h) + n_win : 0; }
  __device__ __forceinline__ int n_items() const { return n_rest + nvert0 + nvert1 + n_win; }
};

// The ring items of a CTA in load order, walked with counters only (one producer lane and the two converged issuing
// warps walk it, and their instruction latency paces the pipeline): the INT8 tiles, then the vertical-line tiles of the
// two heads interleaved (A's j-th, B's j-th, ...), then the window tiles.  INT8 and window items feed both
// heads, a vertical item only its own head.
struct TcItemIter {
  int kind;     // 0 INT8, 1 vertical, 2 window, 3 = past the end
  int j;        // index within the kind
  int hh;       // owning head of a vertical item
  int stage;    // ring slot
  int depth;    // ring depth
  uint32_t par; // phase parity of the slot's "full" barrier for this item
  __device__ __forceinline__ bool valid(const TcPlan& pl) const {
    return kind == 0 ? j < pl.n_rest : kind == 1 ? j < pl.nvert(hh) : j < pl.n_win;
  }
  __device__ __forceinline__ void step(const TcPlan& pl) {
    if (kind == 1) { if (++hh == 2) { hh = 0; ++j; } } else ++j;
    const int lim = kind == 0 ? pl.n_rest : kind == 1 ? max(pl.nvert0, pl.nvert1) : pl.n_win;
    if (j >= lim) { ++kind; j = 0; hh = 0; }
  }
  __device__ __forceinline__ void begin(const TcPlan& pl, int ring_depth) {
    kind = 0; j = 0; hh = 0; stage = 0; par = 0u; depth = ring_depth;
    while (kind < 3 && !valid(pl)) step(pl);
  }
  __device__ __forceinline__ void next(const TcPlan& pl) {
    if (++stage == depth) { stage = 0; par ^= 1u; }
    // the common cases first (a ring is walked by one lane or one warp: every instruction here is latency)
    if (kind == 0 && j + 1 < pl.n_rest) { ++j; return; }
    if (kind == 2) { if (++j >= pl.n_win) kind = 3; return; }
    do step(pl); while (kind < 3 && !valid(pl));
  }
  // at the item behind INT8 tile `last`, whose slot and parity the caller has counted
  __device__ __forceinline__ void resume(const TcPlan& pl, int last, int slot, uint32_t parity) {
    kind = 0; j = last; hh = 0;
    do step(pl); while (kind < 3 && !valid(pl));
    stage = slot; par = parity;
  }
  __device__ __forceinline__ bool done() const { return kind >= 3; }
  __device__ __forceinline__ bool feeds(int h) const { return kind != 1 || hh == h; }
};

// The rare tile of a row whose P values against the current reference may be too large (or that has no
// reference yet): take the true maximum of the tile from the scores in tensor memory, rescale O and the row sum
// if the reference moves, and write the tile's P against the reference as it then stands.  Called by whole
// warps; kept out of line so that the common path keeps its registers.
struct TcSlowResult { float m_ref, l; bool ok; };
// FP8 P V (the arithmetic of the reference's sm_90 kernel, vendor/sageattention/csrc/qattn/attn_utils.cuh:30,354-458 and
// qk_int_sv_f8_cuda_sm90.cu:259-364): P~ = 2^(s - m + 8.807) against the EXACT running maximum m (so P~ <= 448, the largest
// e4m3 value), the row sum taken in fp32 before P~ is rounded to e4m3.
constexpr float kFp8Offset = 8.807f;

// compile-time flag handed to a lambda
struct TcTrue { static constexpr bool value = true; };
struct TcFalse { static constexpr bool value = false; };

// O of a row times alpha, in tensor memory, once every P V issued so far has completed.  Whole warps.
__device__ __noinline__ bool tc_rescale_o(uint32_t tO, float alpha, uint64_t* pv_bar, uint32_t pv_parity, volatile int* abort_flag) {
  if (!__all_sync(0xffffffffu, tc::mbar_wait_abortable(pv_bar, pv_parity, abort_flag))) return false;
  tc::fence_after_sync();
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    uint32_t o[32];
    tc::tmem_ld32(tO + ch * 32, o);
    tc::tmem_wait_ld();
#pragma unroll
    for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
    tc::tmem_st32(tO + ch * 32, o);
  }
  tc::tmem_wait_st();
  return true;
}

__device__ __noinline__ TcSlowResult tc_slow_tile(uint32_t tS, uint32_t tO, const float4* ks4, const float4* kb4, bool is_i8,
                                                  float esc, uint32_t mlo, uint32_t mhi, float m_ref, float l,
                                                  uint64_t* pv_bar, uint32_t pv_parity, volatile int* abort_flag) {
  TcSlowResult res;
  res.ok = true;
  uint32_t sr[64];
  float x[64];
  tc::tmem_ld32(tS, *reinterpret_cast<uint32_t(*)[32]>(&sr[0]));
  tc::tmem_ld32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(&sr[32]));
  tc::tmem_wait_ld();
  if (is_i8) {
#pragma unroll
    for (int c4 = 0; c4 < 16; ++c4) {
      const float4 kk = ks4[c4], bb = kb4[c4];
      x[4 * c4] = fmaf(__int_as_float((int)sr[4 * c4] + 0x4B400000), kk.x, bb.x);
      x[4 * c4 + 1] = fmaf(__int_as_float((int)sr[4 * c4 + 1] + 0x4B400000), kk.y, bb.y);
      x[4 * c4 + 2] = fmaf(__int_as_float((int)sr[4 * c4 + 2] + 0x4B400000), kk.z, bb.z);
      x[4 * c4 + 3] = fmaf(__int_as_float((int)sr[4 * c4 + 3] + 0x4B400000), kk.w, bb.w);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 64; ++c) {
      const uint32_t mw = c < 32 ? mlo : mhi;
      x[c] = ((mw >> (c & 31)) & 1u) ? -INFINITY : __uint_as_float(sr[c]);
    }
  }
  float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int c = 0; c < 64; ++c) m4[c & 3] = fmaxf(m4[c & 3], x[c]);
  const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * esc;      // esc > 0
  // Once here, move the reference all the way up to the maximum seen: with the reference left below it,
  // every later tile with a few scores near that maximum would bring the row back here.
  const bool grow = mx > m_ref;                              // also true for the first finite maximum
  if (__any_sync(0xffffffffu, grow)) {
    const float alpha = (m_ref == -INFINITY) ? 0.f : ex2f(m_ref - mx);
    if (pv_bar != nullptr) {   // O must be quiescent: every P V of this head issued so far has to be complete
      res.ok = tc_rescale_o(tO, grow ? alpha : 1.f, pv_bar, pv_parity, abort_flag);
      if (!res.ok) { res.m_ref = m_ref; res.l = l; return res; }
    }
    if (grow) { l *= alpha; m_ref = mx; }
  }
  const float mu = m_ref == -INFINITY ? 0.f : m_ref;
  float rs[4] = {0.f, 0.f, 0.f, 0.f};
  uint32_t pk[32];
#pragma unroll
  for (int c = 0; c < 64; c += 2) {
    const float p0 = ex2f(fmaf(x[c], esc, -mu)), p1 = ex2f(fmaf(x[c + 1], esc, -mu));
    rs[c & 3] += p0; rs[(c & 3) + 1] += p1;
    __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);       // low half = even column
    pk[c >> 1] = *reinterpret_cast<uint32_t*>(&hh);
  }
  tc::tmem_st32(tS, pk);
  tc::tmem_wait_st();
  res.m_ref = m_ref;
  res.l = l + (rs[0] + rs[1]) + (rs[2] + rs[3]);
  return res;
}

// The output rows of a block that gave up, or that was skipped after one that did: NaN, so that a caller who does not
// read the status word (which takes a synchronisation) never takes memory nobody wrote for a result.  All threads.
__device__ __noinline__ void tc_fill_nan(const PrefillTcParams& p, int b, int hq0, int nheads, int s0) {
  const float nan = __int_as_float(0x7FFFFFFF);
  for (int x = threadIdx.x; x < nheads * 128 * 128; x += kTcThreads) {
    const int h = x >> 14, row = s0 + ((x >> 7) & 127);
    if (row < p.N) store_out(p.out, b * p.o_sb + (hq0 + h) * p.o_sh + (int64_t)row * p.o_sn + (x & 127), nan, p.out_dtype);
  }
}

template <bool kFp8>
__global__ void __launch_bounds__(kTcThreads, 1)
prefill_tc_kernel(const __grid_constant__ CUtensorMap mQi, const __grid_constant__ CUtensorMap mQb,
                  const __grid_constant__ CUtensorMap mKi, const __grid_constant__ CUtensorMap mKb,
                  const __grid_constant__ CUtensorMap mVt, const __grid_constant__ CUtensorMap mXk,
                  const __grid_constant__ CUtensorMap mXv, const __grid_constant__ CUtensorMap mKs,
                  const __grid_constant__ CUtensorMap mKbs, const __grid_constant__ PrefillTcParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TcSmem::Bar);
  uint64_t* q_full = bars + 0;                   // INT8, BF16
  uint64_t* k_full = bars + 2;                   // [kKStages]
  uint64_t* k_empty = k_full + kKStages;         // [kKStages]
  uint64_t* v_full = k_empty + kKStages;         // [kVStages]
  uint64_t* v_empty = v_full + kVStages;         // [kVStages]
  uint64_t* s_full = v_empty + kVStages;         // [head][2]
  uint64_t* p_ready = s_full + 4;                // [head][2]
  uint64_t* pv_done = p_ready + 4;               // [head][2]
  uint64_t* drained = pv_done + 4;               // [head]: the head's last product is done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(drained + 3);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  __shared__ int s_skip;
  if (tid == 0) s_skip = *reinterpret_cast<volatile int*>(p.status) & 2;
  const int R = p.H_Q / p.H_KV, pairs = (R + 1) / 2;
  // Blocks in the order of their length, longest first, over a group of head pairs whose K and V stay in L2 together (the
  // host sizes the groups): head by head, each from its longest block to its shortest, left the SMs that took the last
  // head's long blocks running alone (8192 tokens, 16 pairs: 12 % above an even split; a call 840 -> 780 us), and all
  // heads of 32K tokens at once read K and V past L2 (9.06 -> 9.23 ms).
  const int units = p.B * p.H_KV * pairs;
  const int grp = blockIdx.x / (p.group * p.nqb), in_grp = blockIdx.x - grp * (p.group * p.nqb);
  const int size = min(p.group, units - grp * p.group), level = in_grp / size;
  const int qb = p.nqb - 1 - level, unit = grp * p.group + in_grp - level * size;
  const int b = unit / (p.H_KV * pairs), hp = unit - b * (p.H_KV * pairs);
  const int hkv = hp / pairs, pr = hp - hkv * pairs;
  const int s0 = qb * 128;
  TcPlan plan;
  plan.nheads = (2 * pr + 1 < R) ? 2 : 1;
  const int64_t bhk = (int64_t)b * p.H_KV + hkv;
  const int64_t bhq0 = (int64_t)b * p.H_Q + hkv * R + 2 * pr;
  const int wla = p.W > 0 ? (max(0, s0 - (p.W - 1)) / 64) * 64 : s0;
  plan.n_rest = wla / 64;
  const int win_end = min(p.N, s0 + 128);
  plan.n_win = (win_end - wla + 63) / 64;
  const int nv0 = p.T > 0 ? p.nv_valid[bhq0 * p.nqb + qb] : 0;
  const int nv1 = (p.T > 0 && plan.nheads == 2) ? p.nv_valid[(bhq0 + 1) * p.nqb + qb] : 0;
  plan.nvert0 = (nv0 + 63) / 64;
  plan.nvert1 = (nv1 + 63) / 64;

  // The producer's lane sets up the barriers and asks for the queries that the first products need before the block meets:
  // the loads, the status word, the list lengths and the tensor memory are then waited for together (before, one after the
  // other: 7000 clocks to a block's first scores, with all of Q on one barrier; now 4900).
  auto load_q = [&](bool i8) {
    mbar_expect_tx(q_full + (i8 ? 0 : 1), (uint32_t)plan.nheads * (i8 ? 16384 : 32768));
    for (int h = 0; h < plan.nheads; ++h) {
      const int qrow = (int)((bhq0 + h) * p.N + s0);
      if (i8) {
        tc::tma_load_2d(smem + TcSmem::Qi + h * 16384, &mQi, 0, qrow, q_full);
      } else {
        tc::tma_load_2d(smem + TcSmem::Qb + h * 32768, &mQb, 0, qrow, q_full + 1);
        tc::tma_load_2d(smem + TcSmem::Qb + h * 32768 + 16384, &mQb, 64, qrow, q_full + 1);
      }
    }
  };
  if (warp == 8) {
    if (lane == 0) {
      mbar_init(q_full, 1); mbar_init(q_full + 1, 1);
      // a slot comes back when every head has arrived
      for (int i = 0; i < kKStages; ++i) { mbar_init(k_full + i, 1); mbar_init(k_empty + i, plan.nheads); }
      for (int i = 0; i < kVStages; ++i) { mbar_init(v_full + i, 1); mbar_init(v_empty + i, plan.nheads); }
      for (int i = 0; i < 4; ++i) { mbar_init(s_full + i, 1); mbar_init(p_ready + i, 128); mbar_init(pv_done + i, 1); }
      mbar_init(drained, 1); mbar_init(drained + 1, 1);
      *abort_flag = 0;
      fence_mbar_init();
      fence_proxy_async_smem();
      load_q(plan.n_rest > 0);
      tc::tma_prefetch_desc(&mKi); tc::tma_prefetch_desc(&mKs); tc::tma_prefetch_desc(&mKbs); tc::tma_prefetch_desc(&mVt); tc::tma_prefetch_desc(&mKb);
    }
    __syncwarp();
    tc::tmem_alloc(tmem_slot, kTmemCols);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (s_skip) {                               // an earlier CTA gave up: drain the grid quickly
    if (tid == 256) {
      mbar_wait_bounded(q_full + (plan.n_rest > 0 ? 0 : 1), 0, kDrainPolls);
      *abort_flag = 1;
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      // K tiles and V tiles travel in rings of their own: a K slot comes back as soon as both heads' Q K^T
      // of its item have run, a V slot only after their P V, so K runs further ahead than V.  One thread
      // feeds both rings and never blocks on either.
      TcItemIter ck, cv;
      ck.begin(plan, kKStages);
      cv.begin(plan, kVStages);
      int ks_slot = 0;
      uint32_t idle = 0;
      bool q_due = plan.n_rest > 0;              // BF16 queries, behind the first INT8 tiles
      while (!ck.done() || !cv.done()) {
        bool progress = false;
        if (q_due && (ck.kind != 0 || ck.j == kKStages)) { load_q(false); q_due = false; }
        if (!ck.done() && mbar_test_wait(k_empty + ck.stage, ck.par ^ 1u)) {
          uint8_t* sK = smem + TcSmem::K + ck.stage * 16384;
          uint64_t* full = k_full + ck.stage;
          if (ck.kind == 0) {
            uint8_t* sS = smem + TcSmem::Ks + ks_slot * kKsBytes;
            mbar_expect_tx(full, 8192 + 256 + 256 * (uint32_t)plan.nheads);
            tc::tma_load_2d(sK, &mKi, 0, (int)(bhk * p.N + ck.j * 64), full);
            tc::tma_load_2d(sS, &mKs, ck.j * 64, (int)bhk, full);
            for (int h = 0; h < plan.nheads; ++h) tc::tma_load_2d(sS + 256 + 256 * h, &mKbs, ck.j * 64, (int)(bhq0 + h), full);
            if (++ks_slot == kKsSlots) ks_slot = 0;
          } else {
            const CUtensorMap* m = ck.kind == 1 ? &mXk : &mKb;
            const int krow = ck.kind == 1 ? (int)((bhq0 + ck.hh) * p.Tpad + ck.j * 64) : (int)(bhk * p.N + wla + ck.j * 64);
            mbar_expect_tx(full, 16384);
            tc::tma_load_2d(sK, m, 0, krow, full);
            tc::tma_load_2d(sK + 8192, m, 64, krow, full);
          }
          ck.next(plan);
          progress = true;
        }
        if (!cv.done() && mbar_test_wait(v_empty + cv.stage, cv.par ^ 1u)) {
          uint8_t* sV = smem + TcSmem::V + cv.stage * 16384;
          uint64_t* full = v_full + cv.stage;
          mbar_expect_tx(full, kFp8 ? 8192 : 16384);      // FP8: V^T tiles of 64 one-byte keys
          if (!kFp8 && p.v_rows) {            // two boxes of 64 channels
            for (int x = 0; x < 2; ++x) {
              if (cv.kind == 1) tc::tma_load_2d(sV + 8192 * x, &mXv, 64 * x, (int)((bhq0 + cv.hh) * p.Tpad + cv.j * 64), full);
              else tc::tma_load_4d(sV + 8192 * x, &mVt, 64 * x, (cv.kind == 0 ? 0 : wla) + cv.j * 64, hkv, b, full);
            }
          } else if (cv.kind == 1) tc::tma_load_2d(sV, &mXv, cv.j * 64, (int)((bhq0 + cv.hh) * 128), full);
          else tc::tma_load_2d(sV, &mVt, (cv.kind == 0 ? 0 : wla) + cv.j * 64, (int)(bhk * 128), full);
          cv.next(plan);
          progress = true;
        }
        if (progress) { idle = 0; continue; }
        __nanosleep(64);
        if (*abort_flag) break;
        if (++idle > 2000000u) { *abort_flag = 1; break; }
      }
      // A block must not end with copies under way to its shared memory, also where it gives up: wait for the last load
      // of every slot (a slot without one answers at once)
      bool landed = plan.n_rest == 0 || mbar_wait_bounded(q_full, 0, kDrainPolls);
      if (!q_due) landed = mbar_wait_bounded(q_full + 1, 0, kDrainPolls) && landed;
      for (int i = 0; i < kKStages; ++i) landed = mbar_wait_bounded(k_full + i, i < ck.stage ? ck.par : ck.par ^ 1u, kDrainPolls) && landed;
      for (int i = 0; i < kVStages; ++i) landed = mbar_wait_bounded(v_full + i, i < cv.stage ? cv.par : cv.par ^ 1u, kDrainPolls) && landed;
      if (!landed) *abort_flag = 1;
    }
  } else if (warp >= 9) {
    // ------------------------------------------------------------ MMA issuers: warp 9 for head A, warp 10 for head B
    // The warp walks its loop converged and elects a lane only around the tensor instructions: descriptors and
    // addresses then stay in uniform registers (the issuing loop was as long as the softmax loop when one diverged
    // lane ran it: 32K hybrid 9.98 -> 9.69 ms, FP8 16K 5.91 -> 5.38 ms, 16-bit 2 x 1973 207 -> 189 us per call).
    // In the head's own order: Q K^T of tiles 0 and 1, then for every tile t:
    // P V of t, Q K^T of t + 2 (across a long run of the other head's tiles: P V of all tiles before it, then Q K^T of
    // the next two).  The S buffer that Q K^T of t + 2 overwrites held P of tile t, and the tensor
    // core runs one thread's operations in issue order, so the scores of the next tile are ready while the
    // head's softmax threads are still on the current one.  Ring slots come back when both heads are done
    // with them: a head arrives by tcgen05.commit for an item it used and by a plain arrive for a
    // vertical-line item of the other head, in ring order either way.  No wait may need something of a LATER item than
    // the one it is for, except K of the next few: every pair of tile counts then passes (walked on the CPU with these
    // depths by the tests).
    const int h = warp - 9;
    if (h < plan.nheads) {
      constexpr uint32_t idesc_i8 = tc::make_idesc(2, tc::kFmtS8, tc::kFmtS8, 128, 64);
      constexpr uint32_t idesc_qk = tc::make_idesc(1, tc::kFmtBF16, tc::kFmtBF16, 128, 64);
      const uint32_t idesc_pv = tc::make_idesc(1, tc::kFmtBF16, tc::kFmtBF16, 128, 128) | (p.v_rows ? tc::kBMnMajor : 0u);
      const uint32_t v_step = p.v_rows ? 2048 >> 4 : 32 >> 4;       // 16 keys, in units of the descriptor
      constexpr uint32_t idesc_pv8 = tc::make_idesc(1, tc::kFmtE4M3, tc::kFmtE4M3, 128, 128);
      auto wait = [&](uint64_t* bar, uint32_t par) { return mbar_wait_warp(bar, par, abort_flag); };
      bool ok = wait(q_full + (plan.n_rest > 0 ? 0 : 1), 0), q_bf = plan.n_rest == 0;
      // operand descriptors differ only in their start-address field (16-byte units)
      const uint64_t dQi = tc::smem_desc_k128(smem + TcSmem::Qi + h * 16384, 0);
      const uint64_t dQb = tc::smem_desc_k128(smem + TcSmem::Qb + h * 32768, 0);
      const uint64_t dK = tc::smem_desc_k128(smem + TcSmem::K, 0);
      const uint64_t dV = kFp8 ? tc::smem_desc_k64(smem + TcSmem::V, 0)
                               : p.v_rows ? tc::smem_desc_mn128(smem + TcSmem::V, 8192) : tc::smem_desc_k128(smem + TcSmem::V, 0);
      const uint32_t tS = tmem_base + kColS + 128u * h, tO = tmem_base + kColO + 128u * h;
      const int n_t = plan.n_tiles(h), n_rest = plan.n_rest;
      TcItemIter cq, cp;
      cq.begin(plan, kKStages);
      cp.begin(plan, kVStages);
      int tq = 0;
      auto k_ready = [&]() {     // wait for the next item that feeds this head; hand back the other head's on the way
        for (;;) {
          ok = wait(k_full + cq.stage, cq.par);
          if (!ok || cq.feeds(h)) break;
          if (tc::elect_one()) tc::mbar_arrive(k_empty + cq.stage);
          cq.next(plan);
        }
        if (cq.kind != 0 && !q_bf) { ok = ok && wait(q_full + 1, 0); q_bf = true; }
      };
      auto v_ready = [&]() {
        for (;;) {
          ok = wait(v_full + cp.stage, cp.par);
          if (!ok || cp.feeds(h)) return;
          if (tc::elect_one()) tc::mbar_arrive(v_empty + cp.stage);
          cp.next(plan);
        }
      };
      auto pv_issue = [&](int t, int stage) {    // one lane
        const uint32_t aP = tS + 64u * (t & 1);
        const uint64_t bV = dV + (uint64_t)(stage * 1024);
        if constexpr (kFp8) {     // 64 keys = two K steps of 32 e4m3: 8 columns of P, 32 bytes of a V^T row each
#pragma unroll
          for (int k = 0; k < 2; ++k) tc::mma_f8_ts(tO, aP + 8 * k, bV + 2 * k, idesc_pv8, (t > 0 || k > 0) ? 1u : 0u);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) tc::mma_bf16_ts(tO, aP + 8 * k, bV + v_step * k, idesc_pv, (t > 0 || k > 0) ? 1u : 0u);
        }
        tc::mma_commit(pv_done + 2 * h + (t & 1));
        tc::mma_commit(v_empty + stage);
      };
      auto qk_issue = [&]() {    // one lane
        const uint32_t dS = tS + 64u * (tq & 1);
        const uint64_t bK = dK + (uint64_t)(cq.stage * 1024);
        if (cq.kind == 0) {
#pragma unroll
          for (int k = 0; k < 4; ++k) tc::mma_s8_ss(dS, dQi + 2 * k, bK + 2 * k, idesc_i8, k > 0);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            tc::mma_bf16_ss(dS, dQb + (k >> 2) * 1024 + 2 * (k & 3), bK + (k >> 2) * 512 + 2 * (k & 3), idesc_qk, k > 0);
        }
        tc::mma_commit(s_full + 2 * h + (tq & 1));
        tc::mma_commit(k_empty + cq.stage);
      };
      // The other head's vertical-line items that K's walk still has to hand back before this head's next item, if they are
      // more than kNearRun (where this head's list is the shorter one; in the interleaved part it is one item).
      auto run_ahead = [&]() {
        return cq.kind == 1 && cq.hh != h && cq.j + (h == 0 ? 1 : 0) >= plan.nvert(h) && plan.nvert(1 - h) - cq.j > kNearRun;
      };
      int t = 0;
      while (ok && t < n_t) {
        // the start, or nothing issued ahead across a run of the other head's items: both walks stand here, the run goes
        // back K and V item by item
        while (ok && !cq.feeds(h)) {
          ok = wait(k_full + cq.stage, cq.par);
          if (ok && tc::elect_one()) tc::mbar_arrive(k_empty + cq.stage);
          ok = ok && wait(v_full + cp.stage, cp.par);
          if (ok && tc::elect_one()) tc::mbar_arrive(v_empty + cp.stage);
          cq.next(plan);
          cp.next(plan);
        }
        for (int i = 0; ok && i < 2 && tq < n_t && (i == 0 || !run_ahead()); ++i) {
          k_ready();
          if (!ok) break;
          tc::fence_after_sync();
          if (tc::elect_one()) qk_issue();
          ++tq;
          cq.next(plan);
        }
        if (!ok) break;
        // INT8 tiles whose successor but one is INT8 too: tiles and items are the same, nothing to hand back
        if (t == 0 && tq == 2 && n_rest > 2) {
          int ks = cq.stage, vs = 0;
          uint32_t kpar = cq.par, vpar = 0u;
          for (; t + 2 < n_rest; ++t) {
            const int sl = 2 * h + (t & 1);
            ok = mbar_wait_warp3(v_full + vs, vpar, k_full + ks, kpar, p_ready + sl, (uint32_t)((t >> 1) & 1), abort_flag);
            if (!ok) break;
            tc::fence_after_sync();
            if (tc::elect_one()) {
              pv_issue(t, vs);
              const uint32_t dS = tS + 64u * (t & 1);
              const uint64_t bK = dK + (uint64_t)(ks * 1024);
#pragma unroll
              for (int k = 0; k < 4; ++k) tc::mma_s8_ss(dS, dQi + 2 * k, bK + 2 * k, idesc_i8, k > 0);
              tc::mma_commit(s_full + sl);
              tc::mma_commit(k_empty + ks);
            }
            if (++ks == kKStages) { ks = 0; kpar ^= 1u; }
            if (++vs == kVStages) { vs = 0; vpar ^= 1u; }
          }
          if (!ok) break;
          tq = t + 2;
          cq.resume(plan, tq - 1, ks, kpar);
          cp.resume(plan, t - 1, vs, vpar);
        }
        for (; t < tq; ++t) {
          // the operands first, P last: from the moment P is there nothing is waited for, and P V of t and Q K^T of t + 2
          // are issued together (32K hybrid 9.27 -> 9.05 ms, 8K 867 -> 844 us, while a wait cost the warp some 400 clocks).  Not
          // across a run of the other head's items: that head needs the V slots which P V of t and t + 1 give back to come to the end of its run, and K of t + 2 lies behind it - the two heads
          // would wait for one another (with rings of three and four slots: runs of five items and more).
          const bool more = tq == t + 2 && tq < n_t && !run_ahead();
          v_ready();
          if (ok && more) k_ready();
          if (!ok) break;
          const int sl = 2 * h + (t & 1);
          ok = wait(p_ready + sl, (uint32_t)((t >> 1) & 1));
          if (!ok) break;
          tc::fence_after_sync();
          if (tc::elect_one()) {
            pv_issue(t, cp.stage);
            if (more) qk_issue();
          }
          cp.next(plan);
          if (more) { ++tq; cq.next(plan); }
        }
      }
      // the same for products that write tensor memory
      if (tc::elect_one()) tc::mma_commit(drained + h);
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(drained + h, 0, kDrainPolls))) *abort_flag = 1;
    }
  } else {
    // ------------------------------------------------------------ softmax: one thread per query row and head
    // Warps 0-3 serve head A, warps 4-7 head B; warp w reaches the tensor-memory lanes 32 (w % 4) .. + 31.
    const int h = warp >> 2, wq = warp & 3;
    const int n_tiles = plan.n_tiles(h);
    const int r = wq * 32 + lane;            // query row inside the block = tensor-memory lane
    const int row = s0 + r;
    const int64_t bhq = bhq0 + (h < plan.nheads ? h : 0);
    const uint32_t lane_base = tmem_base + ((uint32_t)(wq * 32) << 16);
    const uint32_t colS = kColS + 128 * h, colO = kColO + 128 * h;
    const int n_rest = plan.n_rest, n_vert = plan.nvert(h), nvh = h ? nv1 : nv0;
    // rows past N compute on a token scale, so that a masked column (-inf) times the scale stays -inf
    const float qs = (row < p.N && n_tiles > 0 && n_rest > 0) ? p.q_scale[bhq * p.Npad + row] : 1e-30f;
    float m_ref = row < p.N ? -INFINITY : 0.f, l = 0.f;
    bool ok = true;
    int ks_slot = 0;
    if constexpr (kFp8) {
      // The scores of tile t.  tcgen05.ld is asynchronous: its wait stands right behind it, because the compiler may copy
      // registers wherever control flow meets and does not know that these are still being written.  (Asking for the
      // next scores before the hand-over of P, with the wait in the next iteration, gave no such guarantee and was not
      // faster either: 16K 2946 us, with load and wait around the hand-over 3208, like this 2936.)
      uint32_t sr[64];
      auto fetch = [&](int t) {
        ok = mbar_wait_warp(s_full + 2 * h + (t & 1), (uint32_t)((t >> 1) & 1), abort_flag);
        if (!ok) return;
        tc::fence_after_sync();
        tc::tmem_ld32(lane_base + colS + (t & 1) * 64, *reinterpret_cast<uint32_t(*)[32]>(&sr[0]));
        tc::tmem_ld32(lane_base + colS + (t & 1) * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&sr[32]));
        tc::tmem_wait_ld();
        tc::tie64(sr);
      };
      auto tile = [&](int t, auto int8_tile) {
        constexpr bool kI8 = decltype(int8_tile)::value;
        const uint32_t tS = lane_base + colS + (t & 1) * 64;
        const float esc = kI8 ? qs : p.sml;                    // > 0
        const float4* ks4 = reinterpret_cast<const float4*>(smem + TcSmem::Ks + ks_slot * kKsBytes);
        const float4* kb4 = ks4 + 16 + 16 * h;
        uint32_t mlo = 0u, mhi = 0u;                           // BF16 tiles: bit c set = column c (of 64) is masked
        if constexpr (kI8) {
          if (++ks_slot == kKsSlots) ks_slot = 0;
        } else {
          int lim;                                             // columns <= lim are visible
          if (t < n_rest + n_vert) lim = min(64, nvh - (t - n_rest) * 64) - 1;
          else lim = min(row, p.N - 1) - (wla + (t - n_rest - n_vert) * 64);
          mlo = lim >= 31 ? 0u : lim < 0 ? 0xFFFFFFFFu : (0xFFFFFFFFu << (lim + 1));
          mhi = lim >= 63 ? 0u : lim < 32 ? 0xFFFFFFFFu : (0xFFFFFFFFu << (lim - 31));
        }
        float* y = reinterpret_cast<float*>(sr);
        // scores before the row's factor `esc` (INT8: s32 -> fp32 by the magic-number add, key scale and bias in one
        // packed fma; BF16 tiles: masked columns -inf)
        if constexpr (kI8) {
#pragma unroll
          for (int c4 = 0; c4 < 16; ++c4) {
            const float4 kk = ks4[c4], bb = kb4[c4];
            const float2 a01 = make_float2(__int_as_float((int)sr[4 * c4] + 0x4B400000), __int_as_float((int)sr[4 * c4 + 1] + 0x4B400000));
            const float2 a23 = make_float2(__int_as_float((int)sr[4 * c4 + 2] + 0x4B400000), __int_as_float((int)sr[4 * c4 + 3] + 0x4B400000));
            const float2 x01 = ffma2(a01, make_float2(kk.x, kk.y), make_float2(bb.x, bb.y));
            const float2 x23 = ffma2(a23, make_float2(kk.z, kk.w), make_float2(bb.z, bb.w));
            y[4 * c4] = x01.x; y[4 * c4 + 1] = x01.y; y[4 * c4 + 2] = x23.x; y[4 * c4 + 3] = x23.y;
          }
        } else if (__any_sync(0xffffffffu, mhi != 0u)) {       // mhi == 0 only if no column is masked
#pragma unroll
          for (int c = 0; c < 64; ++c)
            if (((c < 32 ? mlo : mhi) >> (c & 31)) & 1u) y[c] = -INFINITY;
        }
        // FP8 P V: the exact running maximum is part of the arithmetic (P~ must not pass 448), so the reference moves
        // whenever the row's maximum grows, before the tile's P~ is formed: the warp waits for P V and rescales O.  (With
        // the pass repeated out of line for such tiles - at 16K two of five, counting all 32 rows of a warp - a
        // call took 5.40 ms instead of 3.12.)
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 64; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], y[c]);
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * esc;
        const bool grow = mx > m_ref;                        // also true for a row's first finite maximum
        if (__any_sync(0xffffffffu, grow)) {
          const float alpha = grow ? (m_ref == -INFINITY ? 0.f : ex2f(m_ref - mx)) : 1.f;
          ok = t == 0 || tc_rescale_o(lane_base + colO, alpha, pv_done + 2 * h + ((t - 1) & 1), (uint32_t)(((t - 1) >> 1) & 1), abort_flag);
          if (!ok) return;
          if (grow) { l *= alpha; m_ref = mx; }
        }
        const float mu = m_ref == -INFINITY ? 0.f : m_ref, off = kFp8Offset - mu;
        const float2 esc2 = make_float2(esc, esc), off2 = make_float2(off, off);
#pragma unroll
        for (int c2 = 0; c2 < 32; ++c2) {
          const float2 z = ffma2(make_float2(y[2 * c2], y[2 * c2 + 1]), esc2, off2);
          y[2 * c2] = z.x; y[2 * c2 + 1] = z.y;
        }
#pragma unroll
        for (int c = 0; c < 64; ++c) y[c] = ex2f(y[c]);
        float2 rs4[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int c2 = 0; c2 < 32; ++c2) rs4[c2 & 3] = fadd2(rs4[c2 & 3], make_float2(y[2 * c2], y[2 * c2 + 1]));
        const float2 rs2 = fadd2(fadd2(rs4[0], rs4[2]), fadd2(rs4[1], rs4[3]));
        const float lsum = rs2.x + rs2.y;
        uint32_t pk[16];
#pragma unroll
        for (int c = 0; c < 64; c += 4) pk[c >> 2] = tc::pack_e4m3x4(y[c], y[c + 1], y[c + 2], y[c + 3]);
        l += lsum;
        // P~ as e4m3 over the first 16 columns of the S buffer just read: row r in lane r, keys 4c .. 4c + 3 in column c
        tc::tmem_st16(tS, pk);
        tc::tmem_wait_st();
        tc::fence_before_sync();
        tc::mbar_arrive(p_ready + 2 * h + (t & 1));
        if (t + 1 < n_tiles) fetch(t + 1);
      };
      if (n_tiles > 0) fetch(0);
      int t = 0;
      for (; ok && t < n_rest && t < n_tiles; ++t) tile(t, TcTrue{});
      for (; ok && t < n_tiles; ++t) tile(t, TcFalse{});
    } else {
      // The softmax warps pace the kernel: a tile's pass is some 1350 clocks with the other head's warp on the scheduler, 1050 alone
      // (arithmetic 420, reads of scales and biases 256, exponentials 410, which a warp does not overlap).  Slower here: the next
      // scores asked for before the hand-over of P; four rows x sixteen columns a thread (a third of the shared-memory
      // wavefronts; 8K 650 to 685 us against 647); sixteen softmax warps, two threads per row or tiles taken in turn (773).
      float lim_sum = m_ref == -INFINITY ? -1.f : 256.f, mu = 0.f;      // a row without a reference: any sum calls for one
      auto tile = [&](int t, auto int8_tile) {
        constexpr bool is_i8 = decltype(int8_tile)::value;
        const int slot = t & 1, sl = 2 * h + slot;
        ok = mbar_wait_warp(s_full + sl, (uint32_t)((t >> 1) & 1), abort_flag);
        if (!ok) return;
        tc::fence_after_sync();
        const float esc = is_i8 ? qs : p.sml;                  // > 0
        const float4* ks4 = reinterpret_cast<const float4*>(smem + TcSmem::Ks + ks_slot * kKsBytes);
        const float4* kb4 = ks4 + 16 + 16 * h;
        if (is_i8 && ++ks_slot == kKsSlots) ks_slot = 0;
        uint32_t mlo = 0u, mhi = 0u;                           // BF16 tiles: bit c set = column c (of 64) is masked
        if (!is_i8) {
          int lim;                                             // columns <= lim are visible
          if (t < n_rest + n_vert) lim = min(64, nvh - (t - n_rest) * 64) - 1;
          else lim = min(row, p.N - 1) - (wla + (t - n_rest - n_vert) * 64);
          mlo = lim >= 31 ? 0u : lim < 0 ? 0xFFFFFFFFu : (0xFFFFFFFFu << (lim + 1));
          mhi = lim >= 63 ? 0u : lim < 32 ? 0xFFFFFFFFu : (0xFFFFFFFFu << (lim - 31));
        }
        // One fused pass per tile: score -> exponent units -> 2^(y - mu) against the reference maximum as it
        // stands -> row sum and bf16 P, two columns per instruction where the hardware has packed fp32 forms.
        // The row maximum is not computed: a P value above 2^8 would show in the row sum of the tile, which
        // is then > 2^8.  Only then (and for a row's first finite scores) the scores are read from tensor
        // memory again, the maximum is taken, O is rescaled, the reference moves and the pass is repeated.
        uint32_t pk[32];
        float lsum;
        {
          uint32_t sr[64];
          tc::tmem_ld32(lane_base + colS + slot * 64, *reinterpret_cast<uint32_t(*)[32]>(&sr[0]));
          tc::tmem_ld32(lane_base + colS + slot * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&sr[32]));
          tc::tmem_wait_ld();
          const float2 esc2 = make_float2(esc, esc), nmu2 = make_float2(-mu, -mu);
          float2 rsa = make_float2(0.f, 0.f), rsb = make_float2(0.f, 0.f);
          if constexpr (is_i8) {
            float* y = reinterpret_cast<float*>(sr);
#pragma unroll
            for (int c4 = 0; c4 < 16; ++c4) {
              const float4 kk = ks4[c4], bb = kb4[c4];
              const float2 a01 = make_float2(__int_as_float((int)sr[4 * c4] + 0x4B400000), __int_as_float((int)sr[4 * c4 + 1] + 0x4B400000));
              const float2 a23 = make_float2(__int_as_float((int)sr[4 * c4 + 2] + 0x4B400000), __int_as_float((int)sr[4 * c4 + 3] + 0x4B400000));
              const float2 y01 = ffma2(ffma2(a01, make_float2(kk.x, kk.y), make_float2(bb.x, bb.y)), esc2, nmu2);
              const float2 y23 = ffma2(ffma2(a23, make_float2(kk.z, kk.w), make_float2(bb.z, bb.w)), esc2, nmu2);
              y[4 * c4] = y01.x; y[4 * c4 + 1] = y01.y; y[4 * c4 + 2] = y23.x; y[4 * c4 + 3] = y23.y;
            }
#pragma unroll
            for (int c = 0; c < 64; ++c) y[c] = ex2f(y[c]);
            float2 rsc = make_float2(0.f, 0.f), rsd = make_float2(0.f, 0.f);
#pragma unroll
            for (int c8 = 0; c8 < 8; ++c8) {
              rsa = fadd2(rsa, make_float2(y[8 * c8], y[8 * c8 + 1]));
              rsb = fadd2(rsb, make_float2(y[8 * c8 + 2], y[8 * c8 + 3]));
              rsc = fadd2(rsc, make_float2(y[8 * c8 + 4], y[8 * c8 + 5]));
              rsd = fadd2(rsd, make_float2(y[8 * c8 + 6], y[8 * c8 + 7]));
            }
            rsa = fadd2(rsa, rsc); rsb = fadd2(rsb, rsd);
#pragma unroll
            for (int c2 = 0; c2 < 32; ++c2) {
              __nv_bfloat162 h0 = __floats2bfloat162_rn(y[2 * c2], y[2 * c2 + 1]);
              pk[c2] = *reinterpret_cast<uint32_t*>(&h0);
            }
          } else {
#pragma unroll
            for (int c2 = 0; c2 < 32; ++c2) {
              const uint32_t mw = c2 < 16 ? mlo : mhi;
              float2 y = ffma2(make_float2(__uint_as_float(sr[2 * c2]), __uint_as_float(sr[2 * c2 + 1])), esc2, nmu2);
              if ((mw >> ((2 * c2) & 31)) & 1u) y.x = -INFINITY;
              if ((mw >> ((2 * c2 + 1) & 31)) & 1u) y.y = -INFINITY;
              const float2 pp = make_float2(ex2f(y.x), ex2f(y.y));
              if (c2 & 1) rsb = fadd2(rsb, pp); else rsa = fadd2(rsa, pp);
              __nv_bfloat162 h0 = __floats2bfloat162_rn(pp.x, pp.y);
              pk[c2] = *reinterpret_cast<uint32_t*>(&h0);
            }
          }
          lsum = (rsa.x + rsa.y) + (rsb.x + rsb.y);
        }
        const bool need = !(lsum <= lim_sum);
        if (__builtin_expect(__any_sync(0xffffffffu, need), 0)) {
          // out of line: the maximum, the move of the reference and the tile's P against the new reference
          const bool wait_pv = t > 0;
          const TcSlowResult sr2 = tc_slow_tile(lane_base + colS + slot * 64, lane_base + colO, ks4, kb4, is_i8, esc, mlo, mhi, m_ref, l,
                                                wait_pv ? pv_done + 2 * h + ((t - 1) & 1) : nullptr, (uint32_t)(((t - 1) >> 1) & 1),
                                                abort_flag);
          ok = sr2.ok;
          if (!ok) return;
          m_ref = sr2.m_ref;
          l = sr2.l;
          lim_sum = m_ref == -INFINITY ? -1.f : 256.f;
          mu = m_ref == -INFINITY ? 0.f : m_ref;
        } else {
          l += lsum;
          // P over the first 32 columns of the S buffer just read: row r in lane r, keys 2c, 2c+1 in column c
          tc::tmem_st32(lane_base + colS + slot * 64, pk);
          tc::tmem_wait_st();
        }
        tc::fence_before_sync();
        tc::mbar_arrive(p_ready + sl);
      };
      int t = 0;
      const int n_i8 = min(n_rest, n_tiles);
      for (; ok && t < n_i8; ++t) tile(t, TcTrue{});
      for (; ok && t < n_tiles; ++t) tile(t, TcFalse{});
    }
    // ---- epilogue: O / l
    if (ok && n_tiles > 0)
      ok = __all_sync(0xffffffffu, tc::mbar_wait_abortable(pv_done + 2 * h + ((n_tiles - 1) & 1), (uint32_t)(((n_tiles - 1) >> 1) & 1), abort_flag));
    if (ok && n_tiles > 0) {
      tc::fence_after_sync();
      // A thread holds a row, a store wants a row on neighbouring lanes: BF16 outputs pass through the head's part of the
      // query buffer (its last product is done), sixteen-byte pieces permuted within a row so that neither side meets a
      // bank twice.  Written straight from the row's thread, a store instruction touched 32 rows: 4900
      // clocks a block, now 3400.  (With the start above: 16-bit 2 x 1973 107 -> 104 us per call.)  FP16 and FP32 outputs are
      // written from the row's thread.
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const float* vsc = kFp8 ? p.v_scale + bhk * 128 : nullptr;        // FP8 P V: the channel scales of V come back here
      const int hq = (int)(bhq - (int64_t)b * p.H_Q);
      const int64_t base = b * p.o_sb + hq * p.o_sh;
      uint8_t* stage = smem + TcSmem::Qb + h * 32768 + wq * 32 * 256;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t o[32];
        tc::tmem_ld32(lane_base + colO + ch * 32, o);
        tc::tmem_wait_ld();
        if constexpr (kFp8) {
#pragma unroll
          for (int x = 0; x < 32; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * __ldg(vsc + ch * 32 + x));
        }
        if (p.out_dtype == HQ_BF16) {
          uint32_t w[16];
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(o[2 * x]) * inv, __uint_as_float(o[2 * x + 1]) * inv);
            w[x] = *reinterpret_cast<uint32_t*>(&hh);
          }
#pragma unroll
          for (int x = 0; x < 4; ++x)
            *reinterpret_cast<uint4*>(stage + lane * 256 + (((4 * ch + x) ^ (lane & 15)) << 4)) = make_uint4(w[4 * x], w[4 * x + 1], w[4 * x + 2], w[4 * x + 3]);
        } else if (row < p.N) {
#pragma unroll
          for (int x = 0; x < 32; ++x) store_out(p.out, base + (int64_t)row * p.o_sn + ch * 32 + x, __uint_as_float(o[x]) * inv, p.out_dtype);
        }
      }
      if (p.out_dtype == HQ_BF16) {
        __syncwarp();
        const int piece = lane & 15;
#pragma unroll 4
        for (int i = lane >> 4; i < 32; i += 2) {
          const uint4 v = *reinterpret_cast<const uint4*>(stage + i * 256 + ((piece ^ (i & 15)) << 4));
          const int orow = s0 + wq * 32 + i;
          if (orow < p.N) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + base + (int64_t)orow * p.o_sn + piece * 8) = v;
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0) atomicOr(p.status, 2);
    tc_fill_nan(p, b, hkv * R + 2 * pr, plan.nheads, s0);
  }
  if (warp == 8) tc::tmem_dealloc(tmem_base, kTmemCols);
}

// ---- preparation for the tensor-memory kernel: transposed V tiles ---------------------------
// v [B,H_KV,N,128] (strided) -> vt [B,H_KV,128,Npad] bf16, columns >= N zero
__global__ void __launch_bounds__(256)
transpose_v_kernel(const __nv_bfloat16* __restrict__ v, int64_t sb, int64_t sh, int64_t sn, int H, int N, int Npad,
                   __nv_bfloat16* __restrict__ vt) {
  __shared__ __nv_bfloat16 tile[64][130];
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H, key0 = blockIdx.x * 64, tid = threadIdx.x;
  for (int x = tid; x < 64 * 16; x += 256) {
    const int r = x >> 4, c = (x & 15) * 8;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (key0 + r < N) raw = __ldg(reinterpret_cast<const uint4*>(v + b * sb + h * sh + (int64_t)(key0 + r) * sn + c));
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
    for (int j = 0; j < 8; ++j) tile[r][c + j] = e[j];
  }
  __syncthreads();
  for (int x = tid; x < 128 * 8; x += 256) {
    const int d = x >> 3, k8 = (x & 7) * 8;
    __nv_bfloat16 o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = tile[k8 + j][d];
    *reinterpret_cast<uint4*>(vt + ((int64_t)bh * 128 + d) * Npad + key0 + k8) = *reinterpret_cast<uint4*>(o);
  }
}

// gathered vertical rows: xk [B,H_Q,Tpad,128] (rows >= T zero), and of V xvt [B,H_Q,128,Tpad] (transposed), or as rows like xk
template <bool kRows>
__global__ void __launch_bounds__(256)
vertical_gather_t_kernel(const int* __restrict__ vasc, int T, int Tpad, int N, int H_Q, int H_KV,
                         const __nv_bfloat16* __restrict__ k_bf,
                         const __nv_bfloat16* __restrict__ v, int64_t v_sb, int64_t v_sh, int64_t v_sn,
                         __nv_bfloat16* __restrict__ xk, __nv_bfloat16* __restrict__ xvt) {
  __shared__ __nv_bfloat16 tile[64][130];
  const int64_t bhq = blockIdx.y;
  const int b = (int)(bhq / H_Q), hq = (int)(bhq - (int64_t)b * H_Q), hkv = hq / (H_Q / H_KV);
  const int j0 = blockIdx.x * 64, tid = threadIdx.x;
  for (int x = tid; x < 64 * 16; x += 256) {
    const int r = x >> 4, c = (x & 15) * 8;
    uint4 kr = make_uint4(0, 0, 0, 0), vr = make_uint4(0, 0, 0, 0);
    if (j0 + r < T) {
      const int src = min(max(vasc[bhq * T + j0 + r], 0), N - 1);
      kr = __ldg(reinterpret_cast<const uint4*>(k_bf + (((int64_t)b * H_KV + hkv) * N + src) * 128 + c));
      vr = __ldg(reinterpret_cast<const uint4*>(v + b * v_sb + hkv * v_sh + (int64_t)src * v_sn + c));
    }
    *reinterpret_cast<uint4*>(xk + (bhq * Tpad + j0 + r) * 128 + c) = kr;
    if constexpr (kRows) {
      *reinterpret_cast<uint4*>(xvt + (bhq * Tpad + j0 + r) * 128 + c) = vr;
      continue;
    }
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&vr);
#pragma unroll
    for (int j = 0; j < 8; ++j) tile[r][c + j] = e[j];
  }
  if constexpr (kRows) return;
  __syncthreads();
  for (int x = tid; x < 128 * 8; x += 256) {
    const int d = x >> 3, k8 = (x & 7) * 8;
    __nv_bfloat16 o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = tile[k8 + j][d];
    *reinterpret_cast<uint4*>(xvt + (bhq * 128 + d) * Tpad + j0 + k8) = *reinterpret_cast<uint4*>(o);
  }
}

int prefill_tc_launch(const hq_prefill_args* a, bool v_rows, cudaStream_t st) {
  const int N = a->N, Npad = (N + 63) / 64 * 64, T = a->T, Tpad = (T + 63) / 64 * 64;
  CUtensorMap mQi, mQb, mKi, mKb, mVt, mXk, mXv, mKs, mKbs;
  const uint64_t qrows = (uint64_t)a->B * a->H_Q * N, krows = (uint64_t)a->B * a->H_KV * N;
  int rc;
  if ((rc = tc::make_map_2d(&mQi, a->q_i8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 128, qrows, 128, 128, 128))) return rc;
  if ((rc = tc::make_map_2d(&mQb, a->q_bf, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 128, qrows, 256, 64, 128))) return rc;
  if ((rc = tc::make_map_2d(&mKi, a->k_i8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 128, krows, 128, 128, 64))) return rc;
  if ((rc = tc::make_map_2d(&mKb, a->k_bf, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 128, krows, 256, 64, 64))) return rc;
  const bool fp8 = a->pv_fp8 != 0;
  if (fp8) {       // V^T as e4m3 bytes: 64-key tiles are 64-byte rows, 64-byte swizzle
    if ((rc = tc::make_map_2d(&mVt, a->v_t8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)Npad, (uint64_t)a->B * a->H_KV * 128,
                              (uint64_t)Npad, 64, 128, 64))) return rc;
  } else if (v_rows) {
    if ((rc = tc::make_map_v_rows(&mVt, a->v_t, a->B, a->H_KV, N, a->v_sb, a->v_sh, a->v_sn))) return rc;
  } else if ((rc = tc::make_map_2d(&mVt, a->v_t, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)Npad, (uint64_t)a->B * a->H_KV * 128,
                                   (uint64_t)Npad * 2, 64, 128))) return rc;
  if ((rc = tc::make_map_2d(&mKs, a->k_scale, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)Npad, (uint64_t)a->B * a->H_KV,
                            (uint64_t)Npad * 4, 64, 1, false))) return rc;
  if ((rc = tc::make_map_2d(&mKbs, a->k_bias, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)Npad, (uint64_t)a->B * a->H_Q,
                            (uint64_t)Npad * 4, 64, 1, false))) return rc;
  if (T > 0) {
    if ((rc = tc::make_map_2d(&mXk, a->vert_k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 128, (uint64_t)a->B * a->H_Q * Tpad, 256, 64, 64))) return rc;
    if (fp8) {
      if ((rc = tc::make_map_2d(&mXv, a->vert_vt8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)Tpad, (uint64_t)a->B * a->H_Q * 128,
                                (uint64_t)Tpad, 64, 128, 64))) return rc;
    } else if (v_rows) {
      if ((rc = tc::make_map_2d(&mXv, a->vert_vt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 128, (uint64_t)a->B * a->H_Q * Tpad, 256, 64, 64))) return rc;
    } else if ((rc = tc::make_map_2d(&mXv, a->vert_vt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)Tpad, (uint64_t)a->B * a->H_Q * 128,
                                     (uint64_t)Tpad * 2, 64, 128))) return rc;
  } else {
    mXk = mKb; mXv = mVt;
  }
  PrefillTcParams p{};
  p.q_scale = a->q_scale; p.k_scale = a->k_scale; p.v_scale = a->v_scale8;
  p.nv_valid = a->nv_valid;
  p.out = a->out; p.out_dtype = a->out_dtype; p.o_sb = a->o_sb; p.o_sh = a->o_sh; p.o_sn = a->o_sn;
  p.B = a->B; p.H_Q = a->H_Q; p.H_KV = a->H_KV; p.N = N; p.Npad = Npad; p.W = a->window; p.T = T; p.Tpad = Tpad;
  p.nqb = (N + 127) / 128; p.nkb = (N + 63) / 64;
  p.sml = a->sm_scale * 1.44269504f;
  p.v_rows = v_rows;
  p.status = a->status;
  const size_t smem = TcSmem::Total + 1024;
  static thread_local int attr_dev = -1;
  int dev = 0;
  HQ_CUDA(cudaGetDevice(&dev));
  if (attr_dev != dev) {
    HQ_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HQ_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_dev = dev;
  }
  const int R = a->H_Q / a->H_KV;
  const int pairs = (R + 1) / 2;                                  // two query heads of a KV group per CTA
  // 32 MB of operands (INT8 K, BF16 V: 384 bytes a key) per group: an even finish needs a few hundred blocks in the last
  // group, which 24 to 64 MB all give
  const int64_t in_l2 = (32ll << 20) / ((int64_t)N * 384);
  const int kv_heads = a->B * a->H_KV;
  p.group = pairs * (in_l2 < 1 ? 1 : in_l2 > kv_heads ? kv_heads : (int)in_l2);
  dim3 grid((unsigned)(kv_heads * pairs * p.nqb));
  if (fp8) prefill_tc_kernel<true><<<grid, kTcThreads, smem, st>>>(mQi, mQb, mKi, mKb, mVt, mXk, mXv, mKs, mKbs, p);
  else prefill_tc_kernel<false><<<grid, kTcThreads, smem, st>>>(mQi, mQb, mKi, mKb, mVt, mXk, mXv, mKs, mKbs, p);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

// ---- FP8 P V: V^T as e4m3 with one scale per channel ----------------------------------------------------------
// The reference's per_channel_fp8 (vendor/sageattention/quant.py:134-166 with MeanScaleKernel, csrc/fused/fused.cu:318-429,
// smooth_v off): scale[b, h, d] = max_n |v[b, h, n, d]| / 448, code = e4m3(v * (448 / max)), stored transposed.
__global__ void __launch_bounds__(256)
v_amax_kernel(const __nv_bfloat16* __restrict__ v, int64_t sb, int64_t sh, int64_t sn, int H, int N, unsigned* __restrict__ amax_bits) {
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
  const int d = threadIdx.x & 127, half = threadIdx.x >> 7;
  const int rows_per = (N + gridDim.x - 1) / gridDim.x;
  const int r0 = blockIdx.x * rows_per, r1 = min(N, r0 + rows_per);
  const __nv_bfloat16* base = v + b * sb + h * sh + d;
  float m = 0.f;
  for (int r = r0 + half; r < r1; r += 2) m = fmaxf(m, fabsf(__bfloat162float(base[(int64_t)r * sn])));
  atomicMax(amax_bits + (int64_t)bh * 128 + d, __float_as_uint(m));       // non-negative floats order like their bit patterns
}

// v [B,H_KV,N,128] (strided) -> vt8 [B,H_KV,128,Npad] e4m3 (columns >= N zero), scale [B,H_KV,128] = amax / 448
__global__ void __launch_bounds__(256)
transpose_v_fp8_kernel(const __nv_bfloat16* __restrict__ v, int64_t sb, int64_t sh, int64_t sn, int H, int N, int Npad,
                       const unsigned* __restrict__ amax_bits, uint8_t* __restrict__ vt8, float* __restrict__ scale) {
  __shared__ float tile[64][129];
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H, key0 = blockIdx.x * 64, tid = threadIdx.x;
  for (int x = tid; x < 64 * 16; x += 256) {
    const int r = x >> 4, c = (x & 15) * 8;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (key0 + r < N) raw = __ldg(reinterpret_cast<const uint4*>(v + b * sb + h * sh + (int64_t)(key0 + r) * sn + c));
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
    for (int j = 0; j < 8; ++j) tile[r][c + j] = __bfloat162float(e[j]);
  }
  __syncthreads();
  for (int x = tid; x < 128 * 4; x += 256) {
    const int d = x >> 2, k16 = (x & 3) * 16;
    const float amax = __uint_as_float(amax_bits[(int64_t)bh * 128 + d]);
    const float recip = amax > 0.f ? 448.f / amax : 0.f;
    if (blockIdx.x == 0 && k16 == 0) scale[(int64_t)bh * 128 + d] = amax / 448.f;
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = tc::pack_e4m3x4(tile[k16 + 4 * j][d] * recip, tile[k16 + 4 * j + 1][d] * recip, tile[k16 + 4 * j + 2][d] * recip,
                             tile[k16 + 4 * j + 3][d] * recip);
    *reinterpret_cast<uint4*>(vt8 + ((int64_t)bh * 128 + d) * Npad + key0 + k16) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// gathered vertical-line rows of V for FP8 P V: xvt8 [B,H_Q,128,Tpad] e4m3 (transposed; columns >= T zero), quantised with
// the kv-head's channel scales like the rest of V
__global__ void __launch_bounds__(256)
vertical_gather_v_fp8_kernel(const int* __restrict__ vasc, int T, int Tpad, int N, int H_Q, int H_KV,
                             const __nv_bfloat16* __restrict__ v, int64_t v_sb, int64_t v_sh, int64_t v_sn,
                             const float* __restrict__ v_scale, uint8_t* __restrict__ xvt8) {
  __shared__ float tile[64][129];
  const int64_t bhq = blockIdx.y;
  const int b = (int)(bhq / H_Q), hq = (int)(bhq - (int64_t)b * H_Q), hkv = hq / (H_Q / H_KV);
  const int j0 = blockIdx.x * 64, tid = threadIdx.x;
  for (int x = tid; x < 64 * 16; x += 256) {
    const int r = x >> 4, c = (x & 15) * 8;
    uint4 vr = make_uint4(0, 0, 0, 0);
    if (j0 + r < T) {
      const int src = min(max(vasc[bhq * T + j0 + r], 0), N - 1);
      vr = __ldg(reinterpret_cast<const uint4*>(v + b * v_sb + hkv * v_sh + (int64_t)src * v_sn + c));
    }
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&vr);
#pragma unroll
    for (int j = 0; j < 8; ++j) tile[r][c + j] = __bfloat162float(e[j]);
  }
  __syncthreads();
  for (int x = tid; x < 128 * 4; x += 256) {
    const int d = x >> 2, k16 = (x & 3) * 16;
    const float sc = v_scale[((int64_t)b * H_KV + hkv) * 128 + d];
    const float recip = sc > 0.f ? 1.f / sc : 0.f;          // 448 / amax, the factor the V codes were formed with
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = tc::pack_e4m3x4(tile[k16 + 4 * j][d] * recip, tile[k16 + 4 * j + 1][d] * recip, tile[k16 + 4 * j + 2][d] * recip,
                             tile[k16 + 4 * j + 3][d] * recip);
    *reinterpret_cast<uint4*>(xvt8 + (bhq * 128 + d) * Tpad + j0 + k16) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

int prefill_tc_gather_v_fp8(const int32_t* vasc, int B, int H_Q, int H_KV, int N, int T, const void* v, int64_t v_sb, int64_t v_sh,
                            int64_t v_sn, const float* v_scale, void* xvt8, cudaStream_t st) {
  const int Tpad = (T + 63) / 64 * 64;
  vertical_gather_v_fp8_kernel<<<dim3(Tpad / 64, B * H_Q), 256, 0, st>>>(vasc, T, Tpad, N, H_Q, H_KV, (const __nv_bfloat16*)v, v_sb,
                                                                        v_sh, v_sn, v_scale, (uint8_t*)xvt8);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

int prefill_tc_prepare_v_fp8(const void* v, int64_t sb, int64_t sh, int64_t sn, int B, int H_KV, int N, void* v_t8, float* v_scale,
                             void* amax_scratch, cudaStream_t st) {
  const int Npad = (N + 63) / 64 * 64;
  HQ_CUDA(cudaMemsetAsync(amax_scratch, 0, (size_t)B * H_KV * 128 * 4, st));
  v_amax_kernel<<<dim3(64, B * H_KV), 256, 0, st>>>((const __nv_bfloat16*)v, sb, sh, sn, H_KV, N, (unsigned*)amax_scratch);
  transpose_v_fp8_kernel<<<dim3(Npad / 64, B * H_KV), 256, 0, st>>>((const __nv_bfloat16*)v, sb, sh, sn, H_KV, N, Npad,
                                                                   (const unsigned*)amax_scratch, (uint8_t*)v_t8, v_scale);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

int prefill_tc_prepare_v(const void* v, int64_t sb, int64_t sh, int64_t sn, int B, int H_KV, int N, void* v_t, cudaStream_t st) {
  const int Npad = (N + 63) / 64 * 64;
  transpose_v_kernel<<<dim3(Npad / 64, B * H_KV), 256, 0, st>>>((const __nv_bfloat16*)v, sb, sh, sn, H_KV, N, Npad,
                                                               (__nv_bfloat16*)v_t);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

int prefill_tc_prepare_vertical(bool rows, const int32_t* vasc, int B, int H_Q, int H_KV, int N, int T, const void* k_bf, const void* v,
                                int64_t v_sb, int64_t v_sh, int64_t v_sn, void* xk, void* xvt, cudaStream_t st) {
  const int Tpad = (T + 63) / 64 * 64;
  const auto kernel = rows ? vertical_gather_t_kernel<true> : vertical_gather_t_kernel<false>;
  kernel<<<dim3(Tpad / 64, B * H_Q), 256, 0, st>>>(vasc, T, Tpad, N, H_Q, H_KV, (const __nv_bfloat16*)k_bf, (const __nv_bfloat16*)v, v_sb,
                                                   v_sh, v_sn, (__nv_bfloat16*)xk, (__nv_bfloat16*)xvt);
  HQ_CUDA(cudaGetLastError());
  return HQ_OK;
}

}  // namespace hq
