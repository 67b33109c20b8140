// Which kernel takes a top-k call, over how many blocks a row, and with how much shared memory.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace hq {

constexpr int kTopkMaxK = 16384;
constexpr int kTopkBins = 2048;                 // counters of a radix pass
constexpr int kTopkCluster = 8;                 // most blocks per row
constexpr size_t kTopkSmem = 224 * 1024;        // most dynamic shared memory of a block

struct TopkForm {
  int blocks;       // per row: 1 = a block of 1024 threads, 4 or 8 = a cluster of blocks of 512
  int seg;          // candidates per block
  int list;         // entries a block can select, a power of two: it sorts that many
  bool kept;        // a block's keys stay in shared memory after the first pass (else they are read again from L2)
  size_t smem;
};

inline TopkForm topk_form_of(int blocks, int n, int k) {
  TopkForm f;
  f.blocks = blocks;
  f.seg = blocks == 1 ? n : ((n + blocks - 1) / blocks + 31) & ~31;
  f.list = 64;
  while (f.list < (k < f.seg ? k : f.seg)) f.list <<= 1;
  const size_t need = (size_t)f.list * 8 + (size_t)(blocks == 1 ? 1 : 2) * kTopkBins * 4, with_keys = need + (size_t)f.seg * 4;
  f.kept = with_keys <= kTopkSmem;
  f.smem = f.kept ? with_keys : need;
  return f;
}

// 1 <= k <= n, on a device of `sms` multiprocessors.  A cluster pays while all rows' clusters run at once, from 12K candidates
// on and with slices of 2K or more.  Measured (us; a block / 4 blocks / 8 blocks a row, k a twentieth where not given):
//   few rows: the clusters get an SM per block (a cluster stays within a group of some 18 SMs, so not quite all are of use).
//     8 rows of 8K 13.6 / 14.4 / 14.9, 12K 19.4 / 16.5 / 15.9, 32K 36.8 / 23.8 / 19.5, 64K with k = 16384 149 / 121 / 99;
//     32 rows of 16K 21.4 / 17.7 / 19.5, 128K 149 / 66 / 123, 64K with k = 16384 149 / 122 / 125.
//   two blocks to an SM: while the lists stay short (an eighth of the row; a block's sort and the searches of its entries in
//     the others' lists grow with them and two blocks share the SM's issue slots), and eight blocks only where two fit.
//     32 rows of 32K 36.8 / 24.2 / 24.0, 37 of 64K 76 / 47 / 55, 64 of 16K 21.5 / 20.1 / 25.9, 64 of 128K 150 / 130 / 205;
//     37 of 32K with k = 8192 69 / 84 / 83, 36 of 64K with k = 16384 149 / 231 / 206.
//   more: 74 of 16K 21.5 / 24.6 / 36.2, 148 of 32K 37 / 62 / 73.
// Two blocks a row are as many threads as one block, and more meetings: 74 rows of 16K 22.1 (one block 21.5), 148 of 32K 45 (37).
inline TopkForm topk_form(int rows, int n, int k, int sms) {
  for (int blocks = kTopkCluster; blocks >= 4; blocks >>= 1) {
    if (n < 12288 || n < 2048 * blocks) continue;
    const TopkForm f = topk_form_of(blocks, n, k);
    const int64_t all = (int64_t)rows * blocks;
    if (all <= sms - 4 * blocks) return f;
    if (k > n / 8) continue;
    if (blocks == 8 ? n >= 20480 && f.smem <= kTopkSmem / 2 && all <= 2 * sms : k <= 8192 && all <= 2 * sms - 40) return f;
  }
  return topk_form_of(1, n, k);
}

}  // namespace hq
