// Host-shape-only launch policies, shared by the C ABI and the torch operator library.  None of
// them can change a result: splits of a GEMM or of an attention call are integer partial sums.
#pragma once

#include <algorithm>
#include <cstdint>

#include "../../include/fxpr_b200.h"

namespace fxpr {

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// K-tile of a GEMM that names none (fxpr_vllm/_triton/gemm.py:26-30).
inline int default_k_tile(bool fp32) { return fp32 ? 64 : 128; }

// What the tensor-core attention route takes.  Types, geometry and alignment only, nothing of the batch but
// the grid's limits, so that a token's bits do not depend on the other requests.
struct AttnRoute {
  bool half;                                             // fp16 or bf16
  int64_t head_dim, page_size, num_heads, num_kv_heads, num_reqs;
  int64_t q_st, q_sh, kv_sblock, kv_sslot, kv_shead;     // strides in elements
  const void *q, *k, *v;
};
inline bool attention_tensor_core_route(const AttnRoute& r) {
  const int64_t g = r.num_heads / r.num_kv_heads;
  if (!r.half || (r.head_dim != 64 && r.head_dim != 128) || r.page_size % 16 != 0) return false;
  if (g != 1 && g != 2 && g != 4 && g != 8 && g != 16) return false;
  // 16-byte copies: every row must start on 16 bytes
  if ((r.q_st | r.q_sh | r.kv_sblock | r.kv_sslot | r.kv_shead) % 8 != 0) return false;
  if (((uintptr_t)r.q | (uintptr_t)r.k | (uintptr_t)r.v) & 15) return false;
  return r.num_kv_heads <= 4096 && r.num_reqs <= 65535;  // grid dimensions
}

// ---- which wide GEMM kernel, by estimated microseconds -----------------------------------------
// Above 64 rows three kernels give the same bits: 128 x 128 tiles on single SMs (gemm_tc_fast.cu, K-splits through
// scratch), 256 x 256 on pairs (gemm_tc_pair.cu, unsplit) and 256 weight columns x 96 to 256 rows on pairs
// (gemm_tc_mid.cu, up to four splits in a cluster).  The estimates are clocks per 128 of K at 1850 MHz, fitted to
// sweeps of 80 to 700 rows over ten weight shapes (within 15 % of the measured times, most within 8 %):
//   128 x 128     1300 (K-tile 128) or 1665 (64), 3.5 us a call, 8 + splits for the planes of a split, 8 for two
//                 (with 10 for two: 200 x 4096 x 14336, K-tile 64, 57.7 us in a cluster of two where planes take 55.1,
//                 299 x 3064 x 11912 59.5 unsplit and 51.9)
//   256 x 256     1936 or 2690
//   256 x rows    copies: (256 + rows) requests of 128 bytes a CTA at 2.4 clocks, 3.05 when most SMs fetch; or the
//                 conversion, 7 (14) clocks a row; 3 us a call, 8 a wave when there are several (its waves do not
//                 overlap), 2 to 4.5 for the merge
inline double est_single_us(int64_t M, int64_t N, int64_t K, int64_t k_tile, int split, int num_sms) {
  const double waves = (double)ceil_div(ceil_div(M, 128) * ceil_div(N, 128) * split, num_sms);
  return waves * ((double)K / 128 / split * (k_tile == 64 ? 1665 : 1300) / 1850) + 3.5 + (split > 2 ? 8.0 + split : split == 2 ? 8.0 : 0.0);
}
inline double est_pair_us(int64_t M, int64_t N, int64_t K, int64_t k_tile, int num_sms) {
  const double waves = (double)ceil_div(ceil_div(M, 256) * ceil_div(N, 256), std::max(1, num_sms / 2));
  return waves * ((double)K / 128 * (k_tile == 64 ? 2690 : 1936) / 1850) + 3.5;
}

// gemm_tc_mid.cu with `tiles` row tiles of `rows` rows each.
inline double est_mid_us(int64_t rows, int64_t tiles, int64_t N, int64_t K, int64_t k_tile, int split, int num_sms) {
  const int64_t cols = ceil_div(N, 256), pairs = std::max(1, num_sms / 2);
  // clusters of 4, 6 and 8 whole SMs that are resident at once: they do not pack a GPC
  const int64_t room = split == 1 ? pairs : split == 2 ? num_sms * 34 / 148 : split == 3 ? num_sms * 20 / 148 : num_sms * 14 / 148;
  const double waves = (double)ceil_div(cols * tiles, std::max<int64_t>(1, room));
  const double copies = (double)(256 + rows) * (cols * tiles * split * 2 * 3 >= num_sms * 2 ? 3.05 : 2.4);
  const double convert = (double)rows * (k_tile == 64 ? 14 : 7);
  return waves * ((double)K / 128 / split * std::max(copies, convert) / 1850 + (waves > 1 ? 8 : 3)) +
         (split == 1 ? 0.0 : split == 2 ? 2.0 : split == 3 ? 3.0 : 4.5);
}
// What conversion a call above 64 rows gets and which kernels may run it: any of the three, not the medium-batch one (a
// flag names another), or, beyond the fast conversion's range (gemm_tc_fast_supported), only the plain-conversion kernel.
enum class WideKernels { any, no_mid, plain };
inline constexpr int kFastFracBits = 21;
inline constexpr int64_t kFastKTiles = 510;              // K-tiles of an item whose 32-bit sums cannot overflow
inline WideKernels wide_kernels(int frac_bits, int flags) {
  if (frac_bits > kFastFracBits || (flags & FXPR_GEMM_FORCE_EXACT_TC)) return WideKernels::plain;
  return (flags & (FXPR_GEMM_TILE_N128 | FXPR_GEMM_PAIR)) ? WideKernels::no_mid : WideKernels::any;
}

// Row tiles of gemm_tc_mid.cu for a given split (0: it does not take the call) and their estimate.
struct MidPlan { int row_tiles; double us; };
inline int64_t mid_tile_rows(int64_t M, int64_t tiles) { return std::max<int64_t>(96, ceil_div(ceil_div(M, tiles), 32) * 32); }
inline MidPlan plan_mid_rows(int64_t M, int64_t N, int64_t K, int64_t k_tile, int split, int num_sms) {
  MidPlan best = {0, 1e30};
  if (M <= 64 || N < 128 || split < 1 || split > 4 || (k_tile != 64 && k_tile != 128)) return best;
  if (ceil_div(ceil_div(K, k_tile), split) > kFastKTiles) return best;
  // Of the tile counts that round to the same rows the fewest cost least, so six counts at most are looked at,
  // whatever M (all counts from M / 256 to M / 64 took the host 98 us at a million rows).
  for (int64_t most = split > 1 ? 128 : 256; most >= 96; most -= 32) {
    const int64_t t = ceil_div(M, most);
    if (t > 65535) break;
    const double us = est_mid_us(mid_tile_rows(M, t), t, N, K, k_tile, split, num_sms);
    if (us < best.us) best = {(int)t, us};
  }
  return best;
}
// Row tiles of gemm_tc_mid.cu when it is the kernel for the call, else 0.
inline int mid_route(int64_t M, int64_t N, int64_t K, int64_t k_tile, int split, int num_sms) {
  const MidPlan mid = plan_mid_rows(M, N, K, k_tile, split, num_sms);
  double other = est_single_us(M, N, K, k_tile, split, num_sms);
  if (split == 1) other = std::min(other, est_pair_us(M, N, K, k_tile, num_sms));
  return mid.row_tiles && mid.us < 0.95 * other ? mid.row_tiles : 0;
}

// K-split of a GEMM: split when the output tiles alone cannot fill the GPU.
inline int pick_gemm_split_k(int64_t M, int64_t N, int64_t K, int64_t k_tile, int int_bits, int num_sms,
                             WideKernels kernels = WideKernels::any) {
  if (int_bits == 16) return 1;
  const int64_t tiles = ceil_div(M, 128) * ceil_div(N, 128);
  const int64_t k_tiles = ceil_div(K, k_tile);
  if (tiles >= num_sms || k_tiles < 8) return 1;
  int split = 1;
  if (M <= 64) {
    // decode shapes (cluster merge): the largest power of two that fills the SMs once -- clusters
    // of CTAs that each take a whole SM do not pack the last tenth of the SMs -- and leaves every
    // rank at least 384 of K (below that the fixed cost of a rank wins)
    while (split < 8 && tiles * split * 2 <= num_sms * 9 / 10 && K / (split * 2) >= 384) split *= 2;
    return split;
  }
  // One wave of CTAs at most: a second, partly filled wave costs more than it hides.
  if (kernels == WideKernels::plain) {
    // this kernel's last arriver adds its planes alone (32 fraction bits, 64-bit sums, us: 80 x 768 x 4096 three splits
    // 33.9, four 32.7, eight 42.1, sixteen 64.4; 200 x 2560 x 8192 two 63.1, three 52.5, four, a second wave, 89.3;
    // 80 x 2048 x 2048, sixteen K-tiles, two 24.8, three 27.3, four 27.4)
    return (int)std::max<int64_t>(1, std::min<int64_t>(k_tiles >= 24 ? 4 : 2, num_sms / tiles));
  }
  while (split < 16 && tiles * split * 2 <= num_sms && k_tiles / (split * 2) >= 4) split *= 2;
  if (kernels != WideKernels::any) return split;
  // the splits of a cluster are cheaper to merge
  int best = split;
  double us = est_single_us(M, N, K, k_tile, split, num_sms);
  for (int s = 1; s <= 4 && k_tiles / s >= 2; ++s) {
    const MidPlan mid = plan_mid_rows(M, N, K, k_tile, s, num_sms);
    if (mid.row_tiles && mid.us < us && mid_route(M, N, K, k_tile, s, num_sms)) { best = s; us = mid.us; }
  }
  return best;
}

// KV splits of the CUDA-core attention route: an explicit request wins; otherwise split only long
// contexts on an under-filled GPU, power of two, at most 8.
inline int64_t pick_attention_splits(int64_t requested, int64_t num_requests, int64_t num_q_blocks, int64_t num_heads,
                                     int64_t num_kv_tiles, int64_t num_sms) {
  constexpr int64_t kMinTiles = 32, kMaxSplits = 8, kOversub = 2;
  if (requested >= 1) return requested;
  if (num_kv_tiles <= kMinTiles) return 1;
  if (std::max<int64_t>(1, num_requests * num_q_blocks * num_heads) > kOversub * num_sms) return 1;
  const int64_t split = std::min(num_kv_tiles / kMinTiles, kMaxSplits);
  if (split < 2) return 1;
  int64_t p = 1;
  while (p < split) p *= 2;
  return p;
}

// More ranks than every device can place as one cluster are used where this one can (`fits` asks it), else eight.
inline constexpr int kPortableRanks = 8;
template <typename Fits>
inline int ranks_that_fit(int ranks, Fits fits) {
  return ranks <= kPortableRanks || fits(ranks) ? ranks : kPortableRanks;
}

// KV splits of the tensor-core attention route, where splits are cluster ranks.  Decode keeps each
// CTA's key slice near 1024 keys (small score stash -> more resident CTAs) unless fewer clusters
// than CTA slots call for more ranks; prefill splits only when the row blocks alone cannot fill
// the SMs.
inline int64_t pick_attention_ranks(int64_t requested, int64_t num_requests, int64_t max_query_len, int64_t num_heads,
                                    int64_t num_kv_heads, int64_t max_keys, int64_t num_sms) {
  if (requested >= 1) return std::min<int64_t>(requested, 16);
  const int64_t g = num_heads / num_kv_heads;
  if (max_query_len * g <= 16) {
    // A rank's score stash must leave room for four CTAs per SM (about 19.5 KB: 19 key tiles at
    // 16 bytes per key), which sets the least rank count for long contexts.  Few clusters: enough
    // ranks to fill one wave of 4 CTAs per SM, at least two key tiles each.  Measured on 64
    // requests x 1152 keys: 8 KV heads 70 -> 63 us with 1 rank instead of 2 (when the block table
    // is no wider than that), 2 KV heads 30 -> 20.5 us with 4, 1 KV head 25 -> 16 us with 8.
    const int64_t tiles = ceil_div(max_keys, 64);
    const int64_t key_bytes = g <= 8 ? 4 * g : 64;
    const int64_t budget = 19968 + (g <= 8 ? 2048 : 0);      // eight-row Q tiles leave 2 KB more
    const int64_t cap_tiles = std::max<int64_t>(1, (budget / key_bytes) / 64);
    const int64_t need = ceil_div(tiles, cap_tiles);
    const int64_t by_keys = need > 4 ? 8 : std::max<int64_t>(1, need);
    const int64_t clusters = std::max<int64_t>(1, num_requests * num_kv_heads);
    const int64_t by_fill = std::max<int64_t>(1, std::min<int64_t>({8, (4 * num_sms) / clusters, tiles / 2}));
    // A few clusters with long contexts: sixteen, one CTA per SM (1 request x 3588 keys, 8 KV heads: 14.1 us with
    // eight, 11.3).  The width of the table stands for the contexts; short ones in a wide table lose by it (1 request in 512
    // pages, eight / sixteen ranks, us, 8 KV heads: 200 keys 5.9 / 6.7, 1000 6.8 / 7.0, 3588 12.0 / 11.0, 8000 17.4 / 13.9;
    // 2 KV heads: 5.7 / 5.9, 6.8 / 5.9, 11.5 / 9.0, 16.2 / 11.1).  Merging only the ranks that have keys gives
    // short contexts their time back and costs every other call 1 to 2 %.
    if (clusters * 16 <= num_sms && tiles >= 48) return 16;
    int64_t ranks = std::max(by_keys, by_fill);
    // No last wave of a handful of CTAs: two ranks and not three where two fit one wave at three CTAs per SM (600
    // CTAs of three against 400 of two, 25 requests x 3160 keys, 8 KV heads: 76.6 -> 56.7 us, lengths of 790 to 3160
    // 50.3 -> 43.1).  One and not two: uniform lengths gain as much, mixed ones lose (40 x 2000 74.0 -> 59.8, 400 to
    // 2000 46.2 -> 49.5; 10 x 1640 to 8192 with 32 KV heads 115 -> 162), so two stay.
    const int64_t over = clusters * ranks - 4 * num_sms;
    if (ranks > 2 && over > 0 && over * 8 < 4 * num_sms && clusters * (ranks - 1) <= 3 * num_sms &&
        ceil_div(tiles, ranks - 1) * 64 * key_bytes <= 32 * 1024)
      --ranks;
    return ranks;
  }
  const int64_t blocks = num_requests * num_kv_heads * std::max<int64_t>(1, ceil_div(max_query_len * g, 64));
  if (blocks >= num_sms || max_keys <= 2048) return 1;
  return std::max<int64_t>(1, std::min<int64_t>(8, num_sms / blocks));
}

}  // namespace fxpr
