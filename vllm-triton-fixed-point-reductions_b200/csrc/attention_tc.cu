// Prefill attention on the 5th-generation tensor cores (sm_100a): TMA-fed tcgen05.mma with
// the score tile and the per-tile P.V partial in tensor memory.
//
// Semantics: the fused kernel of the reference, fxpr_vllm/_triton/attention.py:127-301 --
// pass A finds the exact row maxima of s = (q.k) * scale * log2(e) (+ soft-cap, ALiBi, masks),
// pass B recomputes s, forms w = exp2(s - max), sums Q(w) into an integer denominator and,
// per 64-key tile, Q(P.V) with P = w rounded to the io dtype into an integer numerator
// (:259-290); out = num / max(den, 1e-6).  Key tiles are 64 wide from key 0.
//
// Bit compatibility: a tcgen05.mma kind::f16 chain of 16-deep steps in ascending k gives the
// same fp32 bits as the mma.sync.m16n8k16 chain of attention_mma.cu (measured on a B200:
// every element of 128 x 128 x {64, 128} products identical), ex2.approx and the roundings
// are the same instructions, so this kernel's outputs equal that kernel's bit for bit --
// which keeps "a token's bits do not depend on whether it was computed in a prefill block or
// a decode step" (the decode kernel stays on mma.sync) and is what the tests assert.
//
// One CTA = 128 query rows of one KV head: a row is a (token, query head of the GQA group)
// pair, so a K/V tile is fetched once for the whole group.  Roles:
//   producers   two warps: Q by one box per item, K / V pages by one box per page piece (16 or 64
//               slots) and whole head, 128-byte swizzle (attn_kv_map)
//   issuer      one warp: S = Q.K^T (128 x 64 per tile, two tiles ahead in pass B) and P.V (128 x 128,
//               a fresh accumulator per tile), P read from shared memory where the softmax warps put it
//   softmax     two groups of four warps, a thread is one row, a group takes every other key tile.
//               Pass A: row maxima straight from tensor memory, 128 keys a step (a row lives in one
//               lane: no shuffles).  Pass B: weights, integer denominator, P -> shared memory
//   conversion  eight warps: P.V partials to Q-format on the FP32 and integer pipes (packed add of
//               1.5 * 2^(23-f), raw bits summed in 32-bit registers, magnitude screen, exact fix-up
//               from tensor memory) while the other roles work on the next tiles.
// Bound: the softmax groups, as chains of dependent steps and not by any unit's rate.  A tile takes an SM about
// 2430 clocks (its tensor work is 768); a group spends 4860 clocks on a tile of its own and the other group's, of
// which 2050 make weights and P, 565 maxima, 1420 are waits for scores and buffers, and the MMA warp waits for
// copies a tenth of the time.  Issue slots are half busy, ALU 40 %, MUFU 28 %, tensor pipe 27 %.
// 16 prompts of 128 to 4096 tokens, 32/8 heads: 2570 -> 1410 us.
// KV splits are not handled here (the dispatcher sends them to attention_mma.cu: same bits).
// Every wait is bounded; on a time-out the CTA sets the status word and leaves.
#include <algorithm>
#include <type_traits>

#include <cuda.h>

#include "attention_common.cuh"
#include "fxp_common.cuh"
#include "tc_common.cuh"
#include "gemm_tc_fast_common.cuh"

namespace fxpr {

static constexpr int kTcTileN = 64;            // keys per tile (attention.py:32-36)
static constexpr int kTcRows = 128;            // query rows per CTA = tensor-memory lanes
static constexpr int kTcGroupWarps = 4;        // softmax group: thread = one row, all keys of every other tile
static constexpr int kTcSoftWarps = 2 * kTcGroupWarps;
static constexpr int kTcConvWarps = 8;         // conversion: thread = one row and half of the output columns
static constexpr int kTcFirstSoft = 2;         // warp 0: TMA producer, warp 1: MMA issuer
static constexpr int kTcFirstConv = kTcFirstSoft + kTcSoftWarps;
static constexpr int kTcFirstMore = kTcFirstConv + kTcConvWarps;   // further producer warps
static constexpr int kTcProducers = 2;
static constexpr int kTcThreads = (kTcFirstMore + kTcProducers - 1) * 32;
static constexpr int kTcStages = 4;

struct TcAttnShape {
  int rows_per_token;      // GQA group size
  int tokens_per_block;    // 128 / rows_per_token
  int num_q_blocks;
  int page_size;
  int group_shift;         // log2 of the keys per TMA box: 6 when pages are multiples of 64 tokens, else 4
  int page_mask;           // page_size - 1 when the page size is a power of two, else 0
  int head_chunks;         // 64-element chunks from one KV head to the next
  uint32_t idesc_s, idesc_s2, idesc_pv;    // S of 64 keys, S of 128 keys, P.V
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z,
                                            uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];\n\t}"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(elected) : "memory");
}
__device__ __forceinline__ float ex2_approx_tc(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
template <typename T> __device__ __forceinline__ uint32_t pack2_tc(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2_tc<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack2_tc<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <typename T, int HD>
__global__ void __launch_bounds__(kTcThreads, 1)
attn_tc_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const AttnParams p, const TcAttnShape sh,
                       int32_t* status, const int zero /* always 0: keeps the side arrays in local memory */) {
  static_assert(HD == 128, "head size 128");
  constexpr int kQBytes = kTcRows * HD * 2;                // 32 KB: two 64-dim slabs of 128 rows x 128 B
  constexpr int kKBytes = kTcTileN * HD * 2;               // 16 KB: two slabs of 64 keys x 128 B
  constexpr int kStageBytes = 2 * kKBytes;                 // K then V
  constexpr int kPBytes = kTcRows * kTcTileN * 2;          // 16 KB: 128 rows x 128 B
  constexpr int kBarOffset = kQBytes + kTcStages * kStageBytes + 2 * kPBytes;
  constexpr int kHalfCols = HD / 2;                        // P.V columns per conversion thread
  constexpr uint32_t kColS = 0, kColPV = 256;              // tensor-memory columns: S[2] x 128, PV[2] x 128

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t q_s = smem_base, stage0 = smem_base + kQBytes, p_s0 = stage0 + kTcStages * kStageBytes;
  const uint32_t bar_base = smem_base + kBarOffset;
  // barriers: qfull | full[4] empty[4] | sfull[2] sfree[2] | pready[2] | pvfull[2] pvfree[2] | sync | qfree |
  // denfull[2] denfree[2]
  const uint32_t qfull = bar_base, full0 = bar_base + 8, empty0 = full0 + 8 * kTcStages;
  const uint32_t sfull0 = empty0 + 8 * kTcStages, sfree0 = sfull0 + 16, pready0 = sfree0 + 16;
  const uint32_t pvfull0 = pready0 + 16, pvfree0 = pvfull0 + 16, soft_bar = pvfree0 + 16;
  const uint32_t qfree = soft_bar + 8, denfull0 = qfree + 8, denfree0 = denfull0 + 16;
  constexpr int kMisc = 8 * (1 + 2 * kTcStages + 10 + 2 + 4);
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem_gen + kBarOffset + kMisc);
  volatile int* abort_flag = (volatile int*)(smem_gen + kBarOffset + kMisc + 8);
  float* rmax_s = (float*)(smem_gen + kBarOffset + kMisc + 16);                 // [item parity][group][128]
  long long* den_s = (long long*)(smem_gen + kBarOffset + kMisc + 16 + 2048);   // [item parity][group][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // ---- work items ---------------------------------------------------------------------
  // Persistent CTAs over the padded list (request, row block, KV head), later row blocks (more keys)
  // first, dealt out there and back again: straight round robin gives the first CTAs the longer item of
  // every round (16 prompts of 128 to 4096 tokens: the busiest SM 15 % over the mean, 4 % this way).
  // Drawing items from a counter in global memory balances better still but was slower (16 x 2048 tokens
  // 1354 against 1223 us): the CTAs then stay in step and read the same cache lines at the same time.
  // Every role walks the same list and keeps its ring positions and barrier phases running from one item
  // to the next, so the producers fetch the next item's Q and first keys and the MMA warp starts its
  // scores while the conversion warps still finish the current item.
  auto item_of = [&](int r) -> int {
    return r * (int)gridDim.x + (r & 1 ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };
  const int hkv = p.num_kv_heads;
  const int G = sh.rows_per_token;
  const int items_per_req = sh.num_q_blocks * hkv;
  const int total_items = items_per_req * p.num_reqs;
  struct Item { int live, req, kvh, q_start, q_len, tok0, seq_len, ctx, t0, t1; };
  auto decode_item = [&](int w) -> Item {
    Item I;
    I.req = w / items_per_req;
    const int rem = w - I.req * items_per_req;
    const int qb = sh.num_q_blocks - 1 - rem / hkv;
    I.kvh = rem % hkv;
    I.q_start = p.qsl[I.req];
    I.q_len = p.qsl[I.req + 1] - I.q_start;
    I.tok0 = qb * sh.tokens_per_block;
    I.live = I.tok0 < I.q_len;
    I.seq_len = I.live ? p.seq_lens[I.req] : 0;
    I.ctx = I.seq_len - I.q_len;
    const int tok_end = min(I.q_len, I.tok0 + sh.tokens_per_block);
    const int hi_key = p.causal ? min(I.seq_len, I.ctx + tok_end) : I.seq_len;
    const int lo_key = p.window > 0 ? max(0, I.ctx + I.tok0 - p.window + 1) : 0;
    I.t0 = lo_key / kTcTileN;
    I.t1 = max(I.t0, (hi_key + kTcTileN - 1) / kTcTileN);
    return I;
  };

  if (threadIdx.x == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
  }
  if (threadIdx.x == 0) {
    mbar_init(qfull, 1);
    mbar_init(qfree, 1);
    for (int s = 0; s < kTcStages; ++s) { mbar_init(full0 + 8u * s, kTcProducers); mbar_init(empty0 + 8u * s, 1); }
    for (int b = 0; b < 2; ++b) {
      mbar_init(sfull0 + 8u * b, 1); mbar_init(sfree0 + 8u * b, kTcGroupWarps);
      mbar_init(pready0 + 8u * b, kTcGroupWarps);
      mbar_init(pvfull0 + 8u * b, 1); mbar_init(pvfree0 + 8u * b, kTcConvWarps);
      mbar_init(denfull0 + 8u * b, kTcSoftWarps); mbar_init(denfree0 + 8u * b, kTcConvWarps);
    }
    mbar_init(soft_bar, kTcSoftWarps);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32((const void*)tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0 || warp >= kTcFirstMore) {
    // ------------------------------ K / V producers (TMA) -----------------------------
    // A box is a 16-token page piece, or a whole 64-key tile when pages are multiples of 64 tokens, with
    // all 128 head dims: [8-row group][64-dim half][8 rows][128 B], 4 or 16 KB.  The 8-row swizzle atoms
    // of one half then lie 2 KB apart whatever the page size, which is all the MMA descriptors need.
    // A 4 KB box takes the copy unit ~100 clocks and its warp about as long again for coordinates and
    // barriers, with 20 warps on the SM: two warps share the eight boxes of a stage, compute their
    // coordinates before they wait for it, and run loops without run-time choices.  (One warp with boxes
    // of one half head, twice as many: 1760 clocks per stage, which bounded the kernel.)
    // A stage is 32 KB: 128 keys of K in pass A, 64 keys of K and V in pass B.  Nothing is copied,
    // and the block table is not read, past the end of the sequence; V rows there are cleared by the
    // MMA warp before P.V.
    const uint32_t e = elect_one();
    const int me = warp == 0 ? 0 : warp - kTcFirstMore + 1;
    int stage = 0; uint32_t phase = 1;
    uint32_t q_phase = 1;                                    // qfree: the first wait passes
    // Block-table entries are read 32 at a time (lane L: the 16-key group L of an 8-tile block), one
    // block ahead of their use, and handed round by shuffle.
    int page_shift = -1;
    for (int b = 4; b < 31; ++b) if ((1 << b) == sh.page_size) page_shift = b;
    for (int r = 0, w = blockIdx.x; w < total_items; w = item_of(++r)) {
      const Item I = decode_item(w);
      if (!I.live) continue;
      const int kvh = I.kvh, seq_len = I.seq_len, t0 = I.t0, t1 = I.t1;
      const int32_t* bt = p.block_table + (int64_t)I.req * p.bt_stride;
      // Q rows: box {64 dims, G heads, 128 / G tokens} -> row = token * G + head.  Tokens past this
      // request's (they belong to the next one, or lie beyond the tensor: zeros) are rows whose every
      // key is masked and that are never stored.  The buffer is free once the MMA warp's last score
      // MMA of the previous item has completed.
      if (me == 0) {
        if (!__all_sync(0xffffffffu, mbar_wait(qfree, q_phase, abort_flag))) goto producer_done;
        q_phase ^= 1;
        mbar_expect_tx(qfull, kQBytes, e);
        tma_load_3d(q_s, &map_q, qfull, 0, kvh * G, I.q_start + I.tok0, e);
        tma_load_3d(q_s + kQBytes / 2, &map_q, qfull, 64, kvh * G, I.q_start + I.tok0, e);
      }
      auto load_entries = [&](int tb) -> int {
        const int n = tb * kTcTileN + lane * 16;
        return (tb < t1 && n < seq_len) ? bt[page_shift >= 0 ? (n >> page_shift) : (n / sh.page_size)] : 0;
      };
      // one pass over the item's tiles; PASS and GS (log2 of the keys per box) are compile-time
      auto walk = [&](auto pass_c, auto gs_c) -> bool {
        constexpr int PASS = decltype(pass_c)::value, GS = decltype(gs_c)::value;
        constexpr int kStep = PASS ? 1 : 2;                  // tiles per stage
        constexpr int kPieces = (kStep * kTcTileN) >> GS;    // page pieces of K (and of V) per stage
        constexpr int kBoxes = kPieces << PASS;              // box q: piece q of K, or piece q / 2 of K (even q) and V
        constexpr int kMine = (kBoxes + kTcProducers - 1) / kTcProducers;
        int cur = load_entries(t0);
        for (int tb = t0; tb < t1; tb += 8) {
          const int nxt = load_entries(tb + 8);
          for (int tt = 0; tt < 8 && tb + tt < t1; tt += kStep) {
            const int n0 = (tb + tt) * kTcTileN;
            // only pieces that start inside the sequence (pass A: and before t1) are copied
            const int pieces = (min(seq_len, t1 * kTcTileN) - n0 + (1 << GS) - 1) >> GS;
            int blk[kMine], row8[kMine];
            uint32_t bytes = 0;
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
              const int q = me + i * kTcProducers, piece = PASS ? q >> 1 : q;
              blk[i] = __shfl_sync(0xffffffffu, cur, (tt * 4 + (piece << (GS - 4))) & 31);
              const int n = n0 + (piece << GS);
              row8[i] = (sh.page_mask ? (n & sh.page_mask) : (n % sh.page_size)) >> 3;
              if (q < kBoxes && piece < pieces) bytes += 256u << GS;
            }
            if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8u * stage, phase, abort_flag))) return false;
            const uint32_t fb = full0 + 8u * stage, ks = stage0 + stage * kStageBytes;
            mbar_expect_tx(fb, bytes, e);
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
              const int q = me + i * kTcProducers, piece = PASS ? q >> 1 : q;
              const bool v = PASS && (q & 1);
              if (q < kBoxes && piece < pieces)
                tma_load_5d(ks + (uint32_t)((v ? kKBytes : 0) + (piece << (GS + 8))), v ? &map_v : &map_k, fb, 0, 0,
                            kvh * sh.head_chunks, row8[i], blk[i], e);
            }
            if (++stage == kTcStages) { stage = 0; phase ^= 1; }
          }
          cur = nxt;
        }
        return true;
      };
      using std::integral_constant;
      const bool fetched = sh.group_shift == 4
          ? walk(integral_constant<int, 0>{}, integral_constant<int, 4>{}) && walk(integral_constant<int, 1>{}, integral_constant<int, 4>{})
          : walk(integral_constant<int, 0>{}, integral_constant<int, 6>{}) && walk(integral_constant<int, 1>{}, integral_constant<int, 6>{});
      if (!fetched) goto producer_done;
    }
  producer_done:;
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ----------------------------------------
    // S = Q . K^T: both operands K-major (head dim contiguous); Q in two slabs of 64 dims, K with the two
    // halves of every 8-row group side by side
    const uint32_t e = elect_one();
    auto issue_s = [&](int stage, int sbuf, uint32_t idesc) {
      const uint32_t d = tmem_base + kColS + (uint32_t)(sbuf * 128);
      const uint64_t qd = make_smem_desc(q_s, 16, 1024);
      const uint64_t kd = make_smem_desc(stage0 + stage * kStageBytes, 16, 2048);
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
        const uint64_t ao = (uint64_t)((kk >> 2) * (kQBytes / 2) + (kk & 3) * 32) >> 4;
        const uint64_t bo = (uint64_t)((kk >> 2) * 1024 + (kk & 3) * 32) >> 4;
        umma_f16(d, qd + ao, kd + bo, idesc, kk ? 1u : 0u, e);
      }
      umma_commit(sfull0 + 8u * sbuf, e);
    };
    int stage = 0; uint32_t phase = 0;
    int it = 0;                                              // S products issued so far (all items, both passes)
    int jg = 0;                                              // P.V tiles issued so far (all items)
    uint32_t q_phase = 0;
    for (int r = 0, w = blockIdx.x; w < total_items; w = item_of(++r)) {
    const Item I = decode_item(w);
    if (!I.live) continue;
    const int seq_len = I.seq_len, t0 = I.t0, t1 = I.t1, n_tiles = I.t1 - I.t0;
    bool okq = mbar_wait(qfull, q_phase, abort_flag);
    if (!__all_sync(0xffffffffu, okq)) goto issuer_done;
    q_phase ^= 1;
    {
      // pass A: scores only, 128 keys at a time
      for (int t = t0; t < t1; t += 2, ++it) {
        const int sb = it & 1; const uint32_t sph = ((it >> 1) & 1) ^ 1;
        const bool a = mbar_wait(full0 + 8u * stage, phase, abort_flag);
        const bool b = mbar_wait(sfree0 + 8u * sb, sph, abort_flag);
        if (!__all_sync(0xffffffffu, a && b)) goto issuer_done;
        tc_fence_after();
        issue_s(stage, sb, sh.idesc_s2);
        umma_commit(empty0 + 8u * stage, e);
        if (++stage == kTcStages) { stage = 0; phase ^= 1; }
      }
      // pass B: S runs two tiles ahead of P.V, one for each softmax group
      int s_stage = stage; uint32_t s_phase = phase;         // ring position of the next S tile
      auto issue_s_next = [&]() -> bool {
        const int sb = it & 1; const uint32_t sph = ((it >> 1) & 1) ^ 1;
        const bool a = mbar_wait(full0 + 8u * s_stage, s_phase, abort_flag);
        const bool b = mbar_wait(sfree0 + 8u * sb, sph, abort_flag);
        if (!__all_sync(0xffffffffu, a && b)) return false;
        tc_fence_after();
        issue_s(s_stage, sb, sh.idesc_s);
        ++it;
        if (++s_stage == kTcStages) { s_stage = 0; s_phase ^= 1; }
        return true;
      };
      for (int j = 0; j < 2 && j < n_tiles; ++j)
        if (!issue_s_next()) goto issuer_done;
      if (n_tiles <= 2) umma_commit(qfree, e);               // the item's last score MMA is issued
      for (int j = 0; j < n_tiles; ++j, ++jg) {
        if (j + 2 < n_tiles) {
          if (!issue_s_next()) goto issuer_done;
          if (j + 3 == n_tiles) umma_commit(qfree, e);
        }
        const int b = jg & 1; const uint32_t ph = (jg >> 1) & 1;
        const bool r1 = mbar_wait(pready0 + 8u * b, ph, abort_flag);
        const bool r2 = mbar_wait(pvfree0 + 8u * b, ph ^ 1, abort_flag);
        if (!__all_sync(0xffffffffu, r1 && r2)) goto issuer_done;
        tc_fence_after();
        {
          // Keys at or past the end of the sequence: their V rows were not copied (or come
          // from slots nobody wrote) and 0 * NaN would poison the accumulator, so the rows
          // are cleared.  Only the last tile of a sequence has any.
          const int r0 = seq_len - (t0 + j) * kTcTileN;
          if (r0 < kTcTileN) {
            const uint32_t vs = stage0 + stage * kStageBytes + kKBytes;
            for (int idx = lane; idx < (kTcTileN - r0) * 16; idx += 32) {
              const int rr = r0 + (idx >> 4), cc = idx & 15;
              const uint32_t addr = vs + (uint32_t)((rr >> 3) * 2048 + (cc >> 3) * 1024 + (rr & 7) * 128 + (cc & 7) * 16);
              asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0) : "memory");
            }
            fence_proxy_async_smem();
            __syncwarp();
          }
        }
        // PV_j = P_j . V_j: P K-major (keys contiguous), V MN-major (head dim contiguous)
        const uint32_t d = tmem_base + kColPV + (uint32_t)(b * HD);
        const uint64_t pd = make_smem_desc(p_s0 + b * kPBytes, 16, 1024);
        const uint64_t vd = make_smem_desc(stage0 + stage * kStageBytes + kKBytes, 1024, 2048);
#pragma unroll
        for (int kk = 0; kk < kTcTileN / 16; ++kk)
          umma_f16(d, pd + (uint64_t)(kk * 2), vd + (uint64_t)(kk * 256), sh.idesc_pv, kk ? 1u : 0u, e);
        umma_commit(pvfull0 + 8u * b, e);
        umma_commit(empty0 + 8u * stage, e);
        if (++stage == kTcStages) { stage = 0; phase ^= 1; }
      }
    }
    }
  issuer_done:;
  } else if (warp < kTcFirstConv) {
    // ------------------------------ softmax warps -------------------------------------
    const int quarter = warp & 3;
    // Two groups take the score products in turn (group = product number & 1 = S buffer): while one
    // loads or waits, the other keeps the exponential unit busy.
    const int group = (warp - kTcFirstSoft) >> 2;
    const int row = quarter * 32 + lane;                     // tensor-memory lane = query row
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    const float ninf = -__int_as_float(0x7f800000);
    const bool plain_scores = !(p.cap_log2 > 0.0f) && p.alibi == nullptr;
    const bool raw_max = plain_scores && p.ss_log2 > 0.0f;
    const uint64_t zero2 = pack2((uint32_t)zero, (uint32_t)zero);
    const uint64_t ss2 = pack2(__float_as_uint(p.ss_log2), __float_as_uint(p.ss_log2));
    const uint32_t mbits = q_magic_bits(p.inv_scale);
    const uint64_t magic2 = pack2(mbits, mbits);
    uint32_t soft_phase = 0;
    bool ok = true;
    auto soft_sync = [&]() -> bool {                         // bounded barrier over these 8 warps
      __syncwarp();
      if (lane == 0) mbar_arrive(soft_bar);
      const bool done = warp_wait(soft_bar, soft_phase, abort_flag);
      soft_phase ^= 1;
      return done;
    };
    int it = 0;                                              // S products consumed so far (all items, both passes)
    int jg = 0;                                              // P tiles of the items before this one
    int k = -1;                                              // live items so far
    for (int r = 0, w = blockIdx.x; w < total_items && ok; w = item_of(++r)) {
    const Item I = decode_item(w);
    if (!I.live) continue;
    ++k;
    const int kvh = I.kvh, q_len = I.q_len, tok0 = I.tok0, seq_len = I.seq_len, ctx = I.ctx;
    const int t0 = I.t0, t1 = I.t1, n_tiles = I.t1 - I.t0;
    const int tok = tok0 + row / G, head = kvh * G + row % G;
    const bool valid = tok < q_len;
    const int pos = ctx + tok;
    const int kend = valid ? (p.causal ? min(seq_len, pos + 1) : seq_len) : 0;
    const int kbeg = valid ? (p.window > 0 ? max(0, pos - p.window + 1) : 0) : 0;
    const float slope = (p.alibi && valid) ? p.alibi[head] : 0.0f;
    // one score in log2 space with soft-cap and ALiBi (attention.py:103-121, 249-254)
    auto score = [&](uint32_t v, int n) -> float {
      float x = __fmul_rn(__uint_as_float(v), p.ss_log2);
      if (p.cap_log2 > 0.0f) x = __fmul_rn(p.cap_log2, tanhf(__fdiv_rn(x, p.cap_log2)));
      if (p.alibi) x = __fadd_rn(x, __fmul_rn(slope, __fsub_rn((float)n, (float)pos)));
      return x;
    };
    // hand S buffer sb back to the MMA warp (this warp's share is in registers)
    auto release_s = [&](int sb) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sfree0 + 8u * sb);
    };

    // =============================== pass A: row maxima ===============================
    // 128 keys per step, all of them in one thread.  Scaling by a positive constant is monotonic after rounding
    // too, so the maximum is taken over the raw products and scaled once.
    float rmax = ninf;
    for (int t = t0; t < t1 && ok; t += 2, ++it) {
      const int sb = it & 1;
      if (sb != group) continue;
      if (!warp_wait(sfull0 + 8u * sb, (it >> 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      float m = ninf;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld32(tmem_base + lane_sel + kColS + (uint32_t)(sb * 128 + c * 32), v);
        tmem_wait_ld_regs(v);
        if (c == 3) release_s(sb);
        const int n0 = t * kTcTileN + c * 32;
        const bool inside = n0 >= kbeg && n0 + 32 <= kend;
        if (raw_max) {
          if (inside) {
            float m1 = ninf;                                 // two chains
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              m = max3(m, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
              m1 = max3(m1, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
            }
            m = fmaxf(m, m1);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (n0 + i >= kbeg && n0 + i < kend) m = fmaxf(m, __uint_as_float(v[i]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (n0 + i >= kbeg && n0 + i < kend) m = fmaxf(m, score(v[i], n0 + i));
        }
      }
      rmax = fmaxf(rmax, raw_max ? __fmul_rn(m, p.ss_log2) : m);
    }
    float* rmax_k = rmax_s + (k & 1) * (2 * kTcRows);
    rmax_k[group * kTcRows + row] = rmax;
    if (ok && !soft_sync()) ok = false;
    float gmax = fmaxf(rmax_k[row], rmax_k[kTcRows + row]);
    if (gmax == ninf) gmax = 0.0f;                           // rows without keys: exp2 gives 0, not NaN

    // =============================== pass B ===========================================
    uint32_t den32 = 0;
    const uint64_t neg_max2 = pack2(__float_as_uint(-gmax), __float_as_uint(-gmax));
    int mine = 0;                                            // tiles of this group
    for (int j = 0; j < n_tiles && ok; ++j, ++it) {
      const int t = t0 + j;
      const int sb = it & 1;
      if (sb != group) continue;
      ++mine;
      if (!warp_wait(sfull0 + 8u * sb, (it >> 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const int g = jg + j, b = g & 1;
      const uint32_t prow = p_s0 + b * kPBytes + (uint32_t)row * 128u;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[32];
        tmem_ld32(tmem_base + lane_sel + kColS + (uint32_t)(sb * 128 + h * 32), v);
        tmem_wait_ld_regs(v);
        if (h == 1) release_s(sb);
        // d = score - max, rounded twice; the product is an fma with a run-time zero because the
        // assembler contracts a packed multiply and the packed add behind it into one rounding.
        // The weight of a masked key is exp2(-inf) = 0.
        const int n0 = t * kTcTileN + h * 32;
        const bool inside = n0 >= kbeg && n0 + 32 <= kend;
        if (plain_scores) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            uint64_t x;
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(x) : "l"(pack2(v[i], v[i + 1])), "l"(ss2), "l"(zero2));
            asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(neg_max2));
            asm("mov.b64 {%0, %1}, %2;" : "=r"(v[i]), "=r"(v[i + 1]) : "l"(x));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__fsub_rn(score(v[i], n0 + i), gmax));
        }
        if (!inside) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (n0 + i < kbeg || n0 + i >= kend) v[i] = __float_as_uint(ninf);
        }
        // weights, integer denominator, P in the io dtype -> shared memory (A operand of P.V):
        // row = 128 bytes of 64 keys, 16-byte chunks XOR-swizzled with the row number
        // (its buffer is free once the P.V product two tiles back has completed)
        if (h == 0 && g >= 2 && !warp_wait(pvfull0 + 8u * b, ((g - 2) >> 1) & 1, abort_flag)) { ok = false; break; }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float w0 = ex2_approx_tc(__uint_as_float(v[c * 8 + e * 2]));
            const float w1 = ex2_approx_tc(__uint_as_float(v[c * 8 + e * 2 + 1]));
            uint64_t q;
            asm("add.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(pack2(__float_as_uint(w0), __float_as_uint(w1))), "l"(magic2));
            den32 = den32 + (uint32_t)q + (uint32_t)(q >> 32);
            pk[e] = pack2_tc<T>(w0, w1);
          }
          const uint32_t addr = prow + (((uint32_t)(h * 4 + c) ^ (uint32_t)(row & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(pk[0]), "r"(pk[1]), "r"(pk[2]), "r"(pk[3]) : "memory");
        }
      }
      if (!ok) break;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(pready0 + 8u * b);
    }
    if (!ok) break;
    jg += n_tiles;
    // 64 weights per tile went through the packed add in this thread
    if (!warp_wait(denfree0 + 8u * (k & 1), ((k >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
    den_s[(k & 1) * (2 * kTcRows) + group * kTcRows + row] =
        (long long)(int32_t)(den32 - (uint32_t)kTcTileN * (uint32_t)mine * mbits);
    __syncwarp();
    if (lane == 0) mbar_arrive(denfull0 + 8u * (k & 1));
    }
  } else {
    // ------------------------------ conversion warps ----------------------------------
    // Round every P.V partial to Q-format, add, and store the finished rows; the softmax warps are by
    // then in the next item's maximum pass.
    const int quarter = warp & 3;
    const int half = (warp - kTcFirstConv) >> 2;             // which half of the output columns
    const int row = quarter * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    const uint32_t mbits = q_magic_bits(p.inv_scale), one = (uint32_t)zero + 1u;
    const uint64_t magic2 = pack2(mbits, mbits);
    const float screen_limit = q_screen_limit(p.inv_scale);
    int jg = 0;                                              // P.V tiles converted so far (all items)
    int k = -1;                                              // live items so far
    bool ok = true;
    for (int r = 0, w = blockIdx.x; w < total_items && ok; w = item_of(++r)) {
      const Item I = decode_item(w);
      if (!I.live) continue;
      ++k;
      const int n_tiles = I.t1 - I.t0;
      uint32_t acc[kHalfCols];
#pragma unroll
      for (int i = 0; i < kHalfCols; ++i) acc[i] = 0;
      uint32_t corr_raw[kHalfCols];                          // rare path, local memory
      long long corr_q[kHalfCols];
      bool corr_used = false;
      for (int j = 0; j < n_tiles; ++j, ++jg) {
        const int b = jg & 1;
        if (!warp_wait(pvfull0 + 8u * b, (jg >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + lane_sel + kColPV + (uint32_t)(b * HD + half * kHalfCols);
        float screen = 0.0f, tail = 0.0f;
#pragma unroll
        for (int c = 0; c < kHalfCols; c += 16) {
          uint32_t v[16];
          tmem_ld16(taddr + c, v);
          tmem_wait_ld_regs(v);
          if (c + 16 == kHalfCols) {
            // the last chunk is in registers: screen it and hand the buffer back before converting it
#pragma unroll
            for (int i = 0; i < 16; i += 2) screen = max3_abs(screen, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
            if (__any_sync(0xffffffffu, !(screen < screen_limit))) {
              // some partial left the fast range: exact conversion of the offending elements
              if (!corr_used) {
#pragma unroll 1
                for (int z = 0; z < kHalfCols; ++z) { corr_raw[z + zero] = 0; corr_q[z + zero] = 0; }
                corr_used = true;
              }
              fixup_tile(taddr, kHalfCols, mbits, p.scale, p.int_bits, &corr_raw[zero], &corr_q[zero]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(pvfree0 + 8u * b);
          }
          convert16(v, &acc[c], magic2, mbits, one, c + 16 == kHalfCols ? tail : screen);
        }
      }
      if (!ok) break;
      if (!warp_wait(denfull0 + 8u * (k & 1), (k >> 1) & 1, abort_flag)) { ok = false; break; }
      const long long dsum = den_s[(k & 1) * (2 * kTcRows) + row] + den_s[(k & 1) * (2 * kTcRows) + kTcRows + row];
      __syncwarp();
      if (lane == 0) mbar_arrive(denfree0 + 8u * (k & 1));
      const int tok = I.tok0 + row / G, head = I.kvh * G + row % G;
      if (tok < I.q_len) {
        const float dn = fmaxf(fixed_to_float<long long>(wrap_to_bits(dsum, p.int_bits), p.inv_scale), 1.0e-6f);
        T* op = (T*)p.o + (int64_t)(I.q_start + tok) * p.o_st + (int64_t)head * p.o_sh + half * kHalfCols;
        const uint32_t bias_bits = (uint32_t)n_tiles * mbits;   // what the multiply-adds summed on top
#pragma unroll
        for (int g8 = 0; g8 < kHalfCols / 8; ++g8) {
          alignas(16) T out[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int c = g8 * 8 + i;
            uint32_t raw = alu_add(c) ? acc[c] : acc[c] - bias_bits;
            float num;
            if (corr_used) {
              raw -= corr_raw[c + zero];
              const long long tot = (long long)(int32_t)raw + corr_q[c + zero];
              num = fixed_to_float<long long>(wrap_to_bits(tot, p.int_bits), p.inv_scale);
            } else {
              // the sum fits 32 bits: the same value through the cheaper 32-bit conversion
              num = fixed_to_float<int>((int)raw, p.inv_scale);
            }
            out[i] = from_f32<T>(__fdiv_rn(num, dn));
          }
          *reinterpret_cast<uint4*>(op + g8 * 8) = *reinterpret_cast<const uint4*>(out);
        }
      }
    }
  }

  // ------------------------------ teardown ----------------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // let copies that are still in flight land before shared memory is released
    const long long tw = clock64();
    while (clock64() - tw < 200000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && status) atomicExch(status, FXPR_ERR_TIMEOUT);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFnA)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFnA encode_fn() {
  static EncodeTiledFnA fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFnA)ptr;
  }
  return fn;
}

// A plane of the paged cache as [blocks, 8-slot groups, 64-dim chunks (of all heads), 8 slots, 64 dims],
// boxes of box_rows slots x one head: [8-row group][chunk][8 rows][128 B] in shared memory, 128-byte
// swizzle.  The number of blocks is not known here and only bounds the coordinates, which come from the
// block table.
bool attn_kv_map(CUtensorMap* m, const AttnParams& p, int dtype, const void* plane, int box_rows) {
  EncodeTiledFnA fn = encode_fn();
  if (!fn || p.kv_shead % 64 != 0 || p.head_dim % 64 != 0) return false;
  cuuint64_t dims[5] = {64, 8, (cuuint64_t)((p.num_kv_heads - 1) * (p.kv_shead / 64) + p.head_dim / 64),
                        (cuuint64_t)(p.page_size / 8), (cuuint64_t)1 << 31};
  cuuint64_t strides[4] = {(cuuint64_t)p.kv_sslot * 2, 128, (cuuint64_t)p.kv_sslot * 16, (cuuint64_t)p.kv_sblock * 2};
  cuuint32_t box[5] = {64, 8, (cuuint32_t)(p.head_dim / 64), (cuuint32_t)(box_rows / 8), 1}, es[5] = {1, 1, 1, 1, 1};
  return fn(m, dtype == FXPR_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5,
            const_cast<void*>(plane), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The prefill kernel takes head size 128, bf16/fp16, 32- or 64-bit sums with at most 16
// fraction bits, no KV split, a sequence short enough for the 32-bit fast sums, and strides
// a tensor map can express (multiples of 16 bytes, below 2^40).
bool attention_tc_supported(const AttnParams& p, int dtype, int max_query_len, bool force_exact) {
  if (force_exact || p.num_splits != 1) return false;
  if (dtype != FXPR_F16 && dtype != FXPR_BF16) return false;
  if (p.head_dim != 128 || p.page_size % 16 != 0) return false;
  const int G = p.num_heads / p.num_kv_heads;
  if (G != 1 && G != 2 && G != 4 && G != 8 && G != 16) return false;
  if ((int64_t)max_query_len * G <= 16) return false;      // decode shapes: attention_mma.cu
  if (p.int_bits != 32 && p.int_bits != 64) return false;
  if (p.scale > 65536.0f) return false;
  const int64_t max_keys = p.bt_stride * (int64_t)p.page_size;
  if ((max_keys + kTcTileN - 1) / kTcTileN > 500) return false;
  const int64_t strides[] = {p.q_st, p.q_sh, p.o_st, p.o_sh, p.kv_sblock, p.kv_sslot, p.kv_shead};
  for (int64_t st : strides) if (st % 8 != 0 || st <= 0 || st >= (1ll << 35)) return false;
  if (p.kv_shead % 64 != 0) return false;
  if (((uintptr_t)p.q | (uintptr_t)p.k | (uintptr_t)p.v | (uintptr_t)p.o) & 15) return false;
  if (p.num_reqs > 65535) return false;
  return encode_fn() != nullptr;
}

int attention_tc(const AttnParams& p, int dtype, int max_query_len, int32_t* status, cudaStream_t s) {
  EncodeTiledFnA fn = encode_fn();
  if (!fn) return FXPR_ERR_CUDA;
  const int G = p.num_heads / p.num_kv_heads;
  TcAttnShape sh;
  sh.rows_per_token = G;
  sh.tokens_per_block = kTcRows / G;
  sh.num_q_blocks = (max_query_len + sh.tokens_per_block - 1) / sh.tokens_per_block;
  sh.page_size = p.page_size;
  sh.group_shift = (p.page_size % 64 == 0) ? 6 : 4;
  sh.page_mask = (p.page_size & (p.page_size - 1)) == 0 ? p.page_size - 1 : 0;
  const int fmt = dtype == FXPR_BF16 ? 1 : 0;
  sh.idesc_s = make_idesc(fmt, 0, kTcTileN, kTcRows);
  sh.idesc_s2 = make_idesc(fmt, 0, 2 * kTcTileN, kTcRows);
  sh.idesc_pv = make_idesc(fmt, 1, p.head_dim, kTcRows);
  if ((int64_t)sh.num_q_blocks * p.num_kv_heads > 0x7fffffffLL) return FXPR_ERR_UNSUPPORTED;

  const CUtensorMapDataType dt = dtype == FXPR_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap mq, mk, mv;
  {
    // q [tokens, heads, dims]
    cuuint64_t dims[3] = {(cuuint64_t)p.head_dim, (cuuint64_t)p.num_heads, (cuuint64_t)p.total_q};
    cuuint64_t strides[2] = {(cuuint64_t)p.q_sh * 2, (cuuint64_t)p.q_st * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)sh.tokens_per_block};
    cuuint32_t es[3] = {1, 1, 1};
    if (fn(&mq, dt, 3, const_cast<void*>(p.q), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
      set_last_error("cuTensorMapEncodeTiled(Q)", cudaErrorInvalidValue);
      return FXPR_ERR_CUDA;
    }
  }
  sh.head_chunks = (int)(p.kv_shead / 64);
  if (!attn_kv_map(&mk, p, dtype, p.k, 1 << sh.group_shift) || !attn_kv_map(&mv, p, dtype, p.v, 1 << sh.group_shift)) {
    set_last_error("cuTensorMapEncodeTiled(KV)", cudaErrorInvalidValue);
    return FXPR_ERR_CUDA;
  }

  constexpr int kSmem = kTcRows * 128 * 2 + kTcStages * 2 * kTcTileN * 128 * 2 + 2 * kTcRows * kTcTileN * 2 +
                        8 * (1 + 2 * kTcStages + 10 + 2 + 4) + 16 + 2048 + 4096 + 1024;
  // persistent CTAs, one per SM (204 KB of shared memory each), walking the padded item list
  const int64_t total_items = (int64_t)sh.num_q_blocks * p.num_kv_heads * p.num_reqs;
  if (total_items > 0x7fffffffLL) return FXPR_ERR_UNSUPPORTED;
  dim3 grid((unsigned)std::min<int64_t>(total_items, device_sms()), 1, 1);
#define FXPR_TC_ATTN(TT)                                                                              \
  do {                                                                                                \
    auto k = attn_tc_prefill_kernel<TT, 128>;                                                         \
    static bool attr_done_dev[64] = {};                                                               \
    int dev_id = 0;                                                                                   \
    cudaGetDevice(&dev_id);                                                                           \
    if (!attr_done_dev[dev_id & 63]) {                                                                \
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);    \
      if (e != cudaSuccess) { set_last_error("attention_tc smem attribute", e); return FXPR_ERR_CUDA; } \
      attr_done_dev[dev_id & 63] = true;                                                              \
    }                                                                                                 \
    k<<<grid, kTcThreads, kSmem, s>>>(mq, mk, mv, p, sh, status, 0);                                  \
  } while (0)
  if (dtype == FXPR_BF16) FXPR_TC_ATTN(__nv_bfloat16);
  else FXPR_TC_ATTN(__half);
#undef FXPR_TC_ATTN
  return check_launch("attention_tc");
}

}  // namespace fxpr
