// Decode kernel of the tensor-core attention route: at most 16 query rows per KV head
// ((tokens of the step) x (GQA group)), so one 16-row MMA tile per CTA.  The CTA's NW
// warps COOPERATE on every 64-key tile instead of owning tiles:
//   pass A  warp w computes Q.K^T for keys [64/NW * w, ...) of the tile, keeps the row
//           maxima and parks the fp32 scores in the shared-memory stash;
//   weights with the cluster-wide maxima each warp turns its own scores into weights, in place, and
//           counts them into the integer denominator: every weight is made once, not once per warp;
//   pass B  every warp reads the 64 packed weights of a tile and computes P.V for its own HD/NW slice
//           of the head dimension -- the same four m16n8k16 k-steps in the same order as the prefill
//           kernel, so a token's bits do not depend on which kernel served it.
// K is streamed once (pass A), V once (pass B); KV splits are cluster ranks merged through
// distributed shared memory exactly as in attn_mma_kernel.
//
// HBM-bound once a tile costs few enough instructions.  With every warp making all 64 weights and
// clamping conversions a warp spent 765 instructions on a tile, which at 8 clocks each and 16 warps per SM
// held the kernel at two thirds of the copy bandwidth; now about 300.  A tile arrives as four boxes of 16
// keys (one page piece each, attn_kv_map), requested by the warp with the same number: one copy
// instruction per warp and tile where 16-byte cp.async took eight with their address arithmetic.
// P.V partials are converted as in the GEMM (gemm_tc_fast_common.cuh): add 1.5 * 2^(23-f), sum the raw
// bits; a tile with a partial out of range, and 16-bit sums, take the saturating conversion.
// Two stages and four CTAs per SM: a CTA spends a third of its time in barriers of the cluster and in its
// first loads, so more CTAs cover more than deeper rings do (three stages, three CTAs: 6 % slower).
// 64 requests of 512 to 8192 tokens, 8 KV heads: 275 -> 222 us, 4.9 TB/s of keys and values.

// ROWS8: at most 8 of the 16 tile rows are real (e.g. one token x GQA group of 4): the
// second half of every accumulator fragment is known to be masked and is skipped.
// Byte offset of 16-byte chunk c of row r in a tile of attn_kv_map boxes.
template <int HD>
__device__ __forceinline__ uint32_t box_swz(int r, int c) {
  return (uint32_t)((r >> 3) * (HD / 64 * 1024) + (c >> 3) * 1024 + (r & 7) * 128 + (((c & 7) ^ (r & 7)) << 4));
}

template <typename T, int HD, int NW, bool ACC64, bool ROWS8, int NSTAGE, int MINB>
__global__ void __launch_bounds__(NW * 32, MINB)
attn_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const AttnParams p,
                   const MmaAttnShape sh) {
  constexpr int RC = HD / 8;
  constexpr int NT = NW * 32;
  constexpr int kTileBytes = kTileN * HD * 2;
  constexpr int JW = 8 / NW;                       // 8-key groups per warp in pass A
  constexpr int DW = HD / 8 / NW;                  // 8-wide head-dim groups per warp in pass B
  static_assert((NW == 2 || NW == 4 || NW == 8) && (HD / 8 / NW) % 2 == 0, "warps must divide the 8 key groups and the HD/16 pairs");
  constexpr int NE = ROWS8 ? 2 : 4;                // live slots of a C fragment
  constexpr int NH = ROWS8 ? 1 : 2;                // live row halves
  using AccT = typename IntOf<ACC64 ? 64 : 32>::type;

  extern __shared__ __align__(1024) uint8_t stage_s[];            // swizzle atoms are 1 KB
  constexpr int QR = ROWS8 ? 8 : 16;               // Q rows kept in shared memory (rows 8..15 of the MMA tile are zero registers)
  uint8_t* q_s = stage_s + NSTAGE * kTileBytes;                   // QR x HD
  float* rmax_s = reinterpret_cast<float*>(q_s + QR * HD * 2);                    // [NW][16]
  long long* den_s = reinterpret_cast<long long*>(rmax_s + NW * 16);              // [NW][16]
  uint64_t* bars_s = reinterpret_cast<uint64_t*>(den_s + NW * 16);                // kfull[NSTAGE][NW] vfull[NSTAGE] vfree[NSTAGE]
  volatile int* abort_s = reinterpret_cast<volatile int*>(bars_s + NSTAGE * (NW + 2));
  float* stash_s = reinterpret_cast<float*>(bars_s + NSTAGE * (NW + 2) + 2);
  long long* wv_s = reinterpret_cast<long long*>(stage_s);        // [16][HD], reuses the stages
  const uint32_t kfull0 = smem_addr(bars_s), vfull0 = kfull0 + 8u * NSTAGE * NW, vfree0 = vfull0 + 8u * NSTAGE;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NSTAGE * NW; ++i) mbar_init(kfull0 + 8u * i, 1);
    for (int i = 0; i < NSTAGE; ++i) { mbar_init(vfull0 + 8u * i, NW); mbar_init(vfree0 + 8u * i, NW); }
    *abort_s = p.abort_early;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_launch_dependents();
  pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  const int S = gridDim.x, rank = blockIdx.x;
  const int hkv = p.num_kv_heads;
  const int qb = blockIdx.y / hkv, kvh = blockIdx.y % hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;

  const int req = blockIdx.z;
  const int seq_len = p.seq_lens[req];              // with qsl: one round of loads, not one behind the other
  const int q_start = p.qsl[req], q_len = p.qsl[req + 1] - q_start;
  const int G = sh.rows_per_token;
  const int tok0 = qb * sh.tokens_per_block;
  if (tok0 >= q_len) return;
  const int ctx = seq_len - q_len;
  const int tok_end = min(q_len, tok0 + sh.tokens_per_block);
  const int32_t* bt = p.block_table + (int64_t)req * p.bt_stride;

  const int hi_key = p.causal ? min(seq_len, ctx + tok_end) : seq_len;
  const int lo_key = p.window > 0 ? max(0, ctx + tok0 - p.window + 1) : 0;
  const int t_first = lo_key / kTileN;
  const int t_last = max(t_first, (hi_key + kTileN - 1) / kTileN);
  const int per_rank = (t_last - t_first + S - 1) / S;
  const int t0 = min(t_last, t_first + rank * per_rank);
  const int t1 = min(t_last, t0 + per_rank);
  if (per_rank * kTileN > sh.stash_keys) {          // the host sizes the stash from the block-table width
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, FXPR_ERR_SCRATCH);
    return;                                          // the same decision in every CTA of the cluster
  }
  if (smem_addr(stage_s) & 1023u) {                  // a layout the boxes' swizzle does not match
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, FXPR_ERR_CUDA);
    return;
  }

  int r_tok[2], r_kend[2], r_kbeg[2]; float r_slope[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = g + 8 * h;
    r_tok[h] = tok0 + r / G;
    const bool valid = r_tok[h] < q_len;
    const int pos = ctx + r_tok[h];
    r_kend[h] = valid ? (p.causal ? min(seq_len, pos + 1) : seq_len) : 0;
    r_kbeg[h] = valid ? (p.window > 0 ? max(0, pos - p.window + 1) : 0) : 0;
    r_slope[h] = (p.alibi && valid) ? p.alibi[kvh * G + r % G] : 0.0f;
  }

  for (int idx = threadIdx.x; idx < QR * RC; idx += NT) {
    const int r = idx / RC, c = idx % RC;
    const int tok = tok0 + r / G;
    const bool v = tok < q_len;
    const T* src = (const T*)p.q + (int64_t)(q_start + (v ? tok : 0)) * p.q_st +
                   (int64_t)(kvh * G + r % G) * p.q_sh + c * 8;
    cp_async16(smem_addr(q_s) + swz<RC>(r, c), src, v);
  }
  cp_async_commit();

  // Warp w requests keys [16 w, 16 w + 16) of every tile -- one 16-key page group, one block-table
  // entry.  Pass A: it also reads exactly these keys, so its ring needs no other warp and goes on into
  // the V tiles before the maxima are known.  Pass B: every warp reads all 64 keys, so a stage has a
  // barrier that counts the four warps' boxes and one that counts the four warps' being done with it.
  // Keys past the sequence are not requested and never touch the block table.
  static_assert(NW == 4, "one 16-key page group per warp");
  constexpr uint32_t kPiece = kTileBytes / NW;
  const uint32_t elected = elect_one();
  const int pshift = sh.page_shift;
  const int chunk0 = (int)(kvh * (p.kv_shead / 64));
  int ent_t = t0;                                    // lane L holds the block-table entry of tile ent_t + L
  auto load_entries = [&]() -> int {
    const int n = (ent_t + lane) * kTileN + warp * 16;
    return (ent_t + lane < t1 && n < seq_len) ? bt[pshift >= 0 ? (n >> pshift) : n / p.page_size] : 0;
  };
  int ent = load_entries();
  const uint32_t stage0 = smem_addr(stage_s);
  const int n_tiles = t1 - t0;
  int req_i = 0, req_st = 0, req_end = 2 * n_tiles;  // next tile to request: K tiles, then V tiles, round the stages
  auto request = [&]() {
    const bool is_v = req_i >= n_tiles;
    const int t = t0 + (is_v ? req_i - n_tiles : req_i);
    if ((unsigned)(t - ent_t) >= 32u) { ent_t = t; ent = load_entries(); }
    const int blk = __shfl_sync(0xffffffffu, ent, t - ent_t);
    const int n = t * kTileN + warp * 16;
    const int slot = pshift >= 0 ? (n & (p.page_size - 1)) : n % p.page_size;
    const bool any = n < seq_len;
    const uint32_t bar = is_v ? vfull0 + 8u * req_st : kfull0 + 8u * (req_st * NW + warp);
    mbar_expect_tx(bar, any ? kPiece : 0u, elected);
    tma_load_5d(stage0 + req_st * kTileBytes + warp * kPiece, is_v ? &map_v : &map_k, bar, 0, 0, chunk0, slot >> 3, blk,
                any ? elected : 0u);
    ++req_i;
    if (++req_st == NSTAGE) req_st = 0;
  };

  const uint32_t qs_addr = smem_addr(q_s);
  // A bounded wait of the whole warp.  A warp that gave up requests no box any more: the stage may still be
  // waiting for one, and its barrier takes one arrival of this warp a phase.
  auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
    const bool done = __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_s));
    if (!done) req_end = 0;
    return done;
  };
  const float ninf = -__int_as_float(0x7f800000);
  const int srows = sh.stash_rows;
  const int slanes = srows <= 8 ? 4 * srows : 32;
  const bool small_q = p.int_bits >= 32 && p.scale <= 16777216.0f;   // Q(w) <= 2^24 per key, 64 keys per tile

  constexpr int HC = HD / 64;
  constexpr int kGroup = HC * 1024;                  // bytes of 8 keys

  // =============================== pass A =============================================
  float rmax[2] = {ninf, ninf};
  // Scores, later weights: a lane's values of one warp's 16 keys lie together.
  auto stash_at = [&](int t, int w) -> float* {
    return stash_s + ((size_t)((t - t0) * NW + w) * slanes + lane) * (JW * NE);
  };
  {
    __syncthreads();                                 // the barriers exist
#pragma unroll 1
    while (req_i < min(NSTAGE, req_end)) request();
    cp_async_wait<0>();
    __syncthreads();                                 // Q is in shared memory for every warp
    uint32_t qa[HD / 16][ROWS8 ? 2 : 4];
#pragma unroll
    for (int kk2 = 0; kk2 < HD / 32; ++kk2) {
      if constexpr (ROWS8) {
        // eight live rows: one load brings rows 0..7 of four 8-wide k chunks
        ldsm_x4(qs_addr + swz<RC>(lane & 7, kk2 * 4 + (lane >> 3)), qa[2 * kk2][0], qa[2 * kk2][1], qa[2 * kk2 + 1][0],
                qa[2 * kk2 + 1][1]);
      } else {
        ldsm_x4(qs_addr + swz<RC>(lane & 15, kk2 * 4 + (lane >> 4)), qa[2 * kk2][0], qa[2 * kk2][1], qa[2 * kk2][2],
                qa[2 * kk2][3]);
        ldsm_x4(qs_addr + swz<RC>(lane & 15, kk2 * 4 + 2 + (lane >> 4)), qa[2 * kk2 + 1][0], qa[2 * kk2 + 1][1],
                qa[2 * kk2 + 1][2], qa[2 * kk2 + 1][3]);
      }
    }
    const uint32_t k_off = warp * kPiece + box_swz<HD>(lane & 7, lane >> 3);
    int st = 0; uint32_t ph = 0;
#pragma unroll 1
    for (int t = t0; t < t1; ++t) {
      wait(kfull0 + 8u * (st * NW + warp), ph);
      const uint32_t k_addr = stage0 + st * kTileBytes + k_off;
      if (++st == NSTAGE) { st = 0; ph ^= 1; }
      float s[JW][4];
#pragma unroll
      for (int jj = 0; jj < JW; ++jj) { s[jj][0] = s[jj][1] = s[jj][2] = s[jj][3] = 0.0f; }
#pragma unroll
      for (int kk2 = 0; kk2 < HD / 32; ++kk2) {
        uint32_t a0[4], a1[4];
        if constexpr (ROWS8) {
          a0[0] = qa[2 * kk2][0]; a0[2] = qa[2 * kk2][1]; a1[0] = qa[2 * kk2 + 1][0]; a1[2] = qa[2 * kk2 + 1][1];
          a0[1] = a0[3] = a1[1] = a1[3] = 0u;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) { a0[i] = qa[2 * kk2][i]; a1[i] = qa[2 * kk2 + 1][i]; }
        }
#pragma unroll
        for (int jj = 0; jj < JW; ++jj) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4((k_addr ^ ((kk2 & 1) * 64)) + jj * kGroup + (kk2 >> 1) * 1024, b0, b1, b2, b3);
          mma16816<T>(s[jj], a0, b0, b1);
          mma16816<T>(s[jj], a1, b2, b3);
        }
      }
      __syncwarp();
      if (req_i < req_end) request();            // into the rows of this tile, which only this warp reads
#pragma unroll
      for (int jj = 0; jj < JW; ++jj) {
        const int j = warp * JW + jj;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const int h = e >> 1;
          const int n = t * kTileN + j * 8 + 2 * t4 + (e & 1);
          float v = __fmul_rn(s[jj][e], p.ss_log2);
          if (p.cap_log2 > 0.0f) v = __fmul_rn(p.cap_log2, tanhf(__fdiv_rn(v, p.cap_log2)));
          if (p.alibi) v = __fadd_rn(v, __fmul_rn(r_slope[h], __fsub_rn((float)n, (float)(ctx + r_tok[h]))));
          s[jj][e] = (n >= r_kbeg[h] && n < r_kend[h]) ? v : ninf;
        }
        rmax[0] = fmaxf(rmax[0], fmaxf(s[jj][0], s[jj][1]));
        if (!ROWS8) rmax[1] = fmaxf(rmax[1], fmaxf(s[jj][2], s[jj][3]));
      }
      if (lane < slanes) {
        float4* d = reinterpret_cast<float4*>(stash_at(t, warp));
        if constexpr (ROWS8) {
          d[0] = make_float4(s[0][0], s[0][1], s[1][0], s[1][1]);
        } else {
          d[0] = make_float4(s[0][0], s[0][1], s[0][2], s[0][3]);
          d[1] = make_float4(s[1][0], s[1][1], s[1][2], s[1][3]);
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    rmax[h] = fmaxf(rmax[h], __shfl_xor_sync(0xffffffffu, rmax[h], 1));
    rmax[h] = fmaxf(rmax[h], __shfl_xor_sync(0xffffffffu, rmax[h], 2));
    if (t4 == 0) rmax_s[warp * 16 + g + 8 * h] = rmax[h];
  }
  // One maximum per row and CTA for the peers to read: remote reads are paced per request.
  __syncthreads();
  if (threadIdx.x < 16) {
    float m = rmax_s[threadIdx.x];
#pragma unroll
    for (int w = 1; w < NW; ++w) m = fmaxf(m, rmax_s[w * 16 + threadIdx.x]);
    rmax_s[threadIdx.x] = m;
  }
  cluster.sync();
  float gmax[2];
  {
    float m[2] = {ninf, ninf};
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      for (int r = t4; r < S; r += 4) m[h] = fmaxf(m[h], cluster.map_shared_rank(rmax_s, r)[g + 8 * h]);
      m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 1));
      m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 2));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) gmax[h] = (m[h] == ninf) ? 0.0f : m[h];
  }

  // =============================== weights ============================================
  long long den[2] = {0, 0};
  if (lane < slanes) {
#pragma unroll 2
    for (int t = t0; t < t1; ++t) {
      float* d = stash_at(t, warp);
      float w[JW * NE];
#pragma unroll
      for (int i = 0; i < JW * NE; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(d + i);
        w[i] = v.x; w[i + 1] = v.y; w[i + 2] = v.z; w[i + 3] = v.w;
      }
      uint32_t den_tile[2] = {0u, 0u};               // w <= 1, so a tile's Q(w) sum fits 32 bits (f <= 24)
#pragma unroll
      for (int i = 0; i < JW * NE; ++i) {
        const int h = (i % NE) >> 1;
        w[i] = ex2_approx(__fsub_rn(w[i], gmax[h]));  // a masked score is -inf: its weight is 0
        if (small_q) den_tile[h] += (uint32_t)float_to_fixed<32>(w[i], p.scale);
        else den[h] += float_to_fixed_any(w[i], p.scale, p.int_bits);
      }
      den[0] += (long long)den_tile[0];
      if (!ROWS8) den[1] += (long long)den_tile[1];
      if constexpr (ROWS8)
        *reinterpret_cast<uint2*>(d) = make_uint2(pack2_io<T>(w[0], w[1]), pack2_io<T>(w[2], w[3]));
      else
        *reinterpret_cast<uint4*>(d) = make_uint4(pack2_io<T>(w[0], w[1]), pack2_io<T>(w[2], w[3]), pack2_io<T>(w[4], w[5]),
                                                  pack2_io<T>(w[6], w[7]));
    }
  }
  __syncthreads();

  // =============================== pass B =============================================
  AccT acc[DW][NE];
  uint32_t acc32[DW][NE];                            // ACC64: raw sums of at most 256 tiles, 2^22 each
#pragma unroll
  for (int j = 0; j < DW; ++j) {
#pragma unroll
    for (int e = 0; e < NE; ++e) { acc[j][e] = 0; acc32[j][e] = 0u; }
  }
  {
    const uint32_t magic_bits = q_magic_bits(p.inv_scale);
    const float limit = p.int_bits >= 32 ? q_screen_limit(p.inv_scale) : 0.0f;
    const uint32_t v_off = box_swz<HD>(lane & 15, warp * DW + (lane >> 4));
    int st = n_tiles % NSTAGE, use = 0, prev = 0; uint32_t ph = 0, ph_prev = 0;
#pragma unroll 1
    for (int t = t0; t < t1; ++t) {
      if (t > t0 && req_i < req_end) {             // into the stage of tile t - 1: before the wait for tile t, 6 % faster
        if (wait(vfree0 + 8u * prev, ph_prev)) request();
      }
      uint32_t pa[4][4];
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const float* d = stash_at(t, w);
        if constexpr (ROWS8) {
          const uint2 v = lane < slanes ? *reinterpret_cast<const uint2*>(d) : make_uint2(0u, 0u);
          pa[w][0] = v.x; pa[w][2] = v.y;
          pa[w][1] = pa[w][3] = 0u;
        } else {
          const uint4 v = *reinterpret_cast<const uint4*>(d);
          pa[w][0] = v.x; pa[w][1] = v.y; pa[w][2] = v.z; pa[w][3] = v.w;
        }
      }
      wait(vfull0 + 8u * st, ph);
      const uint32_t v_addr = stage0 + st * kTileBytes;
      if (seq_len - t * kTileN < kTileN) {
        // rows past the sequence hold whatever the page holds, or were not requested: 0 * NaN would
        // poison the product, so this warp clears its slice of them
        constexpr int WC = RC / NW;
        const int r0 = max(0, seq_len - t * kTileN);
        for (int idx = lane; idx < (kTileN - r0) * WC; idx += 32)
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};"
                       ::"r"(v_addr + box_swz<HD>(r0 + idx / WC, warp * WC + idx % WC)), "r"(0) : "memory");
        __syncwarp();
      }
      float pv[DW][4];
#pragma unroll
      for (int j = 0; j < DW; ++j) { pv[j][0] = pv[j][1] = pv[j][2] = pv[j][3] = 0.0f; }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
        for (int jj2 = 0; jj2 < DW / 2; ++jj2) {       // pair of 8-wide head-dim groups
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(v_addr + (v_off ^ (jj2 * 32)) + kk * 2 * kGroup, b0, b1, b2, b3);
          mma16816<T>(pv[2 * jj2], pa[kk], b0, b1);
          mma16816<T>(pv[2 * jj2 + 1], pa[kk], b2, b3);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(vfree0 + 8u * st);
      prev = st;
      ph_prev = ph;
      if (++use == NSTAGE) { use = 0; ph ^= 1; }
      if (++st == NSTAGE) st = 0;

      float screen = 0.0f;
#pragma unroll
      for (int j = 0; j < DW; ++j) {
#pragma unroll
        for (int e = 0; e < NE; e += 2) screen = max3_abs(screen, pv[j][e], pv[j][e + 1]);
      }
      if (__all_sync(0xffffffffu, screen < limit)) {
#pragma unroll
        for (int j = 0; j < DW; ++j) {
#pragma unroll
          for (int e = 0; e < NE; ++e) {
            const uint32_t r = __float_as_uint(__fadd_rn(pv[j][e], __uint_as_float(magic_bits))) - magic_bits;
            if (ACC64) acc32[j][e] += r;
            else acc[j][e] += (AccT)r;
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < DW; ++j) {
#pragma unroll
          for (int e = 0; e < NE; ++e)
            acc[j][e] += (AccT)(ACC64 ? float_to_fixed<64>(pv[j][e], p.scale) : float_to_fixed_any(pv[j][e], p.scale, p.int_bits));
        }
      }
      if (ACC64 && (t == t1 - 1 || ((t - t0) & 255) == 255)) {
#pragma unroll
        for (int j = 0; j < DW; ++j) {
#pragma unroll
          for (int e = 0; e < NE; ++e) { acc[j][e] += (AccT)(int32_t)acc32[j][e]; acc32[j][e] = 0u; }
        }
      }
    }
  }

  // =============================== merge ==============================================
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    den[h] += __shfl_xor_sync(0xffffffffu, den[h], 1);
    den[h] += __shfl_xor_sync(0xffffffffu, den[h], 2);
  }
  __syncthreads();                                   // stages are free: reuse them for wv_s
  const int gave_up = *abort_s;                      // one for all threads; looked at last, behind the load's latency
#pragma unroll
  for (int h = 0; h < NH; ++h) {
    const int r = g + 8 * h;
    if (t4 == 0) den_s[warp * 16 + r] = den[h];
#pragma unroll
    for (int jj = 0; jj < DW; ++jj) {
      const int d = (warp * DW + jj) * 8 + 2 * t4;
      wv_s[(size_t)r * HD + d] = (long long)acc[jj][2 * h];
      wv_s[(size_t)r * HD + d + 1] = (long long)acc[jj][2 * h + 1];
    }
  }
  // One denominator per row and CTA (not one per warp): reads over distributed shared memory are
  // paced per request, so the merge below asks for as few and as wide ones as it can.
  __syncthreads();
  long long den_row = 0;
  if (threadIdx.x < 16) {
#pragma unroll
    for (int w = 0; w < NW; ++w) den_row += den_s[w * 16 + threadIdx.x];
  }
  __syncthreads();
  if (threadIdx.x < 16) den_s[threadIdx.x] = den_row;
  cluster.sync();
  {
    // Every rank merges its own slice of the head dimension (integer sums over the ranks are
    // order-free), so the peers' shared memory is needed only for a short, parallel read.
    const int rows_here = min(16, (tok_end - tok0) * G);
    const int cpr = (HD + S - 1) / S;                // columns per rank
    const int c0 = rank * cpr;
    const int ncol = max(0, min(HD, c0 + cpr) - c0);
    const bool pairs = ((cpr | ncol) & 1) == 0;      // then c0 is even too: 16-byte reads
    const int per_row = pairs ? ncol / 2 : ncol;
    for (int idx = threadIdx.x; idx < rows_here * per_row; idx += NT) {
      const int r = idx / per_row, d = c0 + (pairs ? 2 : 1) * (idx % per_row);
      long long dsum = 0, w0 = 0, w1 = 0;
      for (int rr = 0; rr < S; ++rr) {
        dsum += cluster.map_shared_rank(den_s, rr)[r];
        const long long* wp = cluster.map_shared_rank(wv_s, rr) + (size_t)r * HD + d;
        if (pairs) {
          const longlong2 v = *reinterpret_cast<const longlong2*>(wp);
          w0 += v.x;
          w1 += v.y;
        } else {
          w0 += wp[0];
        }
      }
      const float dn = fmaxf(fixed_to_float<long long>(wrap_to_bits(dsum, p.int_bits), p.inv_scale), 1.0e-6f);
      const int tok = tok0 + r / G, head = kvh * G + r % G;
      T* op = (T*)p.o + (int64_t)(q_start + tok) * p.o_st + (int64_t)head * p.o_sh;
      op[d] = from_f32<T>(__fdiv_rn(fixed_to_float<long long>(wrap_to_bits(w0, p.int_bits), p.inv_scale), dn));
      if (pairs)
        op[d + 1] = from_f32<T>(__fdiv_rn(fixed_to_float<long long>(wrap_to_bits(w1, p.int_bits), p.inv_scale), dn));
    }
  }
  if (gave_up) {
    // boxes still in flight must land in this CTA's shared memory, not in its successor's
    const long long since = clock64();
    while (clock64() - since < 200000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, FXPR_ERR_TIMEOUT);
  }
  cluster.sync();
}
