// Tensor-core fixed-point GEMM for medium batches (65 to some 700 rows): the roles of gemm_tc_skinny.cu, weights on the
// M side of the MMA, on pairs of SMs (tcgen05.mma cta_group::2):
//
//     D^T[n, m] = sum_k W[k, n] * X[m, k]        M_mma = 256 (n), N_mma = MP = 96 to 256 (m), K = 16
//
// Each CTA of a pair loads its own 128 weight columns and half of the tile's activation rows; the tensor cores of both
// read both halves of the rows, and each CTA's tensor memory receives its 128 columns x MP rows.  K-splits run as
// one cluster (2 to 4 splits x 2 CTAs) and are merged like the decode-shape kernel's: each split sums a
// slice of the rows that the others send it.
// Bound: copies.  A CTA's copy unit takes 2.4 clocks for a 128-byte row of a box (3.05 when most SMs fetch out of L2), and a
// tile asks for 256 of weights and MP of activations per 128 of K, where two 128 x 128 tiles on single SMs ask for
// 1024 together; the rows of a tile follow the batch (333 rows are three tiles of 111); small weights split K without
// the scratch planes.  Copies and barriers come 128 of K at a time and weights in one box (64 of K, two boxes of 64
// columns: 10 % slower).  At K-tile 64 the conversion is as long.  Against 128 x 128 tiles with planes, K-tile 128, in a graph, us:
//   80 x 4096 x 4096 21.9 -> 12.4, 80 x 768 x 4096 26.7 -> 10.1, 200 x 4096 x 14336 46.6 -> 37.2,
//   333 x 6144 x 4096 26.0 -> 23.3 (a call among others, with bias: 30.8 -> 27.8), 700 x 4096 x 4096 (256 x 256 tiles) 37.7 -> 28.4.
// Which calls come here: mid_route in host_policy.h.
//
// Numerics are those of the other tensor-core kernels: one fresh fp32 accumulator per K-tile, rint-half-even to Q-format
// on the FP32 pipe with the exact fix-up, integer sums (the fixed-point contract: fxpr_vllm/_triton/gemm.py:183-204).
#include <cuda.h>

#include "fxp_common.cuh"
#include "gemm_common.cuh"
#include "host_policy.h"
#include "tc_common.cuh"
#include "gemm_tc_fast_common.cuh"

namespace fxpr {

static constexpr int kMdEpiW = 16;
static constexpr int kMdThreads = (2 + kMdEpiW) * 32;
static constexpr int kMdWBytes = 128 * kBK * 2;           // a CTA's weights of half a stage: 64 of K, 128 columns

template <int MP> struct MdShape {
  static constexpr int kXBytes = MP / 2 * kBK * 2;         // its half of the activation rows
  static constexpr int kHalfBytes = kMdWBytes + kXBytes;   // 64 of K: weights, rows
  static constexpr int kStageBytes = 2 * kHalfBytes;       // a stage is 128 of K: one K-tile of 128 or two of 64
  static constexpr int kStages = (225 * 1024) / kStageBytes;
  static constexpr int kGroups = 512 / MP;                 // accumulators in tensor memory
  static constexpr int kBarOffset = kStages * kStageBytes;
  static constexpr int kBarBytes = 512;
  static constexpr int kSmem = kBarOffset + kBarBytes + 1024;
  // over the stages once they are done: the finished sums, [row][128 columns] of 32 bits, and for the cluster merge
  // (MP <= 128, at most four splits) what the peers send, three quarters of the rows, their flags, this rank's
  // high words
  static constexpr int kRecvOffset = MP * 512, kFlagOffset = kRecvOffset + MP * 384, kHighOffset = kFlagOffset + 1024;
  static_assert(MP * 512 <= kBarOffset, "the sums fit the stages");
  static_assert(MP > 128 || kHighOffset + MP * 512 <= kBarOffset, "the merge fits the stages");
  static_assert(kSmem <= 227 * 1024, "shared memory of an SM");
  static_assert(MP % 32 == 0 && MP <= 256, "16 epilogue warps, whole 8-row groups in either CTA");
};

// grid (2 * splits, column tiles of 256, row tiles), clusters of 2 * splits CTAs; SPLIT: more than one split
template <typename T, int MP, bool SPLIT>
__global__ void __launch_bounds__(kMdThreads, 1)
gemm_tc_mid_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                   const TcParams p, const int tile_rows, const int w_box, const int zero /* always 0: keeps the side arrays in local memory */) {
  using Shape = MdShape<MP>;
  constexpr int STAGES = Shape::kStages, GROUPS = Shape::kGroups;
  constexpr int EPIW = kMdEpiW;
  constexpr int kCols = MP / 4;                            // activation rows per epilogue thread
  constexpr int kStageBytes = Shape::kStageBytes, kHalfBytes = Shape::kHalfBytes, kBarOffset = Shape::kBarOffset;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kBarOffset;
  // full[stage] (leader): its arrive plus the bytes of both CTAs; empty[stage], tfull[group]: one commit, in
  // both CTAs; tempty[group] (leader): the epilogue warps of both CTAs
  const uint32_t full0 = bar_base, empty0 = full0 + 8u * STAGES;
  const uint32_t tfull0 = empty0 + 8u * STAGES, tempty0 = tfull0 + 8u * GROUPS;
  constexpr int kMisc = (8 * (2 * STAGES + 2 * GROUPS) + 15) / 16 * 16;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem_gen + kBarOffset + kMisc);
  volatile int* abort_flag = (volatile int*)(smem_gen + kBarOffset + kMisc + 8);
  const uint32_t epi_bar = bar_base + kMisc + 16u, recv_bar = bar_base + kMisc + 24u;
  volatile int* s_wide = (volatile int*)(smem_gen + kBarOffset + kMisc + 32);   // 16 bytes, copied to the peers
  const uint32_t high_bar = bar_base + kMisc + 48u;
  static_assert(kMisc + 56 <= Shape::kBarBytes, "barrier block");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)blockIdx.x, parity = rank & 1, ks = rank >> 1, S = p.split_k;
  const uint32_t leader = (uint32_t)(rank & ~1);
  const int n0 = ((int)blockIdx.y * 2 + parity) * 128, row0 = (int)blockIdx.z * tile_rows;
  const int live_rows = min(tile_rows, p.M - row0);
  // merge: split s sums rows [s * rows_per, ...) of the live ones over all splits
  const int rows_per = SPLIT ? (live_rows + S - 1) / S : 0;
  auto rows_of = [&](int s) { return max(0, min(live_rows - s * rows_per, rows_per)); };

  pdl_launch_dependents();                                 // the next kernel may start its own setup
  if (threadIdx.x == 64) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tma_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tma_x) : "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8u * s, 1); mbar_init(empty0 + 8u * s, 1); }
    for (int b = 0; b < GROUPS; ++b) { mbar_init(tfull0 + 8u * b, 1); mbar_init(tempty0 + 8u * b, 2 * EPIW); }
    mbar_init(epi_bar, EPIW);
    mbar_init(recv_bar, 1);
    if constexpr (SPLIT) mbar_init(high_bar, (uint32_t)(S - 1));
    *abort_flag = 0;
    for (int i = 0; i < 4; ++i) s_wide[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if constexpr (SPLIT) {
      const int rows = rows_of(ks);
      mbar_expect_tx(recv_bar, rows > 0 ? (uint32_t)((S - 1) * (rows * 512 + 16)) : 0u);
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32((const void*)tmem_slot), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                      // the peers' barriers exist from here on
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                                              // from here on the kernel reads what earlier ones wrote

  const int k_tiles_total = (p.K + p.k_tile - 1) / p.k_tile;
  const int n_kt = (k_tiles_total - ks + S - 1) / S;
  const bool pairs = p.k_tile == 64;                       // two K-tiles per stage
  const int n_st = pairs ? (n_kt + 1) >> 1 : n_kt;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------
    const uint32_t e = elect_one();
    // weights by one box of 64 x 128 where a map can say that: 3 = columns in groups of 64, 2 = an (N, K) row-major
    // view; else (ragged columns) by two of 64 x 64
    const uint32_t full_leader = mapa_u32(full0, leader);  // the leader's barriers count both CTAs' bytes
    const int x_row = row0 + parity * (MP / 2);
    int stage = 0; uint32_t phase = 1;
    for (int j = 0; j < n_st; ++j) {
      const int ka = pairs ? (ks + 2 * j * S) * 64 : (ks + j * S) * 128, kb = pairs ? ka + S * 64 : ka + 64;
      const bool two = !pairs || 2 * j + 1 < n_kt;
      if (!__all_sync(0xffffffffu, mbar_wait_poll(empty0 + 8u * stage, phase, abort_flag))) break;
      const uint32_t fb = full_leader + 8u * stage;
      if (parity == 0) mbar_expect_tx(full0 + 8u * stage, two ? 2 * kStageBytes : kStageBytes, e);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h && !two) break;
        const int kk = h ? kb : ka;
        const uint32_t sw = smem_base + stage * kStageBytes + h * kHalfBytes;
        if (w_box == 3) {
          tma_load_3d_pair(sw, &tma_w, fb, 0, kk, n0 / 64, e);
        } else if (w_box == 2) {
          tma_load_2d_pair(sw, &tma_w, fb, kk, n0, e);
        } else {
          tma_load_2d_pair(sw, &tma_w, fb, n0, kk, e);
          tma_load_2d_pair(sw + 8192, &tma_w, fb, n0 + 64, kk, e);
        }
        tma_load_2d_pair(sw + kMdWBytes, &tma_x, fb, kk, x_row, e);
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader only) ------------------------
    if (parity == 0) {
      const uint64_t wdesc0 = p.b_kmajor ? make_smem_desc(smem_base, 16, 1024) : make_smem_desc(smem_base, 8192, 1024);
      const uint64_t xdesc0 = make_smem_desc(smem_base + kMdWBytes, 16, 1024);
      const uint64_t wks = p.b_kmajor ? 2 : 128;           // (32 B | 2048 B) >> 4 per 16-deep k step
      constexpr uint64_t kStep = kStageBytes >> 4, kHalf = kHalfBytes >> 4;
      const uint32_t idesc = p.idesc, e = elect_one();
      const uint16_t both = (uint16_t)(3u << leader);
      int stage = 0; uint32_t phase = 0; int grp = 0; uint32_t gphase = 1;
      for (int j = 0; j < n_st; ++j) {
        const bool two = !pairs || 2 * j + 1 < n_kt;
        if (!__all_sync(0xffffffffu, mbar_wait_poll(full0 + 8u * stage, phase, abort_flag))) goto issuer_done;
        const uint64_t wd = wdesc0 + (uint64_t)stage * kStep, xd = xdesc0 + (uint64_t)stage * kStep;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h && !two) break;
          const bool fresh = !h || pairs;                  // a K-tile begins: a fresh accumulator
          if (fresh) {
            if (!__all_sync(0xffffffffu, mbar_wait_poll(tempty0 + 8u * grp, gphase, abort_flag))) goto issuer_done;
            tc_fence_after();
          }
          const uint32_t d = tmem_base + (uint32_t)(grp * MP);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            umma_f16_pair(d, wd + h * kHalf + i * wks, xd + h * kHalf + i * 2, idesc, i ? 1u : fresh ? 0u : 1u, e);
          if (h || pairs) {
            if (h || !two) umma_commit_pair(empty0 + 8u * stage, both, e);
            umma_commit_pair(tfull0 + 8u * grp, both, e);
            if (++grp == GROUPS) { grp = 0; gphase ^= 1; }
          }
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    issuer_done:;
    }
  } else {
    // ------------------------------ epilogue warps (both CTAs) ----------------------
    // One output COLUMN n per thread and kCols consecutive activation rows m.
    const int quarter = warp & 3;
    const int cgroup = (warp - 2) >> 2;
    const int n_in_tile = quarter * 32 + lane;
    const int m0 = cgroup * kCols;
    const uint32_t lane_addr = ((uint32_t)(quarter * 32) << 16) + (uint32_t)m0;
    const uint32_t mbits = q_magic_bits(p.inv_scale), one = (uint32_t)zero + 1u;
    const uint64_t magic2 = pack2(mbits, mbits);
    const float screen_limit = q_screen_limit(p.inv_scale);
    const uint32_t tempty_leader = mapa_u32(tempty0, leader);
    int grp = 0; uint32_t gphase = 0; uint32_t epi_phase = 0; bool ok = true;
    auto epi_sync = [&]() -> bool {                        // bounded barrier over the epilogue warps only
      __syncwarp();
      if (lane == 0) mbar_arrive(epi_bar);
      const bool done = warp_wait(epi_bar, epi_phase, abort_flag);
      epi_phase ^= 1;
      return done;
    };
    // Rare-path corrections (local memory, zeroed on first use), as in the other kernels.
    uint32_t corr_raw[kCols];
    long long corr_q[kCols];
    bool corr_used = false;
    bool announced = false;                                // merge: this thread has said that the stages are done
    int* stage32 = reinterpret_cast<int*>(smem_gen);                    // [MP][128]
    long long* stage64 = reinterpret_cast<long long*>(smem_gen);        // [MP / 2][128]
    const bool c_vec4 = ((uintptr_t)p.c & 7) == 0 && p.c_sm % 4 == 0;
    const int n4 = n0 + lane * 4;                          // output columns of this lane
    float bias4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) bias4[i] = p.bias && n4 + i < p.N ? to_f32<T>(((const T*)p.bias)[n4 + i]) : 0.0f;
    // four neighbouring sums of row m, columns n4..n4 + 3, to the outputs
    auto emit = [&](int m, auto q0, auto q1, auto q2, auto q3) {
      using Q = decltype(q0);
      const Q q[4] = {q0, q1, q2, q3};
      const int64_t row = row0 + m;
      if (p.c_int) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (n4 + i >= p.N) continue;
          if (p.int_bits == 64) ((long long*)p.c_int)[row * p.N + n4 + i] = (long long)q[i];
          else ((int32_t*)p.c_int)[row * p.N + n4 + i] = (int32_t)q[i];
        }
      }
      if (!p.c) return;
      alignas(8) T out[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float v = fixed_to_float<Q>(q[i], p.inv_scale);
        if (p.bias) v = __fadd_rn(v, bias4[i]);
        out[i] = from_f32<T>(v);
      }
      T* dst = (T*)p.c + row * p.c_sm + n4;
      if (c_vec4 && n4 + 4 <= p.N) {
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(out);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) if (n4 + i < p.N) dst[i] = out[i];
      }
    };

    uint32_t acc[kCols];
#pragma unroll
    for (int i = 0; i < kCols; ++i) acc[i] = 0;
#pragma unroll 1
    for (int kt = 0; kt < n_kt; ++kt) {
      if (!warp_wait(tfull0 + 8u * grp, gphase, abort_flag)) { ok = false; break; }
      tc_fence_after();
      if constexpr (SPLIT) {
        // the last accumulator is complete, so no MMA or copy touches the stages any more
        if (kt == n_kt - 1) { cluster_arrive(); announced = true; }
      }
      const uint32_t ta = tmem_base + lane_addr + (uint32_t)(grp * MP);
      float screen = 0.0f;
#pragma unroll
      for (int c = 0; c + 16 <= kCols; c += 16) {
        uint32_t v[16];
        tmem_ld16(ta + c, v); tmem_wait_ld_regs(v);
        convert_n<16>(v, acc + c, magic2, mbits, one, screen);
      }
      if constexpr (kCols % 16 == 8) {
        uint32_t v[8];
        tmem_ld8(ta + kCols - 8, v); tmem_wait_ld_regs(v);
        convert_n<8>(v, acc + kCols - 8, magic2, mbits, one, screen);
      }
      if (__any_sync(0xffffffffu, !(screen < screen_limit))) {
        if (!corr_used) {
#pragma unroll 1
          for (int z = 0; z < kCols; ++z) { corr_raw[z + zero] = 0; corr_q[z + zero] = 0; }
          corr_used = true;
        }
        fixup_tile(ta, kCols, mbits, p.scale, p.int_bits, &corr_raw[zero], &corr_q[zero]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_leader + 8u * grp);
      if (++grp == GROUPS) { grp = 0; gphase ^= 1; }
    }
    const uint32_t bias_bits = (uint32_t)n_kt * mbits;     // the multiply-adds summed one magic per K-tile
    auto total32 = [&](int i) -> uint32_t { return alu_add(i) ? acc[i] : acc[i] - bias_bits; };
    // the exact sum where this warp took the fix-up; `raw` is total32
    auto total = [&](uint32_t raw, int i) -> long long {
      const long long t = (long long)(int32_t)(raw - corr_raw[i + zero]) + corr_q[i + zero];
      return p.int_bits == 64 ? t : (long long)(int32_t)t;
    };
    const bool wide_warp = corr_used && p.int_bits == 64;  // sums may exceed 32 bits
    if (ok) {
#pragma unroll
      for (int i = 0; i < kCols; ++i) stage32[(m0 + i) * 128 + n_in_tile] = (int)total32(i);
      if (corr_used) {
        // replace this thread's own words by the exact ones (low words), in a loop
        int* high = reinterpret_cast<int*>(smem_gen + Shape::kHighOffset);
#pragma unroll 1
        for (int i = 0; i < kCols; ++i) {
          const int at = (m0 + i) * 128 + n_in_tile;
          const long long t = total((uint32_t)stage32[at], i);
          if constexpr (!SPLIT) corr_q[i + zero] = t;      // kept for the 64-bit output below
          stage32[at] = (int)t;
          if constexpr (SPLIT) { if (wide_warp) high[at] = (int)(t >> 32); }
        }
        if (wide_warp && lane == 0) atomicOr((int*)s_wide, 1 << (cgroup * 4 + quarter));
      }
    }
    if constexpr (!SPLIT) {
      if (ok) ok = epi_sync();
      if (ok && !*s_wide) {
#pragma unroll 1
        for (int m = warp - 2; m < live_rows; m += EPIW) {
          const int4 v = *reinterpret_cast<const int4*>(stage32 + m * 128 + lane * 4);
          emit(m, v.x, v.y, v.z, v.w);
        }
      } else if (ok) {
        // some sums need 64 bits: half of the rows at a time
#pragma unroll 1
        for (int half = 0; half < 2 && ok; ++half) {
          if (!(ok = epi_sync())) break;
          if (cgroup >> 1 == half) {
#pragma unroll
            for (int i = 0; i < kCols; ++i)
              stage64[(m0 - half * (MP / 2) + i) * 128 + n_in_tile] = corr_used ? corr_q[i + zero] : (long long)(int32_t)total32(i);
          }
          if (!(ok = epi_sync())) break;
#pragma unroll 1
          for (int m = warp - 2; m < MP / 2 && half * (MP / 2) + m < live_rows; m += EPIW) {
            const longlong2 v = *reinterpret_cast<const longlong2*>(stage64 + m * 128 + lane * 4);
            const longlong2 w = *reinterpret_cast<const longlong2*>(stage64 + m * 128 + lane * 4 + 2);
            emit(half * (MP / 2) + m, v.x, v.y, w.x, w.y);
          }
        }
      }
    } else {
      // ------------------------------ merge of the splits ---------------------------
      // As in the decode-shape kernel, among the CTAs of the same columns: once every CTA's stages are done, a split
      // sends each of the others its rows (and its flag) by bulk copies, then sums its own.  Every
      // thread of every CTA arrives at and waits for both cluster barriers, also after a timed-out wait.
      const int my_rows = rows_of(ks);
      if (!announced) cluster_arrive();
      fence_proxy_async_smem();                            // what this thread parked, for the bulk copies
      if (ok) ok = epi_sync();
      cluster_wait();
      if (ok) {
        const int to = warp - 2;                           // warp w sends split w's rows
        if (to < S && to != ks && lane == 0 && rows_of(to) > 0) {
          const int slot = ks < to ? ks : ks - 1;
          const uint32_t peer = (uint32_t)(2 * to + parity), bar = mapa_u32(recv_bar, peer);
          if (*s_wide) mbar_arrive_release_cluster(mapa_u32(high_bar, peer));   // peers read the high words with plain loads
          bulk_copy_cluster(mapa_u32(smem_base + Shape::kRecvOffset + (uint32_t)(slot * rows_of(to) * 512), peer),
                            smem_base + (uint32_t)(to * rows_per * 512), (uint32_t)(rows_of(to) * 512), bar);
          bulk_copy_cluster(mapa_u32(smem_base + Shape::kFlagOffset + (uint32_t)(slot * 16), peer),
                            smem_u32((const void*)s_wide), 16u, bar);
        }
        __syncwarp();
        if (my_rows > 0) ok = warp_wait(recv_bar, 0, abort_flag);
      }
      unsigned long long wide = 0;                         // 16 bits a split: its warps that parked high words
      if (ok && my_rows > 0) {
        const int* flags = reinterpret_cast<const int*>(smem_gen + Shape::kFlagOffset);
        wide = (unsigned long long)(uint32_t)*s_wide << (16 * ks);
        for (int rr = 0; rr < S - 1; ++rr) wide |= (unsigned long long)(uint32_t)flags[rr * 4] << (16 * (rr < ks ? rr : rr + 1));
      }
      if (!wide) cluster_arrive();                         // this CTA has what was sent to it
      if (ok) {
        const int* mine = stage32 + ks * rows_per * 128;
        const int* recv = reinterpret_cast<const int*>(smem_gen + Shape::kRecvOffset);
        if (!wide && (k_tiles_total <= 510 || p.int_bits == 32)) {
          // sums over all splits are below 2^31 in magnitude, or wrap to 32 bits
#pragma unroll 1
          for (int mr = warp - 2; mr < my_rows; mr += EPIW) {
            int4 q = *reinterpret_cast<const int4*>(mine + mr * 128 + lane * 4);
            for (int rr = 0; rr < S - 1; ++rr) {
              const int4 v = *reinterpret_cast<const int4*>(recv + (rr * my_rows + mr) * 128 + lane * 4);
              q.x = wrap_add(q.x, v.x); q.y = wrap_add(q.y, v.y); q.z = wrap_add(q.z, v.z); q.w = wrap_add(q.w, v.w);
            }
            emit(ks * rows_per + mr, q.x, q.y, q.z, q.w);
          }
        } else {
          if (wide) {
            // the high words of every peer that has some; its own arrivals stand for the other peers
            if (warp == 2 && lane == 0) {
              int none = S - 1;
              for (int s = 0; s < S; ++s) none -= s != ks && ((wide >> (16 * s)) & 0xffff);
              if (none) mbar_arrive_n(high_bar, (uint32_t)none);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait_acquire_cluster(high_bar, 0, abort_flag));
          }
#pragma unroll 1
          for (int mr = warp - 2; ok && mr < my_rows; mr += EPIW) {
            const int m = ks * rows_per + mr;
            long long q[4] = {0, 0, 0, 0};
#pragma unroll 1
            for (int s = 0; s < S; ++s) {
              const int* low = s == ks ? mine + mr * 128 : recv + ((s < ks ? s : s - 1) * my_rows + mr) * 128;
              const uint32_t high = mapa_u32(smem_base + Shape::kHighOffset + (uint32_t)((m * 128 + lane * 4) * 4), (uint32_t)(2 * s + parity));
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int lo = low[lane * 4 + i];
                if ((wide >> (16 * s + m / kCols * 4 + (lane >> 3))) & 1) {
                  q[i] += ((long long)ld_cluster_s32(high + 4u * i) << 32) | (long long)(uint32_t)lo;
                } else {
                  q[i] += (long long)lo;
                }
              }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = p.int_bits == 64 ? q[i] : (long long)(int32_t)q[i];
            emit(m, q[0], q[1], q[2], q[3]);
          }
        }
      }
      if (wide) cluster_arrive();
    }
  }
  __syncwarp();
  if constexpr (SPLIT) {
    // the roles' halves of the merge's two barriers
    if (warp < 2) { cluster_arrive(); cluster_wait(); cluster_arrive(); }
    cluster_wait();                                        // the peers have what this CTA sent
  }

  // ------------------------------ teardown ----------------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // let copies that are still in flight land before shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 200000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, FXPR_ERR_TIMEOUT);
    __syncthreads();
  }
  // Neither CTA may leave while the other can still signal its barriers or while MMAs that read its
  // shared memory are in flight (the last tfull commit, which the epilogues wait for, covers those).
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

bool gemm_tc_fast_supported(const GemmArgs& g, int split_k);

// Numeric conditions of gemm_tc_fast.cu; no dump of the partials.
bool gemm_tc_mid_supported(const GemmArgs& g, int split_k) {
  return split_k <= 4 && g.M > 64 && g.N >= 128 && g.partials == nullptr && (g.N + 255) / 256 <= 65535 &&
         gemm_tc_fast_supported(g, split_k);
}

template <typename T, int MP, bool SPLIT>
static int launch_mid(const GemmArgs& g, const CUtensorMap& mw, int w_box, TcParams& p, int row_tiles, cudaStream_t s) {
  constexpr int kSmem = MdShape<MP>::kSmem;
  CUtensorMap mx;
  if (!tc_make_map(&mx, g.dtype, g.a, g.M, g.K, g.a_sm, MP / 2)) {
    set_last_error("cuTensorMapEncodeTiled(X)", cudaErrorInvalidValue);
    return FXPR_ERR_CUDA;
  }
  // M = 256 weight columns, N = activation rows; bit 15: the M-side operand is MN-major
  p.idesc = make_idesc(g.dtype == FXPR_BF16 ? 1 : 0, 0, MP, 256) | (p.b_kmajor ? 0u : (1u << 15));
  auto k = gemm_tc_mid_kernel<T, MP, SPLIT>;
  static bool attr_done_dev[64] = {};            // function attributes are per device
  int dev_id = 0;
  cudaGetDevice(&dev_id);
  bool& attr_done = attr_done_dev[dev_id & 63];
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) { set_last_error("gemm_tc_mid smem attribute", e); return FXPR_ERR_CUDA; }
    attr_done = true;
  }
  const dim3 grid((unsigned)(2 * p.split_k), (unsigned)((p.N + 255) / 256), (unsigned)row_tiles);
  const int tile_rows = (p.M + row_tiles - 1) / row_tiles;
  cudaError_t e = launch_pdl(k, grid, dim3(kMdThreads), kSmem, s, 2u * (unsigned)p.split_k, mw, mx, p, tile_rows, w_box, 0);
  if (e != cudaSuccess) { set_last_error("gemm_tc_mid launch", e); return FXPR_ERR_CUDA; }
  return check_launch("gemm_tc_mid");
}

template <typename T>
static int route_mid(const GemmArgs& g, TcParams& p, int row_tiles, cudaStream_t s) {
  CUtensorMap mw;
  int w_box = 0;
  if (p.b_kmajor) {
    if (tc_make_map(&mw, g.dtype, g.b, g.N, g.K, g.b_sn, 128)) w_box = 2;
  } else if (tc_make_map_groups(&mw, g.dtype, g.b, g.K, g.N, g.b_sk, 64)) {
    w_box = 3;
  }
  if (!w_box && (p.b_kmajor || !tc_make_map(&mw, g.dtype, g.b, g.K, g.N, g.b_sk, 64))) {
    set_last_error("cuTensorMapEncodeTiled(W)", cudaErrorInvalidValue);
    return FXPR_ERR_CUDA;
  }
  const int rows = (p.M + row_tiles - 1) / row_tiles;
  if (p.split_k > 1) {
    if (rows <= 96) return launch_mid<T, 96, true>(g, mw, w_box, p, row_tiles, s);
    return launch_mid<T, 128, true>(g, mw, w_box, p, row_tiles, s);
  }
  if (rows <= 96) return launch_mid<T, 96, false>(g, mw, w_box, p, row_tiles, s);
  if (rows <= 128) return launch_mid<T, 128, false>(g, mw, w_box, p, row_tiles, s);
  if (rows <= 160) return launch_mid<T, 160, false>(g, mw, w_box, p, row_tiles, s);
  if (rows <= 192) return launch_mid<T, 192, false>(g, mw, w_box, p, row_tiles, s);
  if (rows <= 224) return launch_mid<T, 224, false>(g, mw, w_box, p, row_tiles, s);
  return launch_mid<T, 256, false>(g, mw, w_box, p, row_tiles, s);
}

// row_tiles: at most 256 rows each, 128 where K is split.
int gemm_tc_mid(const GemmArgs& g, TcParams& p, int row_tiles, cudaStream_t s) {
  if (g.dtype == FXPR_BF16) return route_mid<__nv_bfloat16>(g, p, row_tiles, s);
  return route_mid<__half>(g, p, row_tiles, s);
}

}  // namespace fxpr
