// Two-SM route of the tensor-core fixed-point GEMM (sm_100a): tcgen05.mma with cta_group::2 on
// clusters of two CTAs, one 256 x 256 output tile per pair.  The default for large products.
//
// What bounds it.  The single-CTA kernels pull 48 KB of operands per 64-deep step of a 128 x 256
// tile out of L2 (~140 us at 4096^3, against 82 us of tensor work).  Here each CTA loads its own 128
// rows of A and its own 128 columns of B, 32 KB per step for the same accumulator; the tensor cores
// of both SMs read both halves of B, and each CTA's tensor memory receives its 128 rows x 256
// columns: with the conversion left out the kernel runs at 100 us.  What is left is the conversion.  By
// itself a K-tile's 32768 partials take an SM about 760 clocks (packed add, integer add, range screen =
// 2.4 issue slots per partial); in the kernel its warps need about 1150, as the four tcgen05.ld of a warp
// are waited for one after the other (103 clocks each) and the other warps take issue slots.  At K-tile 64
// (512 clocks of tensor work, 1350 a K-tile all in) they are at work 84 % of the time, ALU pipe 64 %, and
// the tensor core waits for accumulators; at K-tile 128 (1024 clocks of tensor work) they wait a quarter
// of the time and the tensor pipe is busy 63 %: the hand-over, next to operands at 8.4 TB/s out of L2.  Outputs
// leave by TMA: stored by the threads they held the epilogue warps for 7700-8400 clocks a tile.  4096^3 in a graph,
// outputs by the threads -> by TMA -> with every sum converted in registers: K-tile 64 196 -> 187 -> 186 us, K-tile 128
// 139 -> 134 -> 130 (a call among others at K-tile 64: 218 -> 208 -> 203).
//
// What it depends on, measured at 4096^3 with the conversion left out:
//   - MMAs, commits and copies are predicated instructions of a uniform warp (tc_common.cuh);
//   - the "accumulator drained" arrival crosses to the leader CTA as a plain mbarrier.arrive: with
//     .release.cluster on it (a cluster-wide fence behind the TMA traffic) K-tile 64 took 242 us
//     instead of 126, K-tile 128 156 instead of 109;
//   - one 256-column accumulator per K-tile and two of them in tensor memory: four of 128 columns
//     double the hand-offs and measured 175 us instead of 126 at K-tile 64.
//
// Roles per CTA (18 warps): warp 0 = TMA producer (both CTAs, each for its own shared memory; the
// copies of both complete on the leader's "full" barrier), warp 1 = MMA issuer (leader only; its
// commits arrive on the barriers of both CTAs), warps 2-17 = epilogue: thread = one row and 64
// columns, so the running sums fit the 96 registers an 18-warp CTA has.
//
// Numerics, the conversion with its range screen and exact fix-up are those of gemm_tc_fast.cu
// (gemm_tc_fast_common.cuh); results are bit-identical to it (the fixed-point contract:
// fxpr_vllm/_triton/gemm.py:183-204).  Every wait is bounded.
#include <cstring>
#include <type_traits>

#include <cuda.h>

#include "fxp_common.cuh"
#include "gemm_common.cuh"
#include "tc_common.cuh"
#include "gemm_tc_fast_common.cuh"

namespace fxpr {

static constexpr int kPrEpiW = 16;
static constexpr int kPrFirstEpi = 2;
static constexpr int kPrThreads = (kPrFirstEpi + kPrEpiW) * 32;
static constexpr int kPrGroupM = 4;        // pair-tile rows (256 each) per L2 group

static constexpr int kPrStages = 6;
static constexpr int kPrABytes = kBM * kBK * 2;            // this CTA's 128 rows of A
static constexpr int kPrBBytes = 128 * kBK * 2;            // this CTA's 128 columns of B
static constexpr int kPrStageBytes = kPrABytes + kPrBBytes;
static constexpr int kPrOutBytes = 32 * 64;                // half of a warp's output: 32 rows of 32 columns
static constexpr int kPrSmem = kPrStages * kPrStageBytes + kPrEpiW * kPrOutBytes + 256 + 1024;
static_assert(kPrSmem <= 227 * 1024, "shared memory of an SM");
static constexpr int kPrCols = 64;                         // accumulator columns per epilogue thread

template <typename T, bool INTS>
__global__ void __launch_bounds__(kPrThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                    const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_ci,
                    const TcParams p, const int zero /* always 0: keeps the side arrays in local memory */) {
  constexpr int kOutOffset = kPrStages * kPrStageBytes, kBarOffset = kOutOffset + kPrEpiW * kPrOutBytes;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kBarOffset;
  // full[stage]: the leader's arrive plus the bytes of both CTAs; empty[stage], tfull[buffer]: one
  // commit, in both CTAs; tempty[buffer] (leader): the epilogue warps of both CTAs
  const uint32_t full0 = bar_base, empty0 = full0 + 8u * kPrStages;
  const uint32_t tfull0 = empty0 + 8u * kPrStages, tempty0 = tfull0 + 16u;
  constexpr int kMisc = 16 * kPrStages + 32;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem_gen + kBarOffset + kMisc);
  volatile int* abort_flag = (volatile int*)(smem_gen + kBarOffset + kMisc + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();                 // 0 = leader
  const int pair_id = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPrStages; ++s) { mbar_init(full0 + 8u * s, 1); mbar_init(empty0 + 8u * s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(tfull0 + 8u * b, 1); mbar_init(tempty0 + 8u * b, 2 * kPrEpiW); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32((const void*)tmem_slot), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                      // the peer's barriers exist from here on
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int items = p.tiles_m * p.tiles_n;                 // pair tiles of 256 x 256
  const int n_kt = (p.K + p.k_tile - 1) / p.k_tile;
  const int halves = p.k_tile / 64;                        // stages per K-tile: 1 or 2

  auto tile_coords = [&](int tile, int& pm, int& pn) {
    const int in_group = kPrGroupM * p.tiles_n;
    const int g = tile / in_group;
    const int first = g * kPrGroupM;
    const int gsz = min(p.tiles_m - first, kPrGroupM);
    pm = first + (tile % in_group) % gsz;
    pn = (tile % in_group) / gsz;
  };

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ----------------------
    const uint32_t e = elect_one();
    const bool bk = p.b_kmajor != 0;
    const uint32_t full_leader = mapa_u32(full0, 0);       // the leader's barriers count both CTAs' bytes
    int stage = 0; uint32_t phase = 1;
    for (int item = pair_id; item < items; item += num_pairs) {
      int pm, pn; tile_coords(item, pm, pn);
      const int m0 = pm * 256 + (int)rank * kBM;
      const int n0 = pn * 256 + (int)rank * 128;
      for (int i = 0; i < n_kt * halves; ++i) {
        const int k0 = i * 64;
        if (!__all_sync(0xffffffffu, mbar_wait_poll(empty0 + 8u * stage, phase, abort_flag))) goto producer_done;
        const uint32_t fb = full_leader + 8u * stage;
        const uint32_t sa = smem_base + stage * kPrStageBytes;
        const uint32_t sb = sa + kPrABytes;
        if (rank == 0) mbar_expect_tx(full0 + 8u * stage, 2 * kPrStageBytes, e);
        tma_load_2d_pair(sa, &tma_a, fb, k0, m0, e);
        tma_load_2d_pair(sb, &tma_b, fb, bk ? k0 : n0, bk ? n0 : k0, e);
        tma_load_2d_pair(sb + 8192, &tma_b, fb, bk ? k0 : n0 + 64, bk ? n0 + 64 : k0, e);
        if (++stage == kPrStages) { stage = 0; phase ^= 1; }
      }
    }
  producer_done:;
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader only) ----------------------
    if (rank == 0) {
      const uint32_t e = elect_one();
      const uint64_t adesc0 = make_smem_desc(smem_base, 16, 1024);
      const uint64_t bdesc0 = p.b_kmajor ? make_smem_desc(smem_base + kPrABytes, 16, 1024)
                                         : make_smem_desc(smem_base + kPrABytes, 8192, 1024);
      const uint64_t bks = p.b_kmajor ? 2 : 128;          // (32 B | 2048 B) >> 4 per 16-deep k step
      constexpr uint64_t kStep = kPrStageBytes >> 4;
      const uint32_t idesc = p.idesc;
      int stage = 0; uint32_t phase = 0; int buf = 0; uint32_t bphase = 1;
      for (int item = pair_id; item < items; item += num_pairs) {
        for (int i = 0; i < n_kt; ++i) {
          const uint32_t d = tmem_base + (uint32_t)(buf * 256);
          for (int h = 0; h < halves; ++h) {
            // the operands usually wait for the accumulator, so that is asked last
            if (!__all_sync(0xffffffffu, mbar_wait_poll(full0 + 8u * stage, phase, abort_flag))) goto issuer_done;
            if (h == 0 && !__all_sync(0xffffffffu, mbar_wait_poll(tempty0 + 8u * buf, bphase, abort_flag))) goto issuer_done;
            tc_fence_after();
            const uint64_t ad = adesc0 + (uint64_t)stage * kStep;
            const uint64_t bd = bdesc0 + (uint64_t)stage * kStep;
#pragma unroll
            for (int q = 0; q < 4; ++q) umma_f16_pair(d, ad + 2 * q, bd + q * bks, idesc, (h || q) ? 1u : 0u, e);
            umma_commit_pair(empty0 + 8u * stage, 3, e);
            if (h == halves - 1) umma_commit_pair(tfull0 + 8u * buf, 3, e);
            if (++stage == kPrStages) { stage = 0; phase ^= 1; }
          }
          buf ^= 1; if (buf == 0) bphase ^= 1;
        }
      }
    issuer_done:;
    }
  } else {
    // ------------------------------ epilogue warps (both CTAs) --------------------
    const int quarter = warp & 3;
    const int cgroup = (warp - kPrFirstEpi) >> 2;
    const uint32_t lane_addr = ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cgroup * kPrCols);
    const float scale = p.scale;
    const uint32_t mbits = q_magic_bits(p.inv_scale);
    const uint64_t magic2 = pack2(mbits, mbits);
    const float screen_limit = q_screen_limit(p.inv_scale);
    const uint32_t one = (uint32_t)zero + 1u;
    const uint32_t tempty_leader = mapa_u32(tempty0, 0);
    int buf = 0; uint32_t bphase = 0; bool ok = true;
    // Rare-path corrections (local memory, zeroed on first use): wrap-sum of the raw values the fast
    // add contributed for out-of-range partials, and the exact int64 sum of what the reference
    // conversion gives for them.
    uint32_t corr_raw[kPrCols];
    long long corr_q[kPrCols];
    bool corr_used = false;

    for (int item = pair_id; item < items && ok; item += num_pairs) {
      uint32_t acc[kPrCols];
#pragma unroll
      for (int i = 0; i < kPrCols; ++i) acc[i] = 0;
      corr_used = false;
      for (int kt = 0; kt < n_kt; ++kt) {
        if (!warp_wait(tfull0 + 8u * buf, bphase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + lane_addr + (uint32_t)(buf * 256);
        float screen = 0.0f;
#pragma unroll
        for (int c = 0; c < kPrCols / 16; ++c) {
          uint32_t v[16];
          tmem_ld16(taddr + c * 16, v);
          tmem_wait_ld_regs(v);
          float tail = 0.0f;
          if (c + 1 == kPrCols / 16) {
            // the last chunk is in registers: screen it and hand the buffer back before converting it
#pragma unroll
            for (int i = 0; i < 16; i += 2) screen = max3_abs(screen, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
            if (__any_sync(0xffffffffu, !(screen < screen_limit))) {
              if (!corr_used) {
#pragma unroll 1
                for (int z = 0; z < kPrCols; ++z) { corr_raw[z + zero] = 0; corr_q[z + zero] = 0; }
                corr_used = true;
              }
              fixup_tile(taddr, kPrCols, mbits, scale, p.int_bits, &corr_raw[zero], &corr_q[zero]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(tempty_leader + 8u * buf);
          }
          convert16(v, &acc[c * 16], magic2, mbits, one, c + 1 == kPrCols / 16 ? tail : screen);
        }
        buf ^= 1; if (buf == 0) bphase ^= 1;
      }
      if (!ok) break;

      int pm, pn; tile_coords(item, pm, pn);
      const int row = pm * 256 + (int)rank * kBM + quarter * 32 + lane;
      const int col0 = pn * 256 + cgroup * kPrCols;
      const uint32_t bias_bits = (uint32_t)n_kt * mbits;   // what the multiply-adds summed on top
      const T* bias = (const T*)p.bias;
      // Sums fit 32 bits unless a partial took the fix-up, and are converted to float where the outputs are made, one
      // instruction each, whatever their size.  (Sums below 2^22 allow a shortcut, MAGIC + sum as a float, but its
      // test, and any second form next to it, spills in the main loop: 4096^3, K-tile 128, us: shortcut and a loop out
      // of local memory for larger sums 134 and 314, both in registers 138 and 137, this one 130 and 127; K-tile 64:
      // 187 and 370, 199 and 202, 186 and 187.)  After a fix-up the exact 64-bit sums, as floats, are put together out of
      // local memory, in a loop.
      if (corr_used) {
        uint32_t sums[kPrCols];
#pragma unroll
        for (int i = 0; i < kPrCols; ++i) sums[i + zero] = alu_add(i) ? acc[i] : acc[i] - bias_bits;
#pragma unroll 4
        for (int c = 0; c < kPrCols; ++c) {
          // the in-range part is < 2^31 in magnitude, so it is the sign extension of the wrapped sum once
          // the out-of-range raw values are taken out again
          long long t = (long long)(int32_t)(sums[c + zero] - corr_raw[c + zero]) + corr_q[c + zero];
          if (p.int_bits != 64) t = (long long)(int32_t)t;
          if constexpr (INTS) corr_q[c + zero] = t;
          sums[c + zero] = __float_as_uint(__ll2float_rn(t));
        }
#pragma unroll
        for (int i = 0; i < kPrCols; ++i) acc[i] = sums[i + zero];
      } else {
#pragma unroll
        for (int i = 0; i < kPrCols; ++i) {
          if (!alu_add(i)) acc[i] -= bias_bits;
          if constexpr (INTS) corr_q[i + zero] = (long long)(int)acc[i];
        }
      }
      if (col0 < p.N && row - lane < p.M) {
        // 32 rows x 64 bytes at a time go through shared memory and leave by TMA, which clips them to the matrix, while
        // the next tile is converted.  (Stored by the threads, a row each, an output took the epilogue warps 7700-8400
        // clocks a tile: all SMs write at the same time, and the stores wait.)  A matrix that no tensor map can
        // describe is written from there by rows.
        const uint32_t out_s = smem_base + kOutOffset + (uint32_t)((warp - kPrFirstEpi) * kPrOutBytes);
        auto staging_free = [&]() {
          tma_store_wait_read();                           // the last store has read it
          __syncwarp();
        };
        // 16-byte chunks swizzled with the row, as the tensor maps say
        auto at = [&](int r, int chunk) { return out_s + (uint32_t)(r * 64 + ((chunk ^ ((r >> 1) & 3)) << 4)); };
        auto put = [&](int chunk, const uint32_t* w) {
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                       ::"r"(at(lane, chunk)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        };
        auto leave = [&](const CUtensorMap* map, bool tma, int x, auto* base, int64_t stride) {
          using E = std::remove_pointer_t<decltype(base)>;
          if (tma) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && x < p.N) {
              tma_store_2d(map, out_s, x, row);
              tma_store_commit();
            }
          } else {
            constexpr int kPerRow = 64 / (int)sizeof(E), kRows = 32 / kPerRow;
            const int e = lane % kPerRow;
            __syncwarp();
#pragma unroll 4
            for (int r = lane / kPerRow; r < 32; r += kRows) {
              const uint32_t from = at(r, e * (int)sizeof(E) >> 4) + (uint32_t)(e * (int)sizeof(E) & 15);
              E v;
              memcpy(&v, smem_gen + (from - smem_base), sizeof(E));
              if (row - lane + r < p.M && x + e < p.N) base[(int64_t)(row - lane + r) * stride + x + e] = v;
            }
          }
        };
        if constexpr (INTS) {
          const long long* q = &corr_q[zero];
          if (p.int_bits == 64) {
#pragma unroll 1
            for (int h = 0; h < kPrCols; h += 8) {
              staging_free();
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const long long a = q[h + 2 * g], b = q[h + 2 * g + 1];
                const uint32_t w[4] = {(uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32)};
                put(g, w);
              }
              leave(&tma_ci, p.ci_tma, col0 + h, (long long*)p.c_int, p.N);
            }
          } else {
#pragma unroll 1
            for (int h = 0; h < kPrCols; h += 16) {
              staging_free();
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const int c = h + 4 * g;
                const uint32_t w[4] = {(uint32_t)q[c], (uint32_t)q[c + 1], (uint32_t)q[c + 2], (uint32_t)q[c + 3]};
                put(g, w);
              }
              leave(&tma_ci, p.ci_tma, col0 + h, (int32_t*)p.c_int, p.N);
            }
          }
        }
        if (!INTS || p.c) {
          const float inv = p.inv_scale;
#pragma unroll
          for (int h = 0; h < kPrCols; h += 32) {
            staging_free();
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              alignas(16) T out[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int c = h + g * 8 + i;
                float v = __fmul_rn(corr_used ? __uint_as_float(acc[c]) : __int2float_rn((int)acc[c]), inv);
                if (bias) v = __fadd_rn(v, col0 + c < p.N ? to_f32<T>(bias[col0 + c]) : 0.0f);
                out[i] = from_f32<T>(v);
              }
              put(g, reinterpret_cast<const uint32_t*>(out));
            }
            leave(&tma_c, p.c_tma, col0 + h, (T*)p.c, p.c_sm);
          }
        }
      }
    }
    tma_store_wait_read();                                 // the staging is this CTA's until its stores have read it
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

// Numeric conditions of gemm_tc_fast.cu (int32 / int64 sums, frac_bits <= 21, at most 510 K-tiles);
// no K-split and no dump of the partials.
bool gemm_tc_pair_supported(const GemmArgs& g, int split_k) {
  return split_k == 1 && g.partials == nullptr && g.M > 128 && g.N >= 128 && gemm_tc_fast_supported(g, split_k);
}

template <typename T, bool INTS>
static int launch_pair(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const CUtensorMap& mci,
                       TcParams& p, int sms, cudaStream_t s) {
  auto k = gemm_tc_pair_kernel<T, INTS>;
  static bool attr_done_dev[64] = {};            // function attributes are per device
  int dev_id = 0;
  cudaGetDevice(&dev_id);
  bool& attr_done = attr_done_dev[dev_id & 63];
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrSmem);
    if (e != cudaSuccess) { set_last_error("gemm_tc_pair smem attribute", e); return FXPR_ERR_CUDA; }
    attr_done = true;
  }
  p.tiles_m = (p.M + 255) / 256;
  p.tiles_n = (p.N + 255) / 256;
  const int64_t items = (int64_t)p.tiles_m * p.tiles_n;
  const int pairs = (int)(items < sms / 2 ? items : sms / 2);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
  cfg.blockDim = dim3(kPrThreads, 1, 1);
  cfg.dynamicSmemBytes = kPrSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, k, ma, mb, mc, mci, (const TcParams)p, 0);
  if (e != cudaSuccess) { set_last_error("gemm_tc_pair launch", e); return FXPR_ERR_CUDA; }
  return check_launch("gemm_tc_pair");
}

// ma, mb: the tensor maps of gemm_tc() (A: 128-row boxes, B: 64-row boxes in either layout).
int gemm_tc_pair(const GemmArgs& g, TcParams& p, const CUtensorMap& ma, const CUtensorMap& mb, cudaStream_t s) {
  const int sms = tc_device_sms();
  if (sms < 0) return FXPR_ERR_ARCH;
  p.idesc = make_idesc(g.dtype == FXPR_BF16 ? 1 : 0, p.b_kmajor ? 0 : 1, 256, 256);
  // outputs by TMA where a tensor map can say where they are: rows that start on 16 bytes
  CUtensorMap mc = ma, mci = ma;
  p.c_tma = p.c_vec_ok && tc_make_map(&mc, g.dtype, g.c, g.M, g.N, g.c_sm, 32, 32);
  p.ci_tma = p.c_int && !((uintptr_t)p.c_int & 15) && (int64_t)p.N * (p.int_bits / 8) % 16 == 0 &&
             tc_make_map_int(&mci, p.int_bits, p.c_int, g.M, g.N, 32);
  if (g.dtype == FXPR_BF16)
    return p.c_int ? launch_pair<__nv_bfloat16, true>(ma, mb, mc, mci, p, sms, s) : launch_pair<__nv_bfloat16, false>(ma, mb, mc, mci, p, sms, s);
  return p.c_int ? launch_pair<__half, true>(ma, mb, mc, mci, p, sms, s) : launch_pair<__half, false>(ma, mb, mc, mci, p, sms, s);
}

}  // namespace fxpr
