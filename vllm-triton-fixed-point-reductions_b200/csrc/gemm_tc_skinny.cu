// Tensor-core fixed-point GEMM for decode shapes (M <= 64 rows of activations against a
// large weight matrix): the operands swap roles.  The 128-row side of tcgen05.mma carries
// 128 output COLUMNS (weights), its N side the padded activation rows:
//
//     D^T[n, m] = sum_k W[k, n] * X[m, k]        M_mma = 128 (n), N_mma = 16, 32 or 64 (m), K = 16
//
// so a K-tile's accumulator is 128 x 64 at most (a quarter of the conversion work per byte of weights, next
// to 128 x 128 tiles), rows are padded to 16, 32 or 64, and tensor memory holds four to eight accumulators.
// A stage is 64 deep in K, 16 KB of weights.
// Bound: streaming the weights from HBM once, plus what a call waits for before the first and after the last
// byte.  Against one CTA per SM with persistent tiles, all rows padded to 64, 64-bit partials pulled over
// distributed shared memory and outputs written out of registers (cold weights, CUDA graph, us):
//   16 x 4096 x 4096 13.0 -> 9.9 (weights alone 5.2), 64 x 4096 x 4096 13.3 -> 11.3, 64 x 6144 x 4096 17.6 -> 13.7,
//   64 x 28672 x 4096 46.5 -> 38.7 (weights alone 36.4), 64 x 768 x 4096 9.0 -> 6.9, 64 x 4096 x 512 8.2 -> 6.0.
// More than 32 rows on more tiles than two CTAs an SM are walked by persistent CTAs (route_skinny).
//
// Numerics are those of the other tensor-core kernels: one fp32 partial per K-tile and
// output element from tcgen05.mma (kind::f16, fp32 accumulate, fresh accumulator per
// K-tile), rint-half-even conversion to Q-format on the FP32 pipe with the exact fix-up for
// out-of-range partials, wrap-around integer sums; split-K through per-split partial planes.
// An output element's bits do not depend on M, on the route or on the split count.
#include <cuda.h>

#include "fxp_common.cuh"
#include "gemm_common.cuh"
#include "tc_common.cuh"
#include "gemm_tc_fast_common.cuh"

namespace fxpr {

static constexpr int kSkMaxRows = 64;
static constexpr int kSkWarps = 2 + 8;                    // producer, issuer, 8 epilogue warps
static constexpr int kSkWBytes = 128 * kBK * 2;           // weights of a stage: 64 of K, 128 columns
static constexpr int kSkTmemCols = 256;                   // two CTAs share an SM's 512

// Most rows that one rank of a cluster merge receives, all its peers together, over 2 to 8 ranks: with 64 rows it
// is seven ranks of ten rows (60), not eight of eight.
constexpr int sk_most_received(int rows) {
  int most = 0;
  for (int ranks = 2; ranks <= 8; ++ranks) {
    const int got = (ranks - 1) * ((rows + ranks - 1) / ranks);
    if (got > most) most = got;
  }
  return most;
}

// MP = activation rows of the tile (MMA N).  PER_SM = CTAs that share an SM's memory.  WALK: a CTA takes tile after
// tile, with the sums beside the ring and not over it.
template <int MP, int PER_SM, bool WALK> struct SkShape {
  static constexpr int kStages = (MP == 16 ? 12 : MP == 32 ? 10 : 8) / PER_SM - (WALK ? 1 : 0);
  static constexpr int kXBytes = MP * kBK * 2;
  static constexpr int kStageBytes = kSkWBytes + kXBytes;  // 18, 20 or 24 KB
  static constexpr int kGroups = MP == 64 ? 4 : 8;         // accumulators in tensor memory
  static constexpr int kSumsOffset = WALK ? kStages * kStageBytes : 0;
  static constexpr int kBarOffset = kStages * kStageBytes + (WALK ? MP * 512 : 0);
  static constexpr int kBarBytes = 448;
  static constexpr int kSmem = kBarOffset + kBarBytes + 1024;   // barriers, alignment slack
  // over the stages once they are done: the finished sums, [row][128 columns] of 32 bits; for the cluster merge what the
  // peers send for this rank's rows, their flags, this rank's high words
  static constexpr int kRecvOffset = 32 * 1024, kFlagOffset = 62 * 1024, kHighOffset = 64 * 1024;
  static_assert(MP * 512 <= kRecvOffset && kRecvOffset + sk_most_received(MP) * 512 <= kFlagOffset, "sums and received slices");
  static_assert(kFlagOffset + 7 * 16 <= kHighOffset, "a flag of 16 bytes from each peer");
  static_assert(WALK || kHighOffset + MP * 512 <= kBarOffset, "the merge fits the stages");
  static_assert(PER_SM * (kSmem + 1024) <= 228 * 1024, "shared memory of an SM");
  static_assert(kGroups * MP <= kSkTmemCols, "tensor memory");
};

// One item -- a tile of 128 columns and one K-split -- per CTA, or, with WALK and without splits, tile after tile.
// CLUSTER: split-K as a thread-block cluster (grid = splits x tiles): every rank sums a slice of the rows,
// which the others send it by bulk copies between shared memories -- no global scratch, no fences.
template <typename T, int MP, bool CLUSTER, int PER_SM, bool WALK>
__global__ void __launch_bounds__(kSkWarps * 32, 2)
gemm_tc_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                      const TcParams p, const int zero /* always 0: keeps the side arrays in local memory */) {
  using Shape = SkShape<MP, PER_SM, WALK>;
  static_assert(!(CLUSTER && WALK), "a walk has no splits");
  constexpr int STAGES = Shape::kStages, GROUPS = Shape::kGroups;
  constexpr int EPIW = 8;
  constexpr int kCols = MP / (EPIW / 4);                 // activation rows per epilogue thread
  constexpr int kXBytes = Shape::kXBytes, kStageBytes = Shape::kStageBytes, kBarOffset = Shape::kBarOffset;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kBarOffset;
  const uint32_t full0 = bar_base, empty0 = bar_base + 8u * STAGES;
  const uint32_t tfull0 = bar_base + 8u * (2 * STAGES), tempty0 = tfull0 + 8u * GROUPS;
  constexpr int kMisc = (8 * (2 * STAGES + 2 * GROUPS) + 15) / 16 * 16;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem_gen + kBarOffset + kMisc);
  volatile int* abort_flag = (volatile int*)(smem_gen + kBarOffset + kMisc + 8);
  const uint32_t epi_bar = bar_base + kMisc + 16u;
  volatile int* s_last = (volatile int*)(smem_gen + kBarOffset + kMisc + 24);
  const uint32_t recv_bar = bar_base + kMisc + 32u, high_bar = recv_bar + 8u;
  volatile int* s_wide = (volatile int*)(smem_gen + kBarOffset + kMisc + 48);   // 16 bytes, copied to the peers
  static_assert(kMisc + 64 <= Shape::kBarBytes, "barrier block");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Cluster merge: rank r sums rows [r * rows_per, ...) of the live ones over all ranks.
  const int live_rows = min(p.M, MP);
  const int rows_per = CLUSTER ? (live_rows + p.split_k - 1) / p.split_k : 0;
  auto rows_of = [&](int r) { return max(0, min(live_rows - r * rows_per, rows_per)); };

  pdl_launch_dependents();                               // the next kernel may start its own setup
  if (threadIdx.x == 64) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tma_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tma_x) : "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8u * s, 1); mbar_init(empty0 + 8u * s, 1); }
    for (int b = 0; b < GROUPS; ++b) { mbar_init(tfull0 + 8u * b, 1); mbar_init(tempty0 + 8u * b, EPIW); }
    mbar_init(epi_bar, EPIW);
    if constexpr (CLUSTER) { mbar_init(recv_bar, 1); mbar_init(high_bar, (uint32_t)(p.split_k - 1)); }
    *abort_flag = 0;
    for (int i = 0; i < 4; ++i) s_wide[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if constexpr (CLUSTER) {
      const int rows = rows_of((int)blockIdx.x);
      mbar_expect_tx(recv_bar, rows > 0 ? (uint32_t)((p.split_k - 1) * (rows * 512 + 16)) : 0u);
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32((const void*)tmem_slot), kSkTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Barriers, tensor memory and descriptors are set up; from here on the kernel reads what
  // earlier kernels of the stream wrote -- except, when the caller vouches for it
  // (FXPR_GEMM_WEIGHTS_STATIC), the weights: the producer warp then requests the weight boxes of
  // its first stages BEFORE it waits, so their HBM latency (~2.7 us cold) passes while the
  // previous kernel finishes.
  if (warp != 0) pdl_wait();

  const int tiles_n = p.tiles_n;                         // 128-column tiles; one row tile (M <= 64)
  const int tile0 = CLUSTER ? (int)blockIdx.y : WALK ? (int)blockIdx.x : (int)blockIdx.x / p.split_k;
  const int ks = CLUSTER ? (int)blockIdx.x : WALK ? 0 : (int)blockIdx.x % p.split_k;
  const int k_tiles_total = (p.K + p.k_tile - 1) / p.k_tile;
  const int n_kt = (k_tiles_total - ks + p.split_k - 1) / p.split_k;
  const int deep = p.k_tile >> 6;                        // stages per K-tile: 1 or 2
  const int n_st = n_kt * deep;

  if (warp == 0) {
    // ------------------------------ TMA producer --------------------------------
    const uint32_t e = elect_one();
    const bool wk = p.b_kmajor != 0;                     // weights given as an (N, K) row-major view
    int n0 = tile0 * 128;
    auto k_of = [&](int j) { return deep == 1 ? (ks + j * p.split_k) * 64 : (ks + (j >> 1) * p.split_k) * 128 + (j & 1) * 64; };
    auto load_w = [&](int j, int st) {
      const uint32_t fb = full0 + 8u * st, sw = smem_base + st * kStageBytes;
      const int kk = k_of(j);
      mbar_expect_tx(fb, kStageBytes, e);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        tma_load_2d(sw + h * 8192, &tma_w, fb, wk ? kk : n0 + h * 64, wk ? n0 + h * 64 : kk, e);
    };
    auto load_x = [&](int j, int st) {
      tma_load_2d(smem_base + st * kStageBytes + kSkWBytes, &tma_x, full0 + 8u * st, k_of(j), 0, e);
    };
    const int first = min(STAGES, n_st);
    if (p.w_static) {
      for (int j = 0; j < first; ++j) load_w(j, j);
      pdl_wait();
      for (int j = 0; j < first; ++j) load_x(j, j);
    } else {
      pdl_wait();
      for (int j = 0; j < first; ++j) { load_w(j, j); load_x(j, j); }
    }
    int stage = 0; uint32_t phase = 0;
    if (WALK && first < STAGES) { stage = first; phase = 1; }
    int j = first;
    for (;;) {
      bool fetched = true;
      for (; j < n_st; ++j) {
        if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8u * stage, phase, abort_flag))) { fetched = false; break; }
        load_w(j, stage); load_x(j, stage);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!WALK || !fetched || (n0 += (int)gridDim.x * 128) >= tiles_n * 128) break;
      j = 0;
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ----------------------------------
    // Weights are the 128-row operand: MN-major for a (K, N) row-major matrix, K-major for
    // an (N, K).t() view.  Activations are the K-major operand of MP rows.
    const uint64_t wdesc0 = p.b_kmajor ? make_smem_desc(smem_base, 16, 1024) : make_smem_desc(smem_base, 8192, 1024);
    const uint64_t xdesc0 = make_smem_desc(smem_base + kSkWBytes, 16, 1024);
    const uint64_t wks = p.b_kmajor ? 2 : 128;           // (32 B | 2048 B) >> 4 per 16-deep k step
    constexpr uint64_t kStep = kStageBytes >> 4;
    const uint32_t idesc = p.idesc, e = elect_one();
    int stage = 0; uint32_t phase = 0; int grp = 0; uint32_t gphase = 1;
    int t = tile0;
    do
    for (int kt = 0; kt < n_kt; ++kt) {
      const uint32_t d = tmem_base + (uint32_t)(grp * MP);
      for (int h = 0; h < deep; ++h) {
        const bool r1 = h || mbar_wait(tempty0 + 8u * grp, gphase, abort_flag);
        const bool r2 = mbar_wait(full0 + 8u * stage, phase, abort_flag);
        if (!__all_sync(0xffffffffu, r1 && r2)) goto issuer_done;
        tc_fence_after();
        const uint64_t wd = wdesc0 + (uint64_t)stage * kStep;
        const uint64_t xd = xdesc0 + (uint64_t)stage * kStep;
#pragma unroll
        for (int i = 0; i < 4; ++i) umma_f16(d, wd + i * wks, xd + i * 2, idesc, (h | i) ? 1u : 0u, e);
        umma_commit(empty0 + 8u * stage, e);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      umma_commit(tfull0 + 8u * grp, e);
      if (++grp == GROUPS) { grp = 0; gphase ^= 1; }
    }
    while (WALK && (t += (int)gridDim.x) < tiles_n);
  issuer_done:;
  } else {
#include "gemm_tc_skinny_epilogue.inl"
  }
  if constexpr (CLUSTER) {
    // the roles' halves of the merge's two barriers (gemm_tc_skinny_epilogue.inl)
    __syncwarp();
    if (warp < 2) { cluster_arrive(); cluster_wait(); cluster_arrive(); }
    cluster_wait();                                      // the peers have what this CTA sent
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
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kSkTmemCols);
  }
}

// The skinny route takes what the fast route takes (int32 / int64 sums, frac_bits <= 21,
// k_tile 64 or 128, at most 510 K-tiles per item) when all rows fit one 64-row tile.
bool gemm_tc_fast_supported(const GemmArgs& g, int split_k);

bool gemm_tc_skinny_supported(const GemmArgs& g, int split_k) {
  return g.M <= kSkMaxRows && g.partials == nullptr && gemm_tc_fast_supported(g, split_k);
}

// 2 to 8 splits run as a thread-block cluster (merge through distributed shared memory, no scratch);
// larger split counts use the partial planes in the caller's scratch.  Same bits either way.
bool gemm_tc_skinny_cluster(const GemmArgs& g, int split_k) {
  return split_k >= 2 && split_k <= 8 && (g.N + 127) / 128 <= 65535 && !(g.flags & FXPR_GEMM_NO_CLUSTER);
}

template <typename T, int MP, bool CLUSTER, int PER_SM, bool WALK = false>
static int launch_skinny(const GemmArgs& g, const CUtensorMap& mw, TcParams& p, cudaStream_t s, int walkers = 0) {
  constexpr int kSmem = SkShape<MP, PER_SM, WALK>::kSmem;
  CUtensorMap mx;
  if (!tc_make_map(&mx, g.dtype, g.a, g.M, g.K, g.a_sm, MP)) {
    set_last_error("cuTensorMapEncodeTiled(X)", cudaErrorInvalidValue);
    return FXPR_ERR_CUDA;
  }
  // M = 128 weight columns, N = activation rows; bit 15: the 128-row operand is MN-major
  p.idesc = make_idesc(g.dtype == FXPR_BF16 ? 1 : 0, 0, MP, 128) | (p.b_kmajor ? 0u : (1u << 15));
  auto k = gemm_tc_skinny_kernel<T, MP, CLUSTER, PER_SM, WALK>;
  static bool attr_done_dev[64] = {};            // function attributes are per device
  int dev_id = 0;
  cudaGetDevice(&dev_id);
  bool& attr_done = attr_done_dev[dev_id & 63];
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) { set_last_error("gemm_tc_skinny smem attribute", e); return FXPR_ERR_CUDA; }
    attr_done = true;
  }
  const dim3 grid = CLUSTER ? dim3((unsigned)p.split_k, (unsigned)p.tiles_n, 1) : dim3((unsigned)(WALK ? walkers : p.tiles_n * p.split_k));
  cudaError_t e = launch_pdl(k, grid, dim3(kSkWarps * 32), kSmem, s, CLUSTER ? (unsigned)p.split_k : 1u, mw, mx, p, 0);
  if (e != cudaSuccess) { set_last_error("gemm_tc_skinny launch", e); return FXPR_ERR_CUDA; }
  return check_launch("gemm_tc_skinny");
}

template <typename T, int MP>
static int route_skinny(const GemmArgs& g, const CUtensorMap& mw, TcParams& p, int sms, cudaStream_t s) {
  p.tiles_m = 1;
  p.tiles_n = (p.N + 127) / 128;
  const bool cluster = gemm_tc_skinny_cluster(g, p.split_k);
  // A grid that does not fill the SMs once gives a CTA the whole SM's memory as its ring; more CTAs share an
  // SM, so that the column tiles of large weights all stream at once (64 x 28672 x 4096, 224 tiles: 46.5 us
  // with one CTA and tile after tile per SM, 38.8 with two).  64 x 4096 x 4096 on 128 CTAs: 11.3 us with the
  // whole ring, 12.1 with half of it; 64 x 6144 x 4096 13.7 / 15.9.  With 16 rows half of it holds as many
  // weights as are needed in flight: 16 x 4096 x 4096 10.5 / 9.9, 16 x 4096 x 14336 23.9 / 21.8.  Not so where the rows of
  // the weights start inside a 32-byte sector: every row of a box then touches a sector more at either end, and
  // latency with it (11 x 11928 x 11888 54.6 / 63.8, 5 x 7080 x 18976 49.9 / 58.7, 12 x 8632 x 6384 28.3 / 35.5; rows of 32 bytes
  // and more: 5 x 12576 x 3696 19.1 / 18.3; short ranks, which the half ring all but holds: 11 x 5312 x 920 6.5 / 6.3).  Whole-SM clusters of eight do not all fit from fifteen on (2 x 2016 x 8920,
  // sixteen of them: 17.7 / 11.1).
  // More tiles of 64 rows than two CTAs an SM: a CTA walks from tile to tile, so that its set-up is paid once and the next
  // tile's weights come in under the outputs.  One walker an SM, with seven stages, unless K is short (a CTA per
  // tile / two walkers / one, us): 64 x 128256 x 4096 168 / 168 / 165, 64 x 40008 x 4096 73.1 / 72.1 / 67.2, 64 x 50304 x 4096 73.5 /
  // 75.5 / 68.4, 64 x 152064 x 3584 180.9 / 180.3 / 177.7; 64 x 60000 x 2048 46.6 / 44.6 / 49.2, 64 x 102400 x 2048 74.1 / 69.2 / 72.8.
  // With fewer rows a CTA per tile stays (32 x 128256 x 4096 157.0, one persistent CTA an SM 162.5).
  const int64_t ctas = (int64_t)p.tiles_n * p.split_k;
  bool whole = ctas <= sms;
  if constexpr (MP == 16) {
    const int64_t row_bytes = 2 * (p.b_kmajor ? g.b_sn : g.b_sk);
    whole = whole && p.K >= 1024 * (int64_t)p.split_k && ((row_bytes | (int64_t)(uintptr_t)g.b) & 31) != 0 && (p.split_k <= 4 || p.tiles_n <= sms * 14 / 148);
  }
  if constexpr (MP == 64) {
    if (ctas > 2 * sms && p.split_k == 1) {
      if (p.K >= 3072) return launch_skinny<T, MP, false, 1, true>(g, mw, p, s, sms);
      return launch_skinny<T, MP, false, 2, true>(g, mw, p, s, 2 * sms);
    }
  }
  if (whole)
    return cluster ? launch_skinny<T, MP, true, 1>(g, mw, p, s) : launch_skinny<T, MP, false, 1>(g, mw, p, s);
  return cluster ? launch_skinny<T, MP, true, 2>(g, mw, p, s) : launch_skinny<T, MP, false, 2>(g, mw, p, s);
}

template <typename T>
static int route_rows(const GemmArgs& g, const CUtensorMap& mw, TcParams& p, int sms, cudaStream_t s) {
  // the smallest tile that holds the rows: padded rows would be converted and parked like live ones
  if (p.M <= 16) return route_skinny<T, 16>(g, mw, p, sms, s);
  if (p.M <= 32) return route_skinny<T, 32>(g, mw, p, sms, s);
  return route_skinny<T, 64>(g, mw, p, sms, s);
}

// mw: the weight tensor map of gemm_tc() (64-row boxes in either layout).
int gemm_tc_skinny(const GemmArgs& g, TcParams& p, const CUtensorMap& mw, cudaStream_t s) {
  const int sms = tc_device_sms();
  if (sms < 0) return FXPR_ERR_ARCH;
  if (g.dtype == FXPR_BF16) return route_rows<__nv_bfloat16>(g, mw, p, sms, s);
  return route_rows<__half>(g, mw, p, sms, s);
}

}  // namespace fxpr
