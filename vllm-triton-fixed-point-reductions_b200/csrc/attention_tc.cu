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
// pair, so a K/V tile is fetched once for the whole group.  Roles, 24 warps:
//   producers   two warps for V, four for K: a box per page piece (16 or 64 slots) and whole head, 128-byte
//               swizzle (attn_kv_map); Q by one box per 64 dims.  The first V producer also makes the item list
//   issuers     one warp for S = Q.K^T (128 keys a product in pass A, 64 in pass B), one for P.V (a fresh
//               accumulator per tile); P is the tensor-memory operand, written over the scores it came from
//   softmax     two groups of four warps, a thread is one row.  Pass A: row maxima straight from tensor memory
//               (a row lives in one lane: no shuffles).  Pass B: a group takes every other tile: weights, integer
//               denominator, P
//   conversion  eight warps: P.V partials to Q-format on the FP32 and integer pipes (packed add of
//               1.5 * 2^(23-f), raw bits summed in 32-bit registers, magnitude screen, exact fix-up
//               from tensor memory) while the other roles work on the next tiles.
// Bound: no unit's rate but instructions in flight.  A tile takes an SM about 2000 clocks; its tensor work is 900 (a
// 128 x 64 x 16 product from shared memory takes 48 clocks and not 32: 6 KB of operands at 128 bytes a clock), its
// exponentials 512 on the special-function unit, its copies about 1200 at the rate L2 gives all SMs at once.  The
// schedulers issue 53 % of the time with six warps each, an instruction of a warp at work takes 6 clocks, and the
// softmax warps wait a third of the time for scores, the conversion warps for P.V.
// 16 prompts of 128 to 4096 tokens, 32/8 heads, a call among others, in turn with a kernel with P through shared memory,
// one issuer for both products, every role decoding every item, and exact divisions per output: 1414 -> 1181 us.
// With head size 64 882 us, where the mma.sync kernel takes 3114.
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
static constexpr int kTcOpN = 2 * kTcTileN;    // keys per K stage; pass A scores them in one product, pass B in two
static constexpr int kTcRows = 128;            // query rows per CTA = tensor-memory lanes
static constexpr int kTcSoftWarps = 8;         // two groups of four warps, a group takes every other tile: thread = one row
static constexpr int kTcConvWarps = 8;         // conversion: thread = one row and half of the output columns
// warps 0, 1: score and P.V issuers; 2, 3: V producers (the first also makes the item list); 4-7: K producers
static constexpr int kTcVProducers = 2, kTcKProducers = 4;
static constexpr int kTcFirstV = 2, kTcFirstK = kTcFirstV + kTcVProducers;
static constexpr int kTcFirstSoft = kTcFirstK + kTcKProducers;
static constexpr int kTcFirstConv = kTcFirstSoft + kTcSoftWarps;
static constexpr int kTcThreads = (kTcFirstConv + kTcConvWarps) * 32;
static constexpr int kTcItems = 4;             // ring of work items in shared memory
static constexpr int kTcListGroup = 8;         // requests whose row blocks are dealt out together
static constexpr int kTcItemReaders = kTcThreads / 32;
// Registers: 24 warps, six per scheduler, launch with 80 a thread.  Conversion keeps 64 sums and two loads of
// 16 in registers; the first eight warps give up what that takes.  Per scheduler: 2 x 48 + 2 x 88 + 2 x 104 = 6 x 80.
static constexpr int kTcRegsLaunch = 80, kTcRegsFront = 48, kTcRegsSoft = 88, kTcRegsConv = 104;
static_assert(kTcFirstSoft / 4 * kTcRegsFront + kTcSoftWarps / 4 * kTcRegsSoft + kTcConvWarps / 4 * kTcRegsConv <=
              kTcThreads / 128 * kTcRegsLaunch, "setmaxnreg draws on the registers of the launch");
static_assert(kTcFirstSoft % 4 == 0, "register shares go by groups of four warps");
// (setmaxnreg.dec to more, or .inc to fewer, registers than a warp has is an illegal instruction)
static_assert(kTcRegsFront <= kTcRegsLaunch && kTcRegsSoft >= kTcRegsLaunch && kTcRegsConv >= kTcRegsLaunch,
              "the first eight warps give, the others take");

struct TcAttnShape {
  int rows_per_token;      // GQA group size
  int row_shift;           // log2 of it
  int tokens_per_block;    // 128 / rows_per_token
  int num_q_blocks;
  int page_size;
  int group_shift;         // log2 of the keys per TMA box: 6 when pages are multiples of 64 tokens, else 4
  int page_shift;          // log2 of the page size, -1 where it is no power of two
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

// D (tensor memory) = A (tensor memory, packed 16-bit pairs) . B (shared memory)
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// Bounded wait of a whole warp.  Eight to twelve warps of this kernel wait at any time, so a probe is few
// instructions and little code: it parks for up to a microsecond (an arrival of its own CTA wakes it), probes are
// counted instead of clocks, and the abort flag is looked at every 64.
static constexpr int kParkProbes = 1 << 22;
__device__ __forceinline__ bool mbar_park(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ bool park_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int probes = 0; probes < kParkProbes; ++probes) {
    if (mbar_park(bar, parity)) return true;
    if ((probes & 63) == 63 && __any_sync(0xffffffffu, *abort_flag)) return false;
  }
  *abort_flag = 1;
  return false;
}

template <int HD> struct TcAttnSmem {
  static constexpr int kQBytes = kTcRows * HD * 2;             // slabs of 64 dims: 128 rows x 128 B
  static constexpr int kKBytes = kTcOpN * HD * 2;              // [8-key group][64-dim half][8 keys][128 B]
  static constexpr int kVBytes = kTcTileN * HD * 2;
  static constexpr int kKStages = 3, kVStages = 3;
  static constexpr int kQOff = 0, kKOff = 2 * kQBytes, kVOff = kKOff + kKStages * kKBytes;
  static constexpr int kItemOff = kVOff + kVStages * kVBytes;                    // [kTcItems][8] ints
  static constexpr int kMaxOff = kItemOff + kTcItems * 32;                       // [item parity][group][128] floats
  static constexpr int kDenOff = kMaxOff + 2 * 2 * kTcRows * 4;      // [item parity][group][128] int64
  static constexpr int kGoOff = kDenOff + 2 * 2 * kTcRows * 8;       // [group][item parity] ints
  static constexpr int kBarOff = kGoOff + 64;
  static constexpr int kBars = 4 + 2 * kKStages + 2 * kVStages + 2 * kTcItems + 2 + 4 + 2 + 4 + 4 + 4 + 1 + 4;
  static constexpr int kTotal = kBarOff + kBars * 8 + 16 + 1024;
  static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

// PLAIN: scores are the scaled products (no soft-cap, no ALiBi) and the scale is positive, so a row's maximum
// is the maximum of the raw products, scaled.
template <typename T, int HD, bool PLAIN>
__global__ void __launch_bounds__(kTcThreads, 1)
attn_tc_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const AttnParams p, const TcAttnShape sh,
                       int32_t* status, const int zero /* always 0: keeps the side arrays in local memory */) {
  static_assert(HD == 64 || HD == 128, "head size 64 or 128");
  using Sm = TcAttnSmem<HD>;
  constexpr int KST = Sm::kKStages, VST = Sm::kVStages;
  constexpr int kHalfCols = HD / 2;                        // P.V columns per conversion thread
  // Tensor-memory columns: scores in four buffers of 64 keys (the maximum pass fills two neighbours, "half" 0 or
  // 1; in the weight pass P of a tile replaces the first 32 columns of its scores), then two P.V accumulators
  constexpr uint32_t kColS = 0, kColPV = 256;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t q_s0 = smem_base + Sm::kQOff, k_s0 = smem_base + Sm::kKOff, v_s0 = smem_base + Sm::kVOff;
  const uint32_t qfull0 = smem_base + Sm::kBarOff, qfree0 = qfull0 + 16;          // [2] each
  const uint32_t kfull0 = qfree0 + 16, kempty0 = kfull0 + 8 * KST;
  const uint32_t vfull0 = kempty0 + 8 * KST, vempty0 = vfull0 + 8 * VST;
  const uint32_t ifull0 = vempty0 + 8 * VST, iempty0 = ifull0 + 8 * kTcItems;
  const uint32_t sfa0 = iempty0 + 8 * kTcItems;            // [half]: scores of the maximum pass
  const uint32_t sfb0 = sfa0 + 16;                         // [buffer]: scores of the weight pass
  const uint32_t afree0 = sfb0 + 32;                       // [half]: maximum pass has read the scores
  const uint32_t pready0 = afree0 + 16;                    // [buffer]: P is written
  const uint32_t pdone0 = pready0 + 32;                    // [buffer]: P.V has read it
  const uint32_t pvfull0 = pdone0 + 32, pvfree0 = pvfull0 + 16;                   // [accumulator]
  const uint32_t soft_bar = pvfree0 + 16, denfull0 = soft_bar + 8, denfree0 = denfull0 + 16;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem_gen + Sm::kBarOff + Sm::kBars * 8);
  volatile int* abort_flag = (volatile int*)(smem_gen + Sm::kBarOff + Sm::kBars * 8 + 8);
  float* rmax_s = (float*)(smem_gen + Sm::kMaxOff);
  long long* den_s = (long long*)(smem_gen + Sm::kDenOff);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hkv = p.num_kv_heads;
  const int G = sh.rows_per_token;

  if (threadIdx.x == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(qfull0 + 8u * i, 1); mbar_init(qfree0 + 8u * i, 1); }
    for (int i = 0; i < KST; ++i) { mbar_init(kfull0 + 8u * i, kTcKProducers); mbar_init(kempty0 + 8u * i, 1); }
    for (int i = 0; i < VST; ++i) { mbar_init(vfull0 + 8u * i, kTcVProducers); mbar_init(vempty0 + 8u * i, 1); }
    for (int i = 0; i < kTcItems; ++i) { mbar_init(ifull0 + 8u * i, 1); mbar_init(iempty0 + 8u * i, kTcItemReaders); }
    for (int i = 0; i < 2; ++i) { mbar_init(sfa0 + 8u * i, 1); mbar_init(afree0 + 8u * i, 4); }
    for (int i = 0; i < 4; ++i) { mbar_init(sfb0 + 8u * i, 1); mbar_init(pready0 + 8u * i, 4); mbar_init(pdone0 + 8u * i, 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(pvfull0 + 8u * i, 1); mbar_init(pvfree0 + 8u * i, kTcConvWarps); }
    mbar_init(soft_bar, kTcSoftWarps);
    for (int i = 0; i < 2; ++i) { mbar_init(denfull0 + 8u * i, kTcSoftWarps); mbar_init(denfree0 + 8u * i, kTcConvWarps); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    tmem_alloc(smem_u32((const void*)tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // ---- work items ---------------------------------------------------------------------
  // Persistent CTAs over the live (row block, request, KV head) of eight requests at a time, the last row blocks
  // (most keys) of all of them first, dealt out there and back again.  That gives every CTA about the same work:
  // request by request, a request's last, short items and the next one's long ones fall into one round.  All requests
  // together balance best but spread the CTAs over more keys than L2 holds (16 prompts of 128 to 4096 tokens:
  // requests by 32 1071 us, 8 1046, 1 1062; a static list with the dead entries in it left the busiest SM 10 % over the
  // mean).
  // The first V producer makes the list and leaves it in a ring in shared memory; every
  // role reads them there in order.  (Decoded by each role for itself, two dependent global loads and a
  // division per entry, dead ones included, took the softmax warps some 400 of 4860 clocks per two tiles.)
  // Ring positions and barrier phases run on from one item to the next, so the producers fetch the next item's
  // Q and first keys, and its scores are made, while the current one is still finished.
  struct Item { int req, kvh, q_start, q_len, tok0, seq_len, t0, t1; };
  int ipos = 0; uint32_t iphase = 0;                       // this role's position in the ring
  auto read_item = [&](Item& I) -> bool {                  // ifull[ipos] has been waited for; false: no more items
    const int4* src = reinterpret_cast<const int4*>(smem_gen + Sm::kItemOff + ipos * 32);
    const int4 a = src[0], b = src[1];
    I.req = a.x; I.kvh = a.y; I.q_start = a.z; I.q_len = a.w;
    I.tok0 = b.x; I.seq_len = b.y; I.t0 = b.z; I.t1 = b.w;
    __syncwarp();
    mbar_arrive_if(iempty0 + 8u * ipos, lane == 0);
    if (++ipos == kTcItems) { ipos = 0; iphase ^= 1; }
    return __all_sync(0xffffffffu, I.req >= 0);
  };
  auto next_item = [&](Item& I) -> bool {
    return park_wait(ifull0 + 8u * ipos, iphase, abort_flag) && read_item(I);
  };
  // Softmax and conversion warps work in groups of four, one on each scheduler.  One warp of a group probes the
  // barrier, the others sleep in a hardware barrier: with all 20 probing, half of the issued instructions were
  // probes.  After a wait that gave up a group goes on through its item, on whatever it reads (later waits then
  // fail at once), so that its four warps always meet the same barriers; it leaves, all four, at the next item.
  const int grp = (warp - kTcFirstSoft) >> 2;              // 0, 1 softmax, 2, 3 conversion
  const bool prober = (warp & 3) == grp;
  auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); };
  auto group_wait = [&](uint32_t bar, uint32_t parity) {
    if (prober) (void)park_wait(bar, parity, abort_flag);
    group_sync();
  };
  volatile int* go = (volatile int*)(smem_gen + Sm::kGoOff) + 2 * grp;   // [item parity]: is there an item
  auto group_next = [&](Item& I, int k) -> bool {
    if (prober) {
      const bool ok = park_wait(ifull0 + 8u * ipos, iphase, abort_flag);
      if (lane == 0) go[k & 1] = ok;
    }
    group_sync();
    return go[k & 1] != 0 && read_item(I);
  };

  if (warp < kTcFirstSoft) {
    regs_dec<kTcRegsFront>();
    if (warp == 0) {
      // ------------------------------ score issuer ------------------------------------
      // Item by item the maximum pass, 128 keys a product into alternating halves of the score buffers, then the
      // weight pass, 64 keys into the next of the four buffers: a softmax group then finds its next tile's scores
      // in one buffer while P.V still reads the other (with products of 128 keys here too, a group waited 1250
      // clocks per product for P.V and the next scores, next to 3700 at work).  Scores and P.V have a warp each:
      // in one warp, in turn, the 12 MMAs, 5 commits and 5 waits of a tile were a chain of 1700 clocks next to 770
      // of tensor work.  Everything here is warp-uniform also for the compiler (votes, values read by shuffle).
      const uint32_t e = elect_one();
      int half = 0;                                        // of the next maximum-pass product
      int kst = 0; uint32_t kph = 0;
      int qb = 0; uint32_t qph = 0;
      uint32_t a_pend = 0, a_ph = 0, p_pend = 0, p_ph = 0; // what a half, a buffer is still waited for; phases
      const uint64_t qd0 = make_smem_desc(q_s0, 16, 1024), kd0 = make_smem_desc(k_s0, 16, HD * 16);
      auto half_free = [&](int h) -> bool {                // the maximum pass has read it
        if (!(a_pend >> h & 1)) return true;
        a_pend ^= 1u << h;
        const uint32_t ph = a_ph >> h & 1;
        a_ph ^= 1u << h;
        return park_wait(afree0 + 8u * h, ph, abort_flag);
      };
      auto buffer_free = [&](int b) -> bool {              // P.V has read it
        if (!(p_pend >> b & 1)) return true;
        p_pend ^= 1u << b;
        const uint32_t ph = p_ph >> b & 1;
        p_ph ^= 1u << b;
        return park_wait(pdone0 + 8u * b, ph, abort_flag);
      };
      // S = Q . K^T: both operands K-major (head dim contiguous); Q in slabs of 64 dims, K with the 64-dim
      // halves of every 8-key group side by side
      auto issue = [&](int column, uint64_t qd, uint64_t kd, uint32_t idesc) {
        const uint32_t d = tmem_base + kColS + (uint32_t)column;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t ao = (uint64_t)((kk >> 2) * (kTcRows * 128) + (kk & 3) * 32) >> 4;
          const uint64_t bo = (uint64_t)((kk >> 2) * 1024 + (kk & 3) * 32) >> 4;
          umma_f16(d, qd + ao, kd + bo, idesc, kk ? 1u : 0u, e);
        }
      };
      auto next_stage = [&]() {
        umma_commit(kempty0 + 8u * kst, e);
        if (++kst == KST) { kst = 0; kph ^= 1; }
      };
      Item I;
      while (next_item(I)) {
        const int tiles = __shfl_sync(0xffffffffu, I.t1 - I.t0, 0);
        const uint64_t qd = qd0 + (uint64_t)(qb * (Sm::kQBytes >> 4));
        if (!park_wait(qfull0 + 8u * qb, qph, abort_flag)) goto scores_done;
#pragma unroll 1
        for (int j = 0; j < tiles; j += 2) {
          if (!half_free(half) || !buffer_free(2 * half) || !buffer_free(2 * half + 1)) goto scores_done;
          if (!park_wait(kfull0 + 8u * kst, kph, abort_flag)) goto scores_done;
          tc_fence_after();
          issue(half * 128, qd, kd0 + (uint64_t)(kst * (Sm::kKBytes >> 4)), sh.idesc_s2);
          umma_commit(sfa0 + 8u * half, e);
          a_pend |= 1u << half;
          next_stage();
          half ^= 1;
        }
        int b = 2 * half;
#pragma unroll 1
        for (int j = 0; j < tiles; ++j) {
          if (!half_free(b >> 1) || !buffer_free(b)) goto scores_done;
          if (!(j & 1) && !park_wait(kfull0 + 8u * kst, kph, abort_flag)) goto scores_done;
          tc_fence_after();
          issue(b * 64, qd, kd0 + (uint64_t)(kst * (Sm::kKBytes >> 4) + (j & 1) * (kTcTileN * HD * 2 >> 4)), sh.idesc_s);
          umma_commit(sfb0 + 8u * b, e);
          p_pend |= 1u << b;
          if ((j & 1) || j + 1 == tiles) next_stage();
          half = (b >> 1) ^ 1;                             // not the half of the last tile
          b = (b + 1) & 3;
        }
        umma_commit(qfree0 + 8u * qb, e);
        qb ^= 1; if (qb == 0) qph ^= 1;
      }
    scores_done:;
    } else if (warp == 1) {
      // ------------------------------ P.V issuer --------------------------------------
      const uint32_t e = elect_one();
      int half = 0, acc = 0; uint32_t r_ph = 0, acc_ph = 1;   // half: of the next maximum-pass product
      int vst = 0; uint32_t vph = 0;
      const uint64_t vd0 = make_smem_desc(v_s0, 1024, HD * 16);
      Item I;
      while (next_item(I)) {
        const int tiles = __shfl_sync(0xffffffffu, I.t1 - I.t0, 0);
        const int keys = __shfl_sync(0xffffffffu, I.seq_len - I.t0 * kTcTileN, 0);
        half ^= ((tiles + 1) >> 1) & 1;                    // the maximum pass's products
        int b = 2 * half;
#pragma unroll 1
        for (int j = 0; j < tiles; ++j) {
          if (!park_wait(vfull0 + 8u * vst, vph, abort_flag)) goto pv_done;
          if (!park_wait(pvfree0 + 8u * acc, acc_ph, abort_flag)) goto pv_done;
          if (!park_wait(pready0 + 8u * b, r_ph >> b & 1, abort_flag)) goto pv_done;
          tc_fence_after();
          // Keys at or past the end of the sequence: their V rows were not copied (or come from slots
          // nobody wrote) and 0 * NaN would poison the accumulator, so the rows are cleared.  Only the
          // last tile of a sequence has any.
          const int n0 = keys - j * kTcTileN;
          if (n0 < kTcTileN) {
            const uint32_t vs = v_s0 + vst * Sm::kVBytes;
#pragma unroll 1
            for (int idx = lane; idx < (kTcTileN - n0) * (HD / 8); idx += 32) {
              const int rr = n0 + idx / (HD / 8), cc = idx % (HD / 8);
              const uint32_t addr = vs + (uint32_t)((rr >> 3) * (HD * 16) + (cc >> 3) * 1024 + (rr & 7) * 128 + (cc & 7) * 16);
              asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0) : "memory");
            }
            fence_proxy_async_smem();
            __syncwarp();
          }
          // PV_j = P_j . V_j: P from tensor memory, V MN-major (head dim contiguous)
          const uint32_t d = tmem_base + kColPV + (uint32_t)(acc * HD), pa = tmem_base + kColS + (uint32_t)(b * 64);
          const uint64_t vd = vd0 + (uint64_t)(vst * (Sm::kVBytes >> 4));
#pragma unroll
          for (int kk = 0; kk < kTcTileN / 16; ++kk)
            umma_f16_ts(d, pa + (uint32_t)(kk * 8), vd + (uint64_t)(kk * (HD * 32 >> 4)), sh.idesc_pv, kk ? 1u : 0u, e);
          umma_commit(pvfull0 + 8u * acc, e);
          umma_commit(vempty0 + 8u * vst, e);
          umma_commit(pdone0 + 8u * b, e);
          r_ph ^= 1u << b;
          half = (b >> 1) ^ 1;
          b = (b + 1) & 3;
          acc ^= 1; if (acc == 0) acc_ph ^= 1;
          if (++vst == VST) { vst = 0; vph ^= 1; }
        }
      }
    pv_done:;
    } else {
      // ------------------------------ K / V producers (TMA) ---------------------------
      // A box is a 16-token page piece, or 64 keys when pages are multiples of 64 tokens, with all head
      // dims.  The 8-row swizzle atoms of one 64-dim half lie HD * 16 bytes apart whatever the page size, which
      // is all the MMA descriptors need.  Nothing is copied, and the block table is not read, past the end of
      // the sequence or of the item's tiles; V rows there are cleared by the P.V issuer, scores there belong
      // to no tile or are masked.
      const uint32_t e = elect_one();
      const bool is_v = warp < kTcFirstK, lists = warp == kTcFirstV;
      const int me = is_v ? warp - kTcFirstV : warp - kTcFirstK;
      const CUtensorMap* map = is_v ? &map_v : &map_k;
      const uint32_t ring0 = is_v ? v_s0 : k_s0, full0 = is_v ? vfull0 : kfull0, empty0 = is_v ? vempty0 : kempty0;
      const int step = is_v ? kTcTileN : kTcOpN, stages = is_v ? VST : KST, passes = is_v ? 1 : 2;
      const int stage_bytes = is_v ? Sm::kVBytes : Sm::kKBytes;
      int stage = 0; uint32_t phase = 1;
      int qb = 0; uint32_t q_phase = 1;                    // qfree: the first waits pass
      const int page_shift = sh.page_shift;
      // ---- item list (first V producer): kTcListGroup requests at a time, one a lane
      int l_start = 0, l_q = 0, l_seq = 0, l_blocks = 0;     // this lane's request
      int group = -kTcListGroup, level = -1;                 // first of these requests; row block, from the last down
      uint32_t round = 0, base = 0, target = blockIdx.x;     // live items before this level; this CTA's next one
      bool ended = false;                                    // the end mark (req -1) is written
      int wpos = 0, ahead = 0; uint32_t wphase = 1;          // ahead: items written and not yet read by this warp
      auto fill_list = [&]() -> bool {
        while (!ended && ahead < kTcItems) {
          // wait only for a slot that this warp itself has to read next
          if (ahead == 0) {
            if (!park_wait(iempty0 + 8u * wpos, wphase, abort_flag)) return false;
          } else if (!__all_sync(0xffffffffu, mbar_test_wait(iempty0 + 8u * wpos, wphase))) {
            return true;
          }
          uint32_t live = 0;
          while (!ended) {
            if (level < 0) {
              group += kTcListGroup;
              if (group >= p.num_reqs) { ended = true; break; }
              const int req = group + lane;
              l_q = 0;
              if (lane < kTcListGroup && req < p.num_reqs) { l_start = p.qsl[req]; l_q = p.qsl[req + 1] - l_start; l_seq = p.seq_lens[req]; }
              l_blocks = min(sh.num_q_blocks, (l_q + sh.tokens_per_block - 1) / sh.tokens_per_block);
              level = __reduce_max_sync(0xffffffffu, l_blocks) - 1;
              continue;
            }
            live = __ballot_sync(0xffffffffu, l_blocks > level);
            const uint32_t count = (uint32_t)(__popc(live) * hkv);
            if (target < base + count) break;
            base += count;
            --level;
          }
          int who = 0, kvh = 0;
          if (!ended) {
            const int off = (int)(target - base), nth = off / hkv;
            kvh = off - nth * hkv;
            who = __ffs(__ballot_sync(0xffffffffu, (live >> lane & 1) && __popc(live & ((1u << lane) - 1)) == nth)) - 1;
            ++round;
            target = round * gridDim.x + (round & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
          }
          if (lane == who) {
            const int tok0 = level * sh.tokens_per_block;
            const int ctx = l_seq - l_q, tok_end = min(l_q, tok0 + sh.tokens_per_block);
            const int hi_key = p.causal ? min(l_seq, ctx + tok_end) : l_seq;
            const int lo_key = p.window > 0 ? max(0, ctx + tok0 - p.window + 1) : 0;
            const int t0 = lo_key / kTcTileN, t1 = max(t0, (hi_key + kTcTileN - 1) / kTcTileN);
            int4* dst = reinterpret_cast<int4*>(smem_gen + Sm::kItemOff + wpos * 32);
            dst[0] = make_int4(ended ? -1 : group + lane, kvh, l_start, l_q);
            dst[1] = make_int4(tok0, l_seq, t0, t1);
            mbar_arrive(ifull0 + 8u * wpos);
          }
          __syncwarp();
          ++ahead;
          if (++wpos == kTcItems) { wpos = 0; wphase ^= 1; }
        }
        return true;
      };
      Item I;
      while ((!lists || fill_list()) && next_item(I)) {
        --ahead;
        const int32_t* bt = p.block_table + (int64_t)I.req * p.bt_stride;
        const int end = min(I.seq_len, I.t1 * kTcTileN);   // keys to copy
        // Q rows: box {64 dims, G heads, 128 / G tokens} -> row = token * G + head.  Tokens past this
        // request's (they belong to the next one, or lie beyond the tensor: zeros) are rows whose every
        // key is masked and that are never stored.
        if (!is_v && me == 0) {
          if (!park_wait(qfree0 + 8u * qb, q_phase, abort_flag)) break;
          const uint32_t fb = qfull0 + 8u * qb;
          mbar_expect_tx(fb, Sm::kQBytes, e);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            tma_load_3d(q_s0 + qb * Sm::kQBytes + c * (kTcRows * 128), &map_q, fb, c * 64, I.kvh * G, I.q_start + I.tok0, e);
          qb ^= 1; if (qb == 0) q_phase ^= 1;
        }
        // `passes` walks over the item's keys, `step` keys a stage; GS = log2 of the keys per box, `mine` boxes of
        // a stage from `first` on are this warp's.  Block-table entries are read 32 at a time (lane L: the 16-key
        // group L of a 512-key block), one block ahead of their use, and handed round by shuffle with the row in
        // the page.
        auto walk = [&](auto gs_c) -> bool {
          constexpr int GS = decltype(gs_c)::value;
          constexpr int kBoxBytes = (HD * 2) << GS;
          constexpr int kMine = GS == 4 ? 2 : 1;             // 8 boxes of K over 4 warps, 4 of V over 2; or 2 and 1
          static_assert((kTcOpN >> 4) / kTcKProducers == 2 && (kTcTileN >> 4) / kTcVProducers == 2, "boxes per warp");
          const int first = me * kMine, start = I.t0 * kTcTileN, stop = I.t1 * kTcTileN;
#pragma unroll 1
          for (int pass = 0; pass < passes; ++pass) {
            int cur = 0, cur_row = 0, nxt, nxt_row;
#pragma unroll 1
            for (int nb = start - 512; nb < stop; nb += 512) {
              {
                const int n = nb + 512 + lane * 16, pg = page_shift >= 0 ? n >> page_shift : n / sh.page_size;
                nxt = n < end ? bt[pg] : 0;
                nxt_row = (n - pg * sh.page_size) >> 3;
              }
              const int top = nb < start ? 0 : min(512, stop - nb);
#pragma unroll 1
              for (int off = 0; off < top; off += step) {
                int blk[kMine], row8[kMine];
                // of its boxes, those that start before the end
                const int left = (end - (nb + off) + (1 << GS) - 1) >> GS;
                const int boxes = max(0, min(kMine, min(step >> GS, left) - first));
#pragma unroll
                for (int i = 0; i < kMine; ++i) {
                  const int from = ((off >> 4) + ((first + i) << (GS - 4))) & 31;
                  blk[i] = __shfl_sync(0xffffffffu, cur, from);
                  row8[i] = __shfl_sync(0xffffffffu, cur_row, from);
                }
                const uint32_t fb = full0 + 8u * stage;
                const uint32_t dst = ring0 + (uint32_t)(stage * stage_bytes + first * kBoxBytes);
                if (!park_wait(empty0 + 8u * stage, phase, abort_flag)) return false;
                mbar_expect_tx(fb, (uint32_t)(boxes * kBoxBytes), e);
#pragma unroll
                for (int i = 0; i < kMine; ++i)
                  if (i < boxes)
                    tma_load_5d(dst + (uint32_t)(i * kBoxBytes), map, fb, 0, 0, I.kvh * sh.head_chunks, row8[i], blk[i], e);
                if (++stage == stages) { stage = 0; phase ^= 1; }
              }
              cur = nxt; cur_row = nxt_row;
            }
          }
          return true;
        };
        const bool fetched = sh.group_shift == 4 ? walk(std::integral_constant<int, 4>{}) : walk(std::integral_constant<int, 6>{});
        if (!fetched) break;
      }
    }
  } else if (warp < kTcFirstConv) {
    // ------------------------------ softmax warps -------------------------------------
    regs_inc<kTcRegsSoft>();
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                     // tensor-memory lane = query row
    const uint32_t s_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + kColS;
    const float ninf = -__int_as_float(0x7f800000);
    const uint64_t zero2 = pack2((uint32_t)zero, (uint32_t)zero);
    const uint64_t ss2 = pack2(__float_as_uint(p.ss_log2), __float_as_uint(p.ss_log2));
    const uint32_t mbits = q_magic_bits(p.inv_scale);
    const uint64_t magic2 = pack2(mbits, mbits);
    // Group 0 takes the maximum-pass products in half 0 and, in the weight pass, the buffers 0 and 2, that is every
    // other tile, group 1 the others.
    const uint32_t s_half = s_addr + (uint32_t)(grp * 128);
    uint32_t soft_phase = 0, a_phase = 0, b_phase = 0;       // b_phase: a bit for either buffer
    int half = 0;                                            // of the next maximum-pass product
    int k = -1;                                              // items so far
    Item I;
    while (group_next(I, ++k)) {
      const int n_tiles = I.t1 - I.t0, n_ops = (n_tiles + 1) >> 1;
      const int tok = I.tok0 + (row >> sh.row_shift);
      const bool valid = tok < I.q_len;
      const int pos = I.seq_len - I.q_len + tok;
      const int kend = valid ? (p.causal ? min(I.seq_len, pos + 1) : I.seq_len) : 0;
      const int kbeg = valid ? (p.window > 0 ? max(0, pos - p.window + 1) : 0) : 0;
      const float slope = (!PLAIN && p.alibi && valid) ? p.alibi[I.kvh * G + (row & (G - 1))] : 0.0f;
      // one score in log2 space with soft-cap and ALiBi (attention.py:103-121, 249-254)
      auto score = [&](uint32_t v, int n) -> float {
        float x = __fmul_rn(__uint_as_float(v), p.ss_log2);
        if (p.cap_log2 > 0.0f) x = __fmul_rn(p.cap_log2, tanhf(__fdiv_rn(x, p.cap_log2)));
        if (p.alibi) x = __fadd_rn(x, __fmul_rn(slope, __fsub_rn((float)n, (float)pos)));
        return x;
      };

      // =============================== pass A: row maxima ===============================
      // 128 keys per step, all of them in one thread.  Scaling by a positive constant is monotonic after
      // rounding too, so the maximum is taken over the raw products and scaled once.
      float rmax = ninf;
#pragma unroll 1
      for (int i = half ^ grp; i < n_ops; i += 2) {
        group_wait(sfa0 + 8u * grp, a_phase);
        a_phase ^= 1;
        tc_fence_after();
        float m = ninf;
        const int first = I.t0 * kTcTileN + i * kTcOpN;
        if (PLAIN && __all_sync(0xffffffffu, first >= kbeg && first + kTcOpN <= kend)) {
          // no row of the warp is masked here
          float m1 = ninf;                                   // two chains
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t v[32];
            tmem_ld32(s_half + (uint32_t)(c * 32), v);
            tmem_wait_ld_regs(v);
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
              m = max3(m, __uint_as_float(v[x]), __uint_as_float(v[x + 1]));
              m1 = max3(m1, __uint_as_float(v[x + 2]), __uint_as_float(v[x + 3]));
            }
          }
          m = fmaxf(m, m1);
        } else {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t v[32];
          tmem_ld32(s_half + (uint32_t)(c * 32), v);
          tmem_wait_ld_regs(v);
          const int n0 = first + c * 32;
          if (n0 < kend && n0 + 32 > kbeg) {
#pragma unroll
            for (int x = 0; x < 32; ++x)
              if (n0 + x >= kbeg && n0 + x < kend) m = fmaxf(m, PLAIN ? __uint_as_float(v[x]) : score(v[x], n0 + x));
          }
        }
        }
        // all of it has been read: hand the half back
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(afree0 + 8u * grp, lane == 0);
        rmax = fmaxf(rmax, PLAIN ? __fmul_rn(m, p.ss_log2) : m);
      }
      half ^= n_ops & 1;
      float* rmax_k = rmax_s + (k & 1) * (2 * kTcRows);
      rmax_k[grp * kTcRows + row] = rmax;
      __syncwarp();
      mbar_arrive_if(soft_bar, lane == 0);
      group_wait(soft_bar, soft_phase);
      soft_phase ^= 1;
      float gmax = fmaxf(rmax_k[row], rmax_k[kTcRows + row]);
      if (gmax == ninf) gmax = 0.0f;                         // rows without keys: exp2 gives 0, not NaN

      // =============================== pass B ===========================================
      uint32_t den32 = 0;
      const uint64_t neg_max2 = pack2(__float_as_uint(-gmax), __float_as_uint(-gmax));
      int done = 0;                                          // tiles of this group
#pragma unroll 1
      for (int j = grp; j < n_tiles; j += 2) {
        const int b = (2 * half + j) & 3;
        group_wait(sfb0 + 8u * b, b_phase >> (b >> 1) & 1);
        b_phase ^= 1u << (b >> 1);
        tc_fence_after();
        const uint32_t sb = s_addr + (uint32_t)(b * 64);
        const int first = (I.t0 + j) * kTcTileN;
        const bool masks = __any_sync(0xffffffffu, first < kbeg || first + kTcTileN > kend);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld32(sb + (uint32_t)(c * 32), v);
          tmem_wait_ld_regs(v);
          // d = score - max, rounded twice; the product is an fma with a run-time zero because the
          // assembler contracts a packed multiply and the packed add behind it into one rounding.
          // The weight of a masked key is exp2(-inf) = 0.
          const int n0 = first + c * 32;
          if (PLAIN) {
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
          if (masks) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (n0 + i < kbeg || n0 + i >= kend) v[i] = __float_as_uint(ninf);
          }
          // weights, integer denominator, P in the io dtype over the scores that were read (A operand of
          // P.V: two keys a column)
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float w0 = ex2_approx_tc(__uint_as_float(v[2 * i]));
            const float w1 = ex2_approx_tc(__uint_as_float(v[2 * i + 1]));
            uint64_t q;
            asm("add.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(pack2(__float_as_uint(w0), __float_as_uint(w1))), "l"(magic2));
            den32 = den32 + (uint32_t)q + (uint32_t)(q >> 32);
            pk[i] = pack2_tc<T>(w0, w1);
          }
          tmem_st16(sb + (uint32_t)(c * 16), pk);            // over scores that have been read
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(pready0 + 8u * b, lane == 0);
        ++done;
      }
      if (n_tiles) half = (((2 * half + n_tiles - 1) & 3) >> 1) ^ 1;   // not the half of the last tile
      // 64 weights per tile went through the packed add in this thread
      group_wait(denfree0 + 8u * (k & 1), ((k >> 1) & 1) ^ 1);
      den_s[((k & 1) * 2 + grp) * kTcRows + row] = (long long)(int32_t)(den32 - (uint32_t)kTcTileN * (uint32_t)done * mbits);
      __syncwarp();
      mbar_arrive_if(denfull0 + 8u * (k & 1), lane == 0);
    }
  } else {
    // ------------------------------ conversion warps ----------------------------------
    // Round every P.V partial to Q-format, add, and store the finished rows; the softmax warps are by
    // then in the next item's maximum pass.
    regs_inc<kTcRegsConv>();
    const int quarter = warp & 3;
    const int half = (warp - kTcFirstConv) >> 2;             // which half of the output columns
    const int row = quarter * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    const uint32_t mbits = q_magic_bits(p.inv_scale), one = (uint32_t)zero + 1u;
    const uint64_t magic2 = pack2(mbits, mbits);
    const float screen_limit = q_screen_limit(p.inv_scale);
    int jg = 0;                                              // P.V tiles converted so far (all items)
    int k = -1;                                              // items so far
    Item I;
    while (group_next(I, ++k)) {
      const int n_tiles = I.t1 - I.t0;
      uint32_t acc[kHalfCols];
#pragma unroll
      for (int i = 0; i < kHalfCols; ++i) acc[i] = 0;
      uint32_t corr_raw[kHalfCols];                          // rare path, local memory
      long long corr_q[kHalfCols];
      bool corr_used = false;
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j, ++jg) {
        const int b = jg & 1;
        group_wait(pvfull0 + 8u * b, (jg >> 1) & 1);
        tc_fence_after();
        const uint32_t taddr = tmem_base + lane_sel + kColPV + (uint32_t)(b * HD + half * kHalfCols);
        float screen = 0.0f, tail = 0.0f;
        uint32_t v[2][16];                                   // the next load is under way while one is converted
        tmem_ld16(taddr, v[0]);
#pragma unroll
        for (int c = 0; c < kHalfCols / 16; ++c) {
          uint32_t (&cur)[16] = v[c & 1];
          tmem_wait_ld_regs(cur);
          if (c + 1 < kHalfCols / 16) {
            tmem_ld16(taddr + (c + 1) * 16, v[(c + 1) & 1]);
          } else {
            // the last chunk is in registers: screen it and hand the buffer back before converting it
#pragma unroll
            for (int i = 0; i < 16; i += 2) screen = max3_abs(screen, __uint_as_float(cur[i]), __uint_as_float(cur[i + 1]));
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
            mbar_arrive_if(pvfree0 + 8u * b, lane == 0);
          }
          convert16(cur, &acc[c * 16], magic2, mbits, one, c + 1 == kHalfCols / 16 ? tail : screen);
        }
      }
      group_wait(denfull0 + 8u * (k & 1), (k >> 1) & 1);
      const long long dsum = den_s[(k & 1) * 2 * kTcRows + row] + den_s[((k & 1) * 2 + 1) * kTcRows + row];
      __syncwarp();
      mbar_arrive_if(denfree0 + 8u * (k & 1), lane == 0);
      const int tok = I.tok0 + (row >> sh.row_shift), head = I.kvh * G + (row & (G - 1));
      const bool store = tok < I.q_len && !*abort_flag;
      const float dn = fmaxf(fixed_to_float<long long>(wrap_to_bits(dsum, p.int_bits), p.inv_scale), 1.0e-6f);
      T* op = (T*)p.o + (int64_t)(I.q_start + tok) * p.o_st + (int64_t)head * p.o_sh + half * kHalfCols;
      const uint32_t bias_bits = (uint32_t)n_tiles * mbits;  // what the multiply-adds summed on top
      // acc becomes the sums as floats.  They fit 32 bits unless a partial took the fix-up: one conversion each, whatever
      // their size (16 prompts of 1024 tokens, values of zero mean / mean 0.5, us: a shortcut below 2^22 and an element loop out
      // of local memory above it 296 / 525, this 296 / 297, both in registers, which spilled, 340 / 342).  After a
      // fix-up the exact sums, as floats, are put together out of local memory, in a loop.
      if (corr_used) {
        uint32_t sums[kHalfCols];
#pragma unroll
        for (int i = 0; i < kHalfCols; ++i) sums[i + zero] = alu_add(i) ? acc[i] : acc[i] - bias_bits;
#pragma unroll 4
        for (int c = 0; c < kHalfCols; ++c) {
          const long long t = wrap_to_bits((long long)(int32_t)(sums[c + zero] - corr_raw[c + zero]) + corr_q[c + zero], p.int_bits);
          sums[c + zero] = __float_as_uint(__ll2float_rn(t));
        }
#pragma unroll
        for (int i = 0; i < kHalfCols; ++i) acc[i] = sums[i + zero];
      } else {
#pragma unroll
        for (int i = 0; i < kHalfCols; ++i) acc[i] = __float_as_uint(__int2float_rn((int)(alu_add(i) ? acc[i] : acc[i] - bias_bits)));
      }
      // num / dn correctly rounded from the row's one reciprocal (Markstein, IBM J. Res. Dev. 34, 1990: with y the
      // correctly rounded 1 / b and q within an ulp of a / b, q + (a - b q) y, the remainder by fma, rounds
      // correctly; the first step brings q there).  num = sum * 2^-f over dn is sum over dn * 2^f.
      const float b = __fmul_rn(dn, p.scale), y = __frcp_rn(b);
      const uint64_t y2 = pack2(__float_as_uint(y), __float_as_uint(y)), nb2 = pack2(__float_as_uint(-b), __float_as_uint(-b));
#pragma unroll
      for (int g8 = 0; g8 < kHalfCols / 8; ++g8) {
        uint32_t out[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = g8 * 8 + i * 2;
          const uint64_t a = pack2(acc[c], acc[c + 1]);
          uint64_t q, r;
          asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(a), "l"(y2));
          asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(q), "l"(nb2), "l"(a));
          asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(q) : "l"(r), "l"(y2), "l"(q));
          asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(q), "l"(nb2), "l"(a));
          asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(q) : "l"(r), "l"(y2), "l"(q));
          out[i] = pack2_tc<T>(__uint_as_float((uint32_t)q), __uint_as_float((uint32_t)(q >> 32)));
        }
        if (store) *reinterpret_cast<uint4*>(op + g8 * 8) = make_uint4(out[0], out[1], out[2], out[3]);
      }
    }
  }

  // ------------------------------ teardown ----------------------------------------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // let copies that are still in flight land before shared memory is released
    const long long tw = clock64();
    while (clock64() - tw < 200000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && status) atomicExch(status, FXPR_ERR_TIMEOUT);
    __syncthreads();
  }
  if (warp == 0) {
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

// The prefill kernel takes head sizes 64 and 128, bf16/fp16, 32- or 64-bit sums with at most 16
// fraction bits, no KV split, a sequence short enough for the 32-bit fast sums, and strides
// a tensor map can express (multiples of 16 bytes, below 2^40).
bool attention_tc_supported(const AttnParams& p, int dtype, int max_query_len, bool force_exact) {
  if (force_exact || p.num_splits != 1) return false;
  if (dtype != FXPR_F16 && dtype != FXPR_BF16) return false;
  if ((p.head_dim != 64 && p.head_dim != 128) || p.page_size % 16 != 0) return false;
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
  sh.row_shift = G == 1 ? 0 : G == 2 ? 1 : G == 4 ? 2 : G == 8 ? 3 : 4;
  sh.tokens_per_block = kTcRows / G;
  sh.num_q_blocks = (max_query_len + sh.tokens_per_block - 1) / sh.tokens_per_block;
  sh.page_size = p.page_size;
  sh.group_shift = (p.page_size % 64 == 0) ? 6 : 4;
  sh.page_shift = -1;
  for (int b = 4; b < 31; ++b) if ((1 << b) == p.page_size) sh.page_shift = b;
  const int fmt = dtype == FXPR_BF16 ? 1 : 0;
  sh.idesc_s = make_idesc(fmt, 0, kTcTileN, kTcRows);
  sh.idesc_s2 = make_idesc(fmt, 0, kTcOpN, kTcRows);
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

  // persistent CTAs, one per SM; the list of live items is made on the device
  const int64_t total_items = (int64_t)sh.num_q_blocks * p.num_kv_heads * p.num_reqs;
  if (total_items > 0x7fffffffLL) return FXPR_ERR_UNSUPPORTED;
  dim3 grid((unsigned)std::min<int64_t>(total_items, device_sms()), 1, 1);
  const bool plain = !(p.cap_log2 > 0.0f) && p.alibi == nullptr && p.ss_log2 > 0.0f;
  auto launch = [&](auto k, int smem, bool (&attr_done_dev)[64]) -> int {
    int dev_id = 0;
    cudaGetDevice(&dev_id);
    if (!attr_done_dev[dev_id & 63]) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) { set_last_error("attention_tc smem attribute", e); return FXPR_ERR_CUDA; }
      attr_done_dev[dev_id & 63] = true;
    }
    k<<<grid, kTcThreads, smem, s>>>(mq, mk, mv, p, sh, status, 0);
    return check_launch("attention_tc");
  };
#define FXPR_TC_ATTN(TT, HD, PLAIN)                                                              \
  do {                                                                                           \
    static bool attr_done_dev[64] = {};      /* function attributes are per device */            \
    return launch(attn_tc_prefill_kernel<TT, HD, PLAIN>, TcAttnSmem<HD>::kTotal, attr_done_dev); \
  } while (0)
#define FXPR_TC_ATTN_T(TT)                                                                       \
  do {                                                                                           \
    if (p.head_dim == 128) { if (plain) FXPR_TC_ATTN(TT, 128, true); else FXPR_TC_ATTN(TT, 128, false); } \
    if (plain) FXPR_TC_ATTN(TT, 64, true); else FXPR_TC_ATTN(TT, 64, false);                     \
  } while (0)
  if (dtype == FXPR_BF16) FXPR_TC_ATTN_T(__nv_bfloat16);
  FXPR_TC_ATTN_T(__half);
#undef FXPR_TC_ATTN_T
#undef FXPR_TC_ATTN
}

}  // namespace fxpr
