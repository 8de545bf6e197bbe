// Pieces shared by the fast tensor-core kernels (gemm_tc_fast.cu, gemm_tc_pair.cu, gemm_tc_skinny.cu,
// attention_tc.cu, the decode attention): the magic-number conversion, the exact fix-up of a K-tile
// accumulator and the barrier wait of a whole warp.
#pragma once

#include "fxp_common.cuh"
#include "tc_common.cuh"

namespace fxpr {

static constexpr uint32_t kMagicBits = 0x4B400000u;      // 1.5 * 2^23

static __device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  return __uint_as_float(r);
}

static __device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}

// 1.5 * 2^(23 - f): added to a partial p with |p * 2^f| < 2^22 it rounds p to the Q grid (half to
// even) and leaves rint(p * 2^f) in the low mantissa bits.
static __device__ __forceinline__ uint32_t q_magic_bits(float inv_scale) {
  return __float_as_uint(__fmul_rn(__uint_as_float(kMagicBits), inv_scale));
}

// Which accumulators take the three-input add (these stay bias-free) and which the multiply-add by a
// run-time one (these carry one magic per K-tile).
static __device__ __forceinline__ constexpr bool alu_add(int i) { return (i & 7) < 4; }

// |a| or |b| or |c|, whichever is largest; NaN if any is NaN
static __device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// Partials below this magnitude keep rint(p * 2^f) within +-(2^22 - 1).
static __device__ __forceinline__ float q_screen_limit(float inv_scale) { return __fmul_rn(4194303.0f, inv_scale); }

// N fp32 partials -> Q-format, added to acc; screen keeps the largest magnitude (valid while below
// q_screen_limit).  Per partial half a packed add, one integer add and half a three-input maximum.
// Integer adds run at half rate on the ALU pipe and multiply-adds at half rate on the FMA pipe, so
// they are dealt out evenly: on 128 x 256 partials per SM 760-830 clocks by itself, against 960 with scalar fma
// and the adds left to the compiler (which puts them all on the FMA pipe).
template <int N>
static __device__ __forceinline__ void convert_n(const uint32_t (&v)[N], uint32_t* acc, uint64_t magic2,
                                                 uint32_t magic_bits, uint32_t one, float& screen) {
#pragma unroll
  for (int i = 0; i < N; i += 2) screen = max3_abs(screen, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    uint64_t r;
    uint32_t r0, r1;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(v[i], v[i + 1])), "l"(magic2));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(r0), "=r"(r1) : "l"(r));
    if (alu_add(i)) acc[i] = acc[i] + r0 - magic_bits;
    else asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(acc[i]) : "r"(r0), "r"(one));
    if (alu_add(i + 1)) acc[i + 1] = acc[i + 1] + r1 - magic_bits;
    else asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(acc[i + 1]) : "r"(r1), "r"(one));
  }
}
static __device__ __forceinline__ void convert16(const uint32_t (&v)[16], uint32_t* acc, uint64_t magic2,
                                                 uint32_t magic_bits, uint32_t one, float& screen) {
  convert_n<16>(v, acc, magic2, magic_bits, one, screen);
}

// Rare path, entered by a whole warp (tcgen05.ld is warp-collective): for `ncols` columns of one
// K-tile accumulator, find this lane's out-of-range partials and record (a) the raw value the fast
// path added for them and (b) the reference conversion's result.  Rolled loop, no register arrays:
// small code, off the hot path.
static __device__ __noinline__ void fixup_tile(uint32_t taddr, int ncols, uint32_t magic_bits, float scale, int int_bits,
                                               uint32_t* corr_raw, long long* corr_q) {
#pragma unroll 1
  for (int i = 0; i < ncols; ++i) {
    const float f = tmem_ld1(taddr + i);
    const uint32_t b = __float_as_uint(__fadd_rn(f, __uint_as_float(magic_bits)));
    if (((b ^ magic_bits) >> 23) != 0) {
      corr_raw[i] += b - magic_bits;
      corr_q[i] += (int_bits == 64) ? float_to_fixed<64>(f, scale) : (long long)float_to_fixed<32>(f, scale);
    }
  }
}

// 32-bit sums wrap around, which signed addition must not.
static __device__ __forceinline__ int wrap_add(int a, int b) { return (int)((uint32_t)a + (uint32_t)b); }

// The whole warp probes: 1-7 % faster than one lane probing and a shuffle behind it.
static __device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

}  // namespace fxpr
