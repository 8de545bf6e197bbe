// Portable fixed-point GEMM on CUDA cores: any dtype, any strides, any shape.
//
// It is the route for operands the tensor-core kernel cannot take (fp32 inputs,
// leading dimensions that break TMA's 16-byte rule, very small N or K) and the
// cross-check for that kernel.  Which route a problem takes depends only on
// (dtype, N, K, strides) -- never on M -- so a row's bits never depend on the
// batch it arrives in.
//
// Semantics: fxpr_vllm/_triton/gemm.py:183-204 of the reference.  Per K-tile
// the fp32 partial is formed by adding products in ascending k with separate
// multiply and add (bit-reproducible on a CPU), quantised with float_to_fixed and
// added as an integer; the epilogue converts once, adds the bias in fp32 and
// rounds to the IO dtype.  The K tail is zero padding (adds nothing).
//
// Bound: multiplies and adds are separate instructions, so half the FFMA rate, for large M; reading B for
// small M.  A thread holds RM x 4 outputs (three 16-byte shared-memory reads per 64 instructions at
// RM = 8; 512x4096x4096 fp32 2147 -> 897 us, floor 477), the next chunk of K travels to registers while
// this one is multiplied, both operands are
// read along whichever of their strides is one, and K-tiles are dealt to the ranks of a cluster when
// the tiles of the output leave the GPU idle (integer sums: no bit depends on it).
#include <algorithm>

#include <cooperative_groups.h>

#include "fxp_common.cuh"

namespace cg = cooperative_groups;

namespace fxpr {

static constexpr int kPN = 64;   // output columns per CTA
static constexpr int kPK = 16;   // k chunk staged in shared memory

template <int RM>
constexpr int portable_smem() { return 2 * kPK * (16 * RM + 4 + kPN + 4) * 4 + 16 * RM * kPN * 8; }
constexpr int portable_ctas(int rm) { return rm == 8 ? 2 : rm == 4 ? 3 : 4; }   // resident per SM

template <typename T>
__device__ __forceinline__ void portable_write(int m, int n, long long sum, const T* bias, T* c, void* c_int, int N,
                                               int64_t c_sm, int int_bits, float inv_scale) {
  const long long q = wrap_to_bits(sum, int_bits);
  if (c_int) {
    const int64_t o = (int64_t)m * N + n;
    if (int_bits == 64) ((long long*)c_int)[o] = q;
    else if (int_bits == 32) ((int32_t*)c_int)[o] = (int32_t)q;
    else ((int16_t*)c_int)[o] = (int16_t)q;
  }
  if (c) {
    float v = fixed_to_float<long long>(q, inv_scale);
    if (bias) v = __fadd_rn(v, to_f32<T>(bias[n]));
    c[(int64_t)m * c_sm + n] = from_f32<T>(v);
  }
}

template <typename T, int RM>
__global__ void __launch_bounds__(256, portable_ctas(RM))
gemm_portable_kernel(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ bias,
                     T* __restrict__ c, void* __restrict__ c_int, float* __restrict__ partials,
                     int M, int N, int K, int64_t a_sm, int64_t a_sk, int64_t b_sk, int64_t b_sn,
                     int64_t c_sm, int int_bits, float scale, float inv_scale, int k_tile, int splits, float zero /* 0 */) {
  constexpr int TM = 16 * RM, LA = TM + 4, LB = kPN + 4;
  extern __shared__ __align__(16) uint8_t smem[];
  float* sa = reinterpret_cast<float*>(smem);        // [2][kPK][LA]
  float* sb = sa + 2 * kPK * LA;                      // [2][kPK][LB]
  // Integer sums, touched once per K-tile, each by the thread that owns it: [RM * 4][256].  In registers
  // they would leave one CTA per SM at RM = 8.
  long long* acc = reinterpret_cast<long long*>(sb + 2 * kPK * LB);
  pdl_wait();
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int rank = blockIdx.x % splits;
  const int m0 = blockIdx.y * TM, n0 = (blockIdx.x / splits) * kPN;
  const bool a_along_k = a_sk == 1, b_along_n = b_sn == 1;
  uint64_t p[RM][2];                                 // pairs of neighbouring columns
  const uint64_t zero2 = f2_pack(zero, zero);
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[(i * 4 + j) * 256 + tid] = 0; p[i][j >> 1] = 0; }

  const int tiles = (K + k_tile - 1) / k_tile;
  // element `it` of this thread's share of a chunk: its place in the A and in the B chunk
  auto a_place = [&](int it, int& kk, int& mm) {
    const int idx = tid + it * 256;
    if (a_along_k) { kk = idx & (kPK - 1); mm = idx / kPK; } else { mm = idx % TM; kk = idx / TM; }
  };
  auto b_place = [&](int it, int& kk, int& nn) {
    const int idx = tid + it * 256;
    if (b_along_n) { nn = idx & (kPN - 1); kk = idx / kPN; } else { kk = idx & (kPK - 1); nn = idx / kPK; }
  };
  float ra[RM], rb[4];
  auto fetch = [&](int kc, int kn) {                 // what lies outside is zero and adds nothing
#pragma unroll
    for (int it = 0; it < RM; ++it) {
      int kk, mm;
      a_place(it, kk, mm);
      ra[it] = (kk < kn && m0 + mm < M) ? to_f32<T>(a[(int64_t)(m0 + mm) * a_sm + (int64_t)(kc + kk) * a_sk]) : 0.0f;
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      int kk, nn;
      b_place(it, kk, nn);
      rb[it] = (kk < kn && n0 + nn < N) ? to_f32<T>(b[(int64_t)(kc + kk) * b_sk + (int64_t)(n0 + nn) * b_sn]) : 0.0f;
    }
  };
  auto k_end = [&](int t) { return (int)min((int64_t)K, (int64_t)(t + 1) * k_tile); };

  int t = rank, kc = rank * k_tile, buf = 0;
  if (t < tiles) fetch(kc, k_end(t) - kc);
  while (t < tiles) {
    float* ca = sa + buf * kPK * LA;
    float* cb = sb + buf * kPK * LB;
    buf ^= 1;
#pragma unroll
    for (int it = 0; it < RM; ++it) { int kk, mm; a_place(it, kk, mm); ca[kk * LA + mm] = ra[it]; }
#pragma unroll
    for (int it = 0; it < 4; ++it) { int kk, nn; b_place(it, kk, nn); cb[kk * LB + nn] = rb[it]; }
    __syncthreads();                                 // this chunk is in place, the one before last is free
    const int t_now = t;
    kc += kPK;
    const bool tile_done = kc >= k_end(t);
    if (tile_done) { t += splits; kc = t < tiles ? t * k_tile : 0; }
    if (t < tiles) fetch(kc, k_end(t) - kc);
#pragma unroll
    for (int kk = 0; kk < kPK; ++kk) {
      float av[RM];
      if constexpr (RM >= 4) {
#pragma unroll
        for (int i = 0; i < RM; i += 4) *reinterpret_cast<float4*>(av + i) = *reinterpret_cast<const float4*>(ca + kk * LA + ty * RM + i);
      } else {
#pragma unroll
        for (int i = 0; i < RM; ++i) av[i] = ca[kk * LA + ty * RM + i];
      }
      const ulonglong2 bv = *reinterpret_cast<const ulonglong2*>(cb + kk * LB + tx * 4);
      // Two columns per instruction.  The product is an fma with a run-time zero: ptxas contracts a packed
      // multiply and the add behind it, which would round once instead of twice.
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const uint64_t a2 = f2_pack(av[i], av[i]);
        p[i][0] = f2_add(p[i][0], f2_fma(a2, bv.x, zero2));
        p[i][1] = f2_add(p[i][1], f2_fma(a2, bv.y, zero2));
      }
    }
    if (tile_done) {
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        float v[4];
        f2_unpack(p[i][0], v[0], v[1]);
        f2_unpack(p[i][1], v[2], v[3]);
        p[i][0] = p[i][1] = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[(i * 4 + j) * 256 + tid] += float_to_fixed_any(v[j], scale, int_bits);
          if (partials) {
            const int m = m0 + ty * RM + i, n = n0 + tx * 4 + j;
            if (m < M && n < N) partials[((int64_t)t_now * M + m) * N + n] = v[j];
          }
        }
      }
    }
  }

  // where the idx-th sum of a CTA belongs
  auto place = [&](int idx, int& m, int& n) {
    m = m0 + ((idx & 255) >> 4) * RM + (idx >> 10);
    n = n0 + (idx & 15) * 4 + ((idx >> 8) & 3);
    return m < M && n < N;
  };
  if (splits == 1) {
    for (int idx = tid; idx < TM * kPN; idx += 256) {
      int m, n;
      if (place(idx, m, n)) portable_write(m, n, acc[idx], bias, c, c_int, N, c_sm, int_bits, inv_scale);
    }
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int idx = rank * 256 + tid; idx < TM * kPN; idx += splits * 256) {
    int m, n;
    if (!place(idx, m, n)) continue;
    long long sum = 0;
    for (int r = 0; r < splits; ++r) sum += cluster.map_shared_rank(acc, r)[idx];
    portable_write(m, n, sum, bias, c, c_int, N, c_sm, int_bits, inv_scale);
  }
  cluster.sync();                                    // peers may still be reading this CTA's sums
}

// Few rows: bound by reading B, which here goes straight to registers, 16 bytes per lane and
// eight rows of K at a time.  K-tiles are independent up to their integer sums, so every warp of a CTA (and
// of the cluster) takes its own: a warp is 128 columns x R rows of one K-tile.  fp32, K-tile 128, against
// the tiled kernel above: 1x4096x4096 67 -> 18 us, 8x28672x4096 453 -> 161.
template <typename T, int R>
__global__ void __launch_bounds__(256, 2)
gemm_portable_rows_kernel(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ bias,
                          T* __restrict__ c, void* __restrict__ c_int, float* __restrict__ partials,
                          int M, int N, int K, int64_t a_sm, int64_t a_sk, int64_t b_sk,
                          int64_t c_sm, int int_bits, float scale, float inv_scale, int k_tile, int splits,
                          float zero /* 0 */) {
  struct alignas(4 * sizeof(T)) Vec { T v[4]; };
  __shared__ __align__(16) float sa[8][32][R + 4];   // a warp's slice of A, k-major
  __shared__ unsigned long long acc[R * 128];
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % splits, n0 = (blockIdx.x / splits) * 128;
  const int n = n0 + lane * 4, m0 = blockIdx.y * R;
  for (int i = tid; i < R * 128; i += 256) acc[i] = 0;
  __syncthreads();
  const uint64_t zero2 = f2_pack(zero, zero);
  const int tiles = (K + k_tile - 1) / k_tile;
  for (int t = rank * 8 + warp; t < tiles; t += splits * 8) {
    uint64_t p[R][2];
#pragma unroll
    for (int i = 0; i < R; ++i) p[i][0] = p[i][1] = 0;
    const int k_hi = (int)min((int64_t)K, (int64_t)(t + 1) * k_tile);
    for (int kc = t * k_tile; kc < k_hi; kc += 32) {
      __syncwarp();
#pragma unroll
      for (int m = 0; m < R; ++m)
        sa[warp][lane][m] = (m0 + m < M && kc + lane < k_hi) ? to_f32<T>(a[(int64_t)(m0 + m) * a_sm + (int64_t)(kc + lane) * a_sk]) : 0.0f;
      __syncwarp();
#pragma unroll 1
      for (int k8 = 0; k8 < 32 && kc + k8 < k_hi; k8 += 8) {
        Vec bv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int k = kc + k8 + u;
          if (k < k_hi && n < N) bv[u] = *reinterpret_cast<const Vec*>(b + (int64_t)k * b_sk + n);
          else bv[u] = Vec{};
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint64_t b01 = f2_pack(to_f32<T>(bv[u].v[0]), to_f32<T>(bv[u].v[1]));
          const uint64_t b23 = f2_pack(to_f32<T>(bv[u].v[2]), to_f32<T>(bv[u].v[3]));
#pragma unroll
          for (int m4 = 0; m4 < R; m4 += 4) {
            const float4 av = *reinterpret_cast<const float4*>(&sa[warp][k8 + u][m4]);
            const float am[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint64_t a2 = f2_pack(am[i], am[i]);
              p[m4 + i][0] = f2_add(p[m4 + i][0], f2_fma(a2, b01, zero2));
              p[m4 + i][1] = f2_add(p[m4 + i][1], f2_fma(a2, b23, zero2));
            }
          }
        }
      }
    }
#pragma unroll
    for (int m = 0; m < R; ++m) {
      if (m0 + m >= M || n >= N) continue;
      float v[4];
      f2_unpack(p[m][0], v[0], v[1]);
      f2_unpack(p[m][1], v[2], v[3]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        atomicAdd(&acc[m * 128 + lane * 4 + j], (unsigned long long)float_to_fixed_any(v[j], scale, int_bits));
        if (partials) partials[((int64_t)t * M + m0 + m) * N + n + j] = v[j];
      }
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (splits > 1) cluster.sync(); else __syncthreads();
  for (int idx = rank * 256 + tid; idx < R * 128; idx += splits * 256) {
    const int m = m0 + (idx >> 7), col = n0 + (idx & 127);
    if (m >= M || col >= N) continue;
    long long sum = 0;
    if (splits > 1) {
      for (int r = 0; r < splits; ++r) sum += (long long)cluster.map_shared_rank(acc, r)[idx];
    } else {
      sum = (long long)acc[idx];
    }
    portable_write(m, col, sum, bias, c, c_int, N, c_sm, int_bits, inv_scale);
  }
  if (splits > 1) cluster.sync();                    // peers may still be reading this CTA's sums
}

// c = T(fp32(c_int) * 2^-frac + bias)
template <typename T, typename I>
__global__ void __launch_bounds__(256)
epilogue_from_int_kernel(const I* __restrict__ c_int, const T* __restrict__ bias, T* __restrict__ c,
                         int64_t M, int64_t N, int64_t c_sm, float inv_scale) {
  const int64_t total = M * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = i / N, n = i - m * N;
    float v = fixed_to_float<I>(c_int[i], inv_scale);
    if (bias) v = __fadd_rn(v, to_f32<T>(bias[n]));
    c[m * c_sm + n] = from_f32<T>(v);
  }
}

template <typename T>
int gemm_portable_launch(const void* a, const void* b, const void* bias, void* c, void* c_int,
                         float* partials, int64_t M, int64_t N, int64_t K, int64_t a_sm,
                         int64_t a_sk, int64_t b_sk, int64_t b_sn, int64_t c_sm, int int_bits,
                         int frac_bits, int k_tile, cudaStream_t s) {
  const float scale = (float)(1ull << frac_bits);
  // Few rows, B readable 4 columns at a time and K-tiles for the eight warps of a CTA: one K-tile per warp,
  // 8 or 16 rows.  Three such row blocks cost less than one 64-row tile (27x28672x4096 fp32 836 -> 499 us).
  const int k_tiles = ceil_div_i(K, k_tile), sms = device_sms();
  if (M <= 48 && k_tiles >= 8 && b_sn == 1 && b_sk % 4 == 0 && N % 4 == 0 && ((uintptr_t)b % (4 * sizeof(T))) == 0) {
    const int64_t cols = ceil_div_i(N, 128), blocks = ceil_div_i(M, M <= 8 ? 8 : 16);
    int splits = 1;
    while (splits < 8 && splits * 8 < k_tiles && cols * blocks * splits * 2 <= 4 * sms) splits *= 2;
    auto rows = [&](auto kernel) {
      const cudaError_t e = launch_pdl(kernel, dim3((unsigned)(cols * splits), (unsigned)blocks), dim3(256), 0, s, (unsigned)splits,
                                       (const T*)a, (const T*)b, (const T*)bias, (T*)c, c_int, partials, (int)M, (int)N,
                                       (int)K, a_sm, a_sk, b_sk, c_sm, int_bits, scale, 1.0f / scale, k_tile, splits, 0.0f);
      if (e != cudaSuccess) { set_last_error("gemm_portable launch", e); return (int)FXPR_ERR_CUDA; }
      return check_launch("gemm_portable");
    };
    return M <= 8 ? rows(gemm_portable_rows_kernel<T, 8>) : rows(gemm_portable_rows_kernel<T, 16>);
  }
  // Rows per CTA: 16 when that covers M.  Otherwise 64 or 128 (whose products cost a sixth less), and for
  // every choice 1 to 8 cluster ranks that share the K-tiles: whichever gives the shortest rounds, counted
  // in rows of work per SM.  A doubling of the ranks costs about 3 % (the merge).
  const int64_t tiles_n = ceil_div_i(N, kPN);
  int rm = 1, splits = 1;
  double best = 1e300;
  for (int r : {1, 4, 8}) {
    if ((r == 1) != (M <= 16)) continue;
    const int64_t ctas = tiles_n * ceil_div_i(M, 16 * r);
    double fee = r == 4 ? 1.17 : 1.0;
    for (int n = 1; n <= 8 && n <= std::max(1, ceil_div_i(K, k_tile)); n *= 2, fee *= 1.03) {
      const int per_sm = portable_ctas(r);
      const int64_t whole = ctas * n / (sms * per_sm), rest = ctas * n % (sms * per_sm);
      // a last round of fewer CTAs per SM is shorter, but never as short as its share
      const double rounds = (double)whole * per_sm + (rest ? std::max(0.6 * per_sm, (double)ceil_div_i(rest, sms)) : 0.0);
      const double cost = rounds * r / n * fee;
      if (cost < best) { best = cost; rm = r; splits = n; }
    }
  }
  const int64_t tiles_m = ceil_div_i(M, 16 * rm);
  auto launch = [&](auto kernel, int smem) {
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) { set_last_error("gemm_portable smem attribute", e); return (int)FXPR_ERR_CUDA; }
    }
    const cudaError_t e = launch_pdl(kernel, dim3((unsigned)(tiles_n * splits), (unsigned)tiles_m), dim3(256), smem, s,
                                     (unsigned)splits, (const T*)a, (const T*)b, (const T*)bias, (T*)c, c_int, partials,
                                     (int)M, (int)N, (int)K, a_sm, a_sk, b_sk, b_sn, c_sm, int_bits, scale, 1.0f / scale,
                                     k_tile, splits, 0.0f);
    if (e != cudaSuccess) { set_last_error("gemm_portable launch", e); return (int)FXPR_ERR_CUDA; }
    return check_launch("gemm_portable");
  };
  if (rm == 1) return launch(gemm_portable_kernel<T, 1>, portable_smem<1>());
  if (rm == 4) return launch(gemm_portable_kernel<T, 4>, portable_smem<4>());
  return launch(gemm_portable_kernel<T, 8>, portable_smem<8>());
}

int gemm_portable(const void* a, const void* b, const void* bias, void* c, void* c_int,
                  float* partials, int dtype, int64_t M, int64_t N, int64_t K, int64_t a_sm,
                  int64_t a_sk, int64_t b_sk, int64_t b_sn, int64_t c_sm, int int_bits,
                  int frac_bits, int k_tile, cudaStream_t s) {
  switch (dtype) {
    case FXPR_F32:
      return gemm_portable_launch<float>(a, b, bias, c, c_int, partials, M, N, K, a_sm, a_sk, b_sk, b_sn, c_sm, int_bits, frac_bits, k_tile, s);
    case FXPR_F16:
      return gemm_portable_launch<__half>(a, b, bias, c, c_int, partials, M, N, K, a_sm, a_sk, b_sk, b_sn, c_sm, int_bits, frac_bits, k_tile, s);
    case FXPR_BF16:
      return gemm_portable_launch<__nv_bfloat16>(a, b, bias, c, c_int, partials, M, N, K, a_sm, a_sk, b_sk, b_sn, c_sm, int_bits, frac_bits, k_tile, s);
  }
  return FXPR_ERR_UNSUPPORTED;
}

template <typename T>
static int epilogue_dispatch(const void* c_int, int int_bits, const void* bias, void* c, int64_t M,
                             int64_t N, int64_t c_sm, float inv, cudaStream_t s) {
  const int64_t total = M * N;
  int grid = (int)((total + 255) / 256);
  grid = std::min(grid, device_sms() * 16);
  if (int_bits == 64)
    epilogue_from_int_kernel<T, long long><<<grid, 256, 0, s>>>((const long long*)c_int, (const T*)bias, (T*)c, M, N, c_sm, inv);
  else if (int_bits == 32)
    epilogue_from_int_kernel<T, int32_t><<<grid, 256, 0, s>>>((const int32_t*)c_int, (const T*)bias, (T*)c, M, N, c_sm, inv);
  else
    epilogue_from_int_kernel<T, int16_t><<<grid, 256, 0, s>>>((const int16_t*)c_int, (const T*)bias, (T*)c, M, N, c_sm, inv);
  return check_launch("gemm_epilogue_from_int");
}

}  // namespace fxpr

using namespace fxpr;

extern "C" int fxpr_gemm_epilogue_from_int(const void* c_int, int int_bits, const void* bias,
                                           void* c, int dtype, int64_t M, int64_t N, int64_t c_sm,
                                           int frac_bits, void* stream) {
  if (M < 0 || N < 0 || frac_bits < 0 || frac_bits >= 64) return FXPR_ERR_BAD_ARG;
  if (int_bits != 16 && int_bits != 32 && int_bits != 64) return FXPR_ERR_BAD_ARG;
  if (M == 0 || N == 0) return FXPR_OK;
  if (!c_int || !c) return FXPR_ERR_BAD_ARG;
  const float inv = 1.0f / (float)(1ull << frac_bits);
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case FXPR_F32: return epilogue_dispatch<float>(c_int, int_bits, bias, c, M, N, c_sm, inv, s);
    case FXPR_F16: return epilogue_dispatch<__half>(c_int, int_bits, bias, c, M, N, c_sm, inv, s);
    case FXPR_BF16: return epilogue_dispatch<__nv_bfloat16>(c_int, int_bits, bias, c, M, N, c_sm, inv, s);
  }
  return FXPR_ERR_UNSUPPORTED;
}
