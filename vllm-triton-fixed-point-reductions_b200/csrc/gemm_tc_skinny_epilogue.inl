// Epilogue-warp body of gemm_tc_skinny_kernel (included inside the kernel).  Warp w owns TMEM lanes
// 32*(w%4).. -- one output COLUMN n per thread -- and kCols consecutive TMEM columns, which are
// activation rows m.  Same conversion as gemm_tc_fast_epilogue.inl.
//
// Output: the sums go through shared memory as [row][128 columns] of 32-bit integers (they fit unless a
// partial took the exact fix-up), then a warp writes whole rows, four columns a lane.  Written out of the
// registers, a column per thread, the same outputs cost 32 two-byte stores, 32 conversions from 64 bits
// and several KB of straight-line code that runs once a tile: 64 x 4096 x 512 8.2 us, 16 rows 5.3.
{
  const int quarter = warp & 3;
  const int cgroup = (warp - 2) >> 2;
  const int n_in_tile = quarter * 32 + lane;
  const int m0 = cgroup * kCols;
  const uint32_t lane_addr = ((uint32_t)(quarter * 32) << 16) + (uint32_t)m0;
  const uint32_t mbits = q_magic_bits(p.inv_scale), one = (uint32_t)zero + 1u;
  const uint64_t magic2 = pack2(mbits, mbits);
  const float screen_limit = q_screen_limit(p.inv_scale);
  const float scale = p.scale;
  int grp = 0; uint32_t gphase = 0; uint32_t epi_phase = 0; bool ok = true;
  auto epi_sync = [&]() -> bool {   // bounded barrier over the epilogue warps only
    __syncwarp();
    if (lane == 0) mbar_arrive(epi_bar);
    const bool done = warp_wait(epi_bar, epi_phase, abort_flag);
    epi_phase ^= 1;
    return done;
  };

  // Rare-path corrections (local memory, zeroed on first use), as in the wide kernel.
  uint32_t corr_raw[kCols];
  long long corr_q[kCols];
  bool corr_used = false;
  bool announced = false;      // cluster merge: this thread has said that the stages are done

  int* stage32 = reinterpret_cast<int*>(smem_gen + Shape::kSumsOffset);              // [MP][128]
  long long* stage64 = reinterpret_cast<long long*>(smem_gen + Shape::kSumsOffset);  // [MP / 2][128]
  const bool c_vec4 = ((uintptr_t)p.c & 7) == 0 && p.c_sm % 4 == 0;
  float bias4[4];

  // four neighbouring sums of row m, columns n4..n4 + 3, to the outputs; called by whole warps
  auto emit = [&](int m, int n4, auto q0, auto q1, auto q2, auto q3) {
    using Q = decltype(q0);
    Q q[4] = {q0, q1, q2, q3};
    if (p.c_int) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (n4 + i >= p.N) continue;
        if (p.int_bits == 64) ((long long*)p.c_int)[(int64_t)m * p.N + n4 + i] = (long long)q[i];
        else ((int32_t*)p.c_int)[(int64_t)m * p.N + n4 + i] = (int32_t)q[i];
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
    if (p.silu_mul) {
      // columns come in (gate, up) pairs: the outputs as the io dtype holds them give columns n4 / 2 and
      // n4 / 2 + 1 of the [M, N / 2] result
      T* dst = (T*)p.c + (int64_t)m * p.c_sm + (n4 >> 1);
      if (n4 + 1 < p.N) dst[0] = silu_mul_io<T>(to_f32<T>(out[0]), to_f32<T>(out[1]));
      if (n4 + 3 < p.N) dst[1] = silu_mul_io<T>(to_f32<T>(out[2]), to_f32<T>(out[3]));
      return;
    }
    T* dst = (T*)p.c + (int64_t)m * p.c_sm + n4;
    if (c_vec4 && n4 + 4 <= p.N) {
      *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(out);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) if (n4 + i < p.N) dst[i] = out[i];
    }
    if (p.best) {
      // Greedy sampling without a pass over the logits: the best (value, column) key of the row's 128
      // columns, one atomic maximum
      unsigned long long key = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (n4 + i >= p.N) continue;
        const unsigned long long k = argmax_key(to_f32<T>(out[i]), p.n_offset + (unsigned int)(n4 + i));
        key = key > k ? key : k;
      }
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, d);
        key = key > other ? key : other;
      }
      if (lane == 0 && key != 0ull) atomicMax(p.best + m, key);
    }
  };

  int n4 = 0;                                            // output columns of this lane
  for (int tile = tile0, it = 0;; ++it) {
  const int flag = WALK ? it & 1 : 0;                    // of s_wide
  n4 = tile * 128 + lane * 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) bias4[i] = p.bias && n4 + i < p.N ? to_f32<T>(((const T*)p.bias)[n4 + i]) : 0.0f;
  corr_used = false;
  uint32_t acc[kCols];
#pragma unroll
  for (int i = 0; i < kCols; ++i) acc[i] = 0;

  for (int kt = 0; kt < n_kt; ++kt) {
    if (!warp_wait(tfull0 + 8u * grp, gphase, abort_flag)) { ok = false; break; }
    tc_fence_after();
    if constexpr (CLUSTER) {
      // the last accumulator is complete, so no MMA or copy touches the stages any more
      if (kt == n_kt - 1) { cluster_arrive(); announced = true; }
    }
    const uint32_t ta = tmem_base + lane_addr + (uint32_t)(grp * MP);
    float screen = 0.0f;
    if constexpr (kCols == 32) {
      // two loads are requested before the wait
      uint32_t va[16], vb[16];
      tmem_ld16(ta, va); tmem_ld16(ta + 16, vb); tmem_wait_ld_regs2(va, vb);
      convert_n<16>(va, acc, magic2, mbits, one, screen); convert_n<16>(vb, acc + 16, magic2, mbits, one, screen);
    } else {
      uint32_t v[kCols];
      if constexpr (kCols == 16) tmem_ld16(ta, v); else tmem_ld8(ta, v);
      tmem_wait_ld_regs(v);
      convert_n<kCols>(v, acc, magic2, mbits, one, screen);
    }
    if (__any_sync(0xffffffffu, !(screen < screen_limit))) {
      if (!corr_used) {
#pragma unroll 1
        for (int z = 0; z < kCols; ++z) { corr_raw[z + zero] = 0; corr_q[z + zero] = 0; }
        corr_used = true;
      }
      fixup_tile(ta, kCols, mbits, scale, p.int_bits, &corr_raw[zero], &corr_q[zero]);
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(tempty0 + 8u * grp);
    if (++grp == GROUPS) { grp = 0; gphase ^= 1; }
  }
  if (WALK && ok && it) ok = epi_sync();                 // the last tile's sums have been read
  if (ok) {
    const uint32_t bias_bits = (uint32_t)n_kt * mbits;   // the multiply-adds summed one magic per K-tile
    // the sum without corrections is below 2^31 in magnitude (at most 510 K-tiles of less than 2^22)
    auto total32 = [&](int i) -> uint32_t { return alu_add(i) ? acc[i] : acc[i] - bias_bits; };
    auto total = [&](int i) -> long long {
      uint32_t raw = total32(i);
      long long t;
      if (corr_used) {
        raw -= corr_raw[i + zero];
        t = (long long)(int32_t)raw + corr_q[i + zero];
      } else {
        t = (long long)(int32_t)raw;
      }
      return p.int_bits == 64 ? t : (long long)(int32_t)t;
    };
    // low words of the sums to shared memory; with a fix-up in this warp the exact ones
    auto park32 = [&]() {
      if (!corr_used) {
#pragma unroll
        for (int i = 0; i < kCols; ++i) stage32[(m0 + i) * 128 + n_in_tile] = (int)total32(i);
      } else {
#pragma unroll
        for (int i = 0; i < kCols; ++i) stage32[(m0 + i) * 128 + n_in_tile] = (int)total(i);
      }
    };

    if constexpr (CLUSTER) {
      // This split's sums go to shared memory, 32 bits each; where a fix-up made some of them larger,
      // the high words too, and the rank says so in its flag.
      park32();
      if (corr_used && p.int_bits == 64) {
        int* high = reinterpret_cast<int*>(smem_gen + Shape::kHighOffset);
#pragma unroll
        for (int i = 0; i < kCols; ++i) high[(m0 + i) * 128 + n_in_tile] = (int)(total(i) >> 32);
        if (lane == 0) atomicOr((int*)s_wide, 1 << (cgroup * 4 + quarter));
      }
    } else {
      // Split-K: per-split integer partial planes, column-major inside the 128 x MP tile (the
      // warp's 32 output columns are 32 consecutive words); the last arriver adds the others.
      bool do_store = true;
      const bool split = p.split_k > 1;
      const int64_t plane_elems = (int64_t)128 * MP;
      const int64_t plane_stride = (int64_t)tiles_n * plane_elems;
      const int64_t plane_off = (int64_t)tile * plane_elems + (int64_t)m0 * 128 + n_in_tile;
      if (split) {
        if (p.int_bits == 64) {
          long long* dst = (long long*)p.acc_scratch + ks * plane_stride + plane_off;
#pragma unroll
          for (int i = 0; i < kCols; ++i) __stcg(dst + i * 128, total(i));
        } else {
          int* dst = (int*)p.acc_scratch + ks * plane_stride + plane_off;
#pragma unroll
          for (int i = 0; i < kCols; ++i) __stcg(dst + i * 128, (int)total(i));
        }
        __threadfence();
        ok = epi_sync();
        if (threadIdx.x == 64) *s_last = (atomicAdd(p.locks + tile, 1) == p.split_k - 1) ? 1 : 0;
        ok = ok && epi_sync();
        do_store = ok && *s_last != 0;
        if (do_store) __threadfence();
      } else {
        if (corr_used && p.int_bits == 64) s_wide[flag] = 1;
        else park32();                                   // not read when another warp makes the tile a wide one
        do_store = ok = epi_sync();
        if (WALK && threadIdx.x == 64) s_wide[flag ^ 1] = 0;   // read by all before this tile's first barrier
      }
      if (do_store && !split && !s_wide[flag]) {
        for (int m = warp - 2; m < live_rows; m += EPIW) {
          const int4 v = *reinterpret_cast<const int4*>(stage32 + m * 128 + lane * 4);
          emit(m, n4, v.x, v.y, v.z, v.w);
        }
      } else if (do_store) {
        // 64-bit sums, half of the rows at a time
        for (int half = 0; half < 2; ++half) {
          if (!epi_sync()) { ok = false; break; }
          if (cgroup == half) {
#pragma unroll
            for (int i = 0; i < kCols; ++i) {
              long long q = total(i);
              if (split) {
                for (int s2 = 0; s2 < p.split_k; ++s2) {
                  if (s2 == ks) continue;
                  const int64_t at = s2 * plane_stride + plane_off + i * 128;
                  q += p.int_bits == 64 ? __ldcg((const long long*)p.acc_scratch + at)
                                        : (long long)__ldcg((const int*)p.acc_scratch + at);
                }
                if (p.int_bits != 64) q = (long long)(int32_t)q;
              }
              stage64[i * 128 + n_in_tile] = q;
            }
          }
          if (!epi_sync()) { ok = false; break; }
          const int base = half * kCols;
          for (int m = warp - 2; m < kCols && base + m < live_rows; m += EPIW) {
            const longlong2 v = *reinterpret_cast<const longlong2*>(stage64 + m * 128 + lane * 4);
            const longlong2 w = *reinterpret_cast<const longlong2*>(stage64 + m * 128 + lane * 4 + 2);
            emit(base + m, n4, v.x, v.y, w.x, w.y);
          }
        }
      }
      if (split && do_store && threadIdx.x == 64) p.locks[tile] = 0;
    }
  }
  if (!WALK || !ok || (tile += (int)gridDim.x) >= tiles_n) break;
  }

  if constexpr (CLUSTER) {
    // ------------------------------ cluster merge ---------------------------------
    // Every rank has parked its sums and announced, at its last accumulator, that its stages are done.
    // Once all have, a rank sends each of the others its rows by one bulk copy (and its flag by
    // another) into the stages there, then sums its own rows out of its own shared memory.  Pulling
    // them with loads over distributed shared memory instead took 64-bit sums of all 64 padded rows
    // 2.5 us longer at 16 x 4096 x 4096.  Every thread of every CTA arrives at and waits for both cluster
    // barriers, also after a timed-out wait.
    const int S = p.split_k, rank = (int)blockIdx.x, my_rows = rows_of(rank);
    if (!announced) cluster_arrive();
    fence_proxy_async_smem();                            // what this thread parked, for the bulk copies
    if (ok) ok = epi_sync();
    cluster_wait();
    if (ok) {
      const int to = warp - 2;                           // warp w sends rank w's rows
      if (to < S && to != rank && lane == 0 && rows_of(to) > 0) {
        const int slot = rank < to ? rank : rank - 1;
        if (*s_wide) mbar_arrive_release_cluster(mapa_u32(high_bar, (uint32_t)to));   // peers read the high words with plain loads
        const uint32_t bar = mapa_u32(recv_bar, (uint32_t)to);
        bulk_copy_cluster(mapa_u32(smem_base + Shape::kRecvOffset + (uint32_t)(slot * rows_of(to) * 512), (uint32_t)to),
                          smem_base + (uint32_t)(to * rows_per * 512), (uint32_t)(rows_of(to) * 512), bar);
        bulk_copy_cluster(mapa_u32(smem_base + Shape::kFlagOffset + (uint32_t)(slot * 16), (uint32_t)to),
                          smem_u32((const void*)s_wide), 16u, bar);
      }
      __syncwarp();
      if (my_rows > 0) ok = warp_wait(recv_bar, 0, abort_flag);
    }
    unsigned long long wide = 0;                         // a byte per rank: its warps that parked high words
    if (ok && my_rows > 0) {
      const int* flags = reinterpret_cast<const int*>(smem_gen + Shape::kFlagOffset);
      wide = (unsigned long long)*s_wide << (8 * rank);
      for (int rr = 0; rr < S - 1; ++rr) wide |= (unsigned long long)flags[rr * 4] << (8 * (rr < rank ? rr : rr + 1));
    }
    if (wide) {
      // the high words of every peer that has some; its own arrivals stand for the other peers
      if (warp == 2 && lane == 0) {
        int none = S - 1;
        for (int r = 0; r < S; ++r) none -= r != rank && ((wide >> (8 * r)) & 0xff);
        if (none) mbar_arrive_n(high_bar, (uint32_t)none);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait_acquire_cluster(high_bar, 0, abort_flag));
    } else {
      cluster_arrive();                                  // this rank has what was sent to it
    }
    if (ok) {
      const int* mine = stage32 + rank * rows_per * 128;
      const int* recv = reinterpret_cast<const int*>(smem_gen + Shape::kRecvOffset);
      if (!wide && (k_tiles_total <= 510 || p.int_bits == 32)) {
        // sums over all ranks are below 2^31 in magnitude, or wrap to 32 bits
        for (int mr = warp - 2; mr < my_rows; mr += EPIW) {
          int4 q = *reinterpret_cast<const int4*>(mine + mr * 128 + lane * 4);
          for (int rr = 0; rr < S - 1; ++rr) {
            const int4 v = *reinterpret_cast<const int4*>(recv + (rr * my_rows + mr) * 128 + lane * 4);
            q.x = wrap_add(q.x, v.x); q.y = wrap_add(q.y, v.y); q.z = wrap_add(q.z, v.z); q.w = wrap_add(q.w, v.w);
          }
          emit(rank * rows_per + mr, n4, q.x, q.y, q.z, q.w);
        }
      } else {
#pragma unroll 1
        for (int mr = warp - 2; mr < my_rows; mr += EPIW) {
          const int m = rank * rows_per + mr;
          long long q[4] = {0, 0, 0, 0};
#pragma unroll 1
          for (int r = 0; r < S; ++r) {
            const int* low = r == rank ? mine + mr * 128 : recv + ((r < rank ? r : r - 1) * my_rows + mr) * 128;
            const uint32_t high = mapa_u32(smem_base + Shape::kHighOffset + (uint32_t)((m * 128 + lane * 4) * 4), (uint32_t)r);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int lo = low[lane * 4 + i];
              if ((wide >> (8 * r + m / kCols * 4 + (lane >> 3))) & 1) {
                q[i] += ((long long)ld_cluster_s32(high + 4u * i) << 32) | (long long)(uint32_t)lo;
              } else {
                q[i] += (long long)lo;
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) q[i] = p.int_bits == 64 ? q[i] : (long long)(int32_t)q[i];
          emit(m, n4, q[0], q[1], q[2], q[3]);
        }
      }
    }
    if (wide) cluster_arrive();
  }
}
