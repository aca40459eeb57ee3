// Index scores of prefill rows on the tcgen05 tensor cores.  Included by indexer.cu inside its anonymous
// namespace (ScoreParams).
//
//   S[key, (row, head)] = K[key, :] . Q[row, head, :]       A = 128 keys, B = 256 / heads rows of all heads
//   score[row, key]     = sum_h relu(S) w[row, h]
//
// With the keys as rows of the MMA an epilogue thread owns one key: the sum over the heads is a sum over its own
// columns (no shuffles) and a warp stores 32 consecutive keys of a row.  The mma.sync kernel has 16 (row,
// head) pairs as rows, dequantises every key tile for 32 rows only and exchanges the heads between
// lanes: 0.14 PFLOP/s, 4.0 ms for 16,384 rows x 16,384 keys on average x 8 heads of 128.
//
// Work item = (row tile, up to `per` key tiles); persistent CTAs, one per SM:
//   warps 0-3   Q of the item (bf16 -> f16, two buffers), then its key tiles: one key per thread, e2m1 ->
//               f16 (value times block scale), two stages
//   warps 4-7, 9-12   epilogue, one 32-lane quadrant and half of the columns each; also blank the columns past a row's
//               valid keys
//   warp 8      one thread issues the MMAs (128 x 256 x 128, two accumulators of 256 columns)
// 2,048 rows x 32,768 keys x 8 heads: 269 us (0.51 PFLOP/s).  Four epilogue warps, each row's sums behind the store of the
// one before, and keys converted through fp32 took 318.  The MMAs keep the tensor pipe busy for a quarter of it; the
// issue slots are 57 % taken (relu and weighted sum of every product on the ALU and FMA pipes), and without MMAs and
// stores the rest still takes 220 us.
// Every wait is bounded: on a time-out the CTA raises its abort flag and the other roles leave; the epilogue stops waiting
// and runs out its items, so that the scores it writes from then on are void (the status word of the step says so).
// Then the tensor memory is freed.
#pragma once
#include "tc.cuh"

constexpr int kItKeys = 128, kItCols = 256;
constexpr int kItProd = 4;
constexpr int kItThreads = (kItProd + 9) * 32;
constexpr int kItKSub = kItKeys * 128;               // 64 dims of 128 keys
constexpr int kItQSub = kItCols * 128;               // 64 dims of 256 (row, head) pairs
constexpr int kItSmem = 2 * 2 * kItKSub + 2 * 2 * kItQSub + 1024 + 256 + 2 * kItCols * 4 + 2 * 32 * 4;

__device__ __forceinline__ uint32_t it_sw128(int row, int colb) {
  return (uint32_t)(row * 128 + ((((colb >> 4) ^ (row & 7)) << 4) | (colb & 15)));
}
// two packed e2m1 values (low nibble first) -> f16x2, exact
__device__ __forceinline__ uint32_t e2m1x2_to_h2(uint32_t byte) {
  uint32_t r;
  asm("{\n\t.reg .b8 b, z0, z1, z2;\n\tmov.b32 {b, z0, z1, z2}, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, b;\n\t}" : "=r"(r) : "r"(byte));
  return r;
}
__device__ __forceinline__ uint32_t it_pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// row0, row count and key tiles of work item `item`; every lane of the calling warp gets them
struct ItItem {
  int row0, nrows, key0, tiles, valid;               // tiles with a valid key; largest valid count of the rows
};

template <int HI>
__global__ void __launch_bounds__(kItThreads, 1) index_score_tc_kernel(ScoreParams p, int per, int items, TfStatusWord* st) {
  tf_pdl_sync();
  constexpr int DI = 128, RT = kItCols / HI;         // rows per tile
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - raw);
  const uint32_t q_s = base, k_s = base + 4 * kItQSub;
  uint8_t *q_g = aligned, *k_g = aligned + 4 * kItQSub;
  uint8_t* tail = k_g + 4 * kItKSub;
  const uint32_t bar0 = k_s + 4 * kItKSub;
  auto k_full = [&](int s) { return bar0 + 8u * s; };             // key tile written     (4 warps)
  auto k_empty = [&](int s) { return bar0 + 16u + 8u * s; };      // its MMAs are done    (commit)
  auto s_ready = [&](int s) { return bar0 + 32u + 8u * s; };      // accumulator ready    (commit)
  auto s_free = [&](int s) { return bar0 + 48u + 8u * s; };       // accumulator read     (8 warps)
  auto q_ready = [&](int s) { return bar0 + 64u + 8u * s; };      // Q tile written       (4 warps)
  auto q_free = [&](int s) { return bar0 + 80u + 8u * s; };       // the item's MMAs done (commit)
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail + 96);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 104);
  float* wtab = reinterpret_cast<float*>(tail + 256);             // [2][256] head weights of the item's rows

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(k_full(s), kItProd);
      tc::mbar_init(k_empty(s), 1);
      tc::mbar_init(s_ready(s), 1);
      tc::mbar_init(s_free(s), 8);
      tc::mbar_init(q_ready(s), kItProd);
      tc::mbar_init(q_free(s), 1);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == kItProd + 4) tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // Items go down the rows first: the CTAs running together read the same keys.  All warps walk the same
  // sequence and skip items without a valid key in the same way.
  const int row_tiles = (p.T + RT - 1) / RT;
  auto get = [&](int item) -> ItItem {
    ItItem it;
    const int seg = item / row_tiles;
    it.row0 = (item - seg * row_tiles) * RT;
    it.nrows = min(RT, p.T - it.row0);
    it.key0 = p.key_lo + seg * per * kItKeys;
    int v = 0;
    for (int i = lane; i < it.nrows; i += 32) v = max(v, p.nvalid[it.row0 + i]);
    it.valid = min(__reduce_max_sync(0xffffffffu, v), p.key_hi);
    it.tiles = max(0, min(per, (it.valid - it.key0 + kItKeys - 1) / kItKeys));
    return it;
  };

  if (warp < kItProd) {
    // ------------------------------------------------------------------ Q and key tiles
    int kt = 0, n_item = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const ItItem it = get(item);
      if (it.tiles == 0) continue;
      const int qb = n_item & 1;
      if (!(ok = tc::mbar_wait(q_free(qb), ((n_item >> 1) & 1) ^ 1, abort_flag))) break;
      __syncwarp();
      {
        const int live = it.nrows * HI;              // (row, head) pairs; 16 pieces of 16 bytes each
        const uint4* src = reinterpret_cast<const uint4*>(p.q + (long)it.row0 * HI * DI);
#pragma unroll 8
        for (int j = 0; j < kItCols * 16 / 128; ++j) {
          const int piece = threadIdx.x + 128 * j, c = piece >> 4, c16 = piece & 15;
          uint4 v = c < live ? __ldg(src + piece) : make_uint4(0u, 0u, 0u, 0u);
          uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&vw[e]));
            vw[e] = it_pack_h2(f.x, f.y);
          }
          *reinterpret_cast<uint4*>(q_g + (qb * 2 + (c16 >> 3)) * kItQSub + it_sw128(c, (c16 & 7) * 16)) = v;
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(q_ready(qb));
      }
      ++n_item;
      const uint8_t* kb = p.keys + (long)p.region[it.row0] * p.key_region_stride;
      const int key = threadIdx.x;
      uint32_t raw_k[DI / 8 + 1];
      auto load = [&](int t) {
        const int k = it.key0 + t * kItKeys + key;
        if (t < it.tiles && k < it.valid) {
          const uint32_t* row = reinterpret_cast<const uint32_t*>(kb + (long)k * p.key_row);
#pragma unroll
          for (int j = 0; j < DI / 8 + 1; ++j) raw_k[j] = __ldg(row + j);
        } else {
#pragma unroll
          for (int j = 0; j < DI / 8 + 1; ++j) raw_k[j] = 0u;
        }
      };
      load(0);
      for (int t = 0; t < it.tiles; ++t, ++kt) {
        const int s = kt & 1;
        if (!(ok = tc::mbar_wait(k_empty(s), ((kt >> 1) & 1) ^ 1, abort_flag))) break;
        uint8_t* dst = k_g + s * 2 * kItKSub;
        // Block scales of 2^-23 to 2^15 are f16 numbers, and an e2m1 value times one is rounded (or overflows) as in fp32
        // with a conversion behind it; outside of them the fp32 form is taken.
        uint32_t outside = 0;
#pragma unroll
        for (int blk = 0; blk < DI / 32; ++blk) outside |= ((raw_k[DI / 8] >> (8 * blk)) & 0xffu) - 104u > 38u;
        if (!outside) {
#pragma unroll
          for (int blk = 0; blk < DI / 32; ++blk) {
            const float sf = ue8m0_to_float((raw_k[DI / 8] >> (8 * blk)) & 0xffu);
            const __half2 s2 = __floats2half2_rn(sf, sf);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t o[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint32_t h = e2m1x2_to_h2(raw_k[blk * 4 + q] >> (8 * j));
                const __half2 v = __hmul2(*reinterpret_cast<__half2*>(&h), s2);
                o[j] = *reinterpret_cast<const uint32_t*>(&v);
              }
              const int d = blk * 32 + q * 8;
              *reinterpret_cast<uint4*>(dst + (d >> 6) * kItKSub + it_sw128(key, (d & 63) * 2)) =
                  make_uint4(o[0], o[1], o[2], o[3]);
            }
          }
        } else {
#pragma unroll
          for (int blk = 0; blk < DI / 32; ++blk) {
            // unpacked halves hold value * 2^-14: the block scale takes the 2^14 (in fp32: no overflow)
            const float s14 = ue8m0_to_float((raw_k[DI / 8] >> (8 * blk)) & 0xffu) * 16384.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t h4[4], o[4];
              e2m1x8_to_h2x4_scaled(raw_k[blk * 4 + q], h4);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 f = __half22float2(*reinterpret_cast<__half2*>(&h4[j]));
                o[j] = it_pack_h2(f.x * s14, f.y * s14);
              }
              const int d = blk * 32 + q * 8;
              *reinterpret_cast<uint4*>(dst + (d >> 6) * kItKSub + it_sw128(key, (d & 63) * 2)) =
                  make_uint4(o[0], o[1], o[2], o[3]);
            }
          }
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(k_full(s));
        load(t + 1);
      }
    }
  } else if (warp == kItProd + 4) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = tc::instr_desc(0, 0, 128, kItCols);
    int kt = 0, n_item = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const ItItem it = get(item);
      if (it.tiles == 0) continue;
      const int qb = n_item & 1;
      if (tc::elect_one()) {
        ok = tc::mbar_wait(q_ready(qb), (n_item >> 1) & 1, abort_flag);
        for (int t = 0; t < it.tiles && ok; ++t) {
          const int s = (kt + t) & 1;
          const uint32_t ph = ((kt + t) >> 1) & 1;
          if (!(ok = tc::mbar_wait(k_full(s), ph, abort_flag))) break;
          if (!(ok = tc::mbar_wait(s_free(s), ph ^ 1, abort_flag))) break;
          tc::tc_fence_after();
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tc::mma_f16(tmem_base + s * kItCols, tc::smem_desc_sw128(k_s + (s * 2 + j) * kItKSub) + 2 * k,
                          tc::smem_desc_sw128(q_s + (qb * 2 + j) * kItQSub) + 2 * k, idesc, (j | k) ? 1u : 0u);
          tc::mma_commit(k_empty(s));
          tc::mma_commit(s_ready(s));
        }
        if (ok) tc::mma_commit(q_free(qb));
      }
      ok = __all_sync(0xffffffffu, ok);
      kt += it.tiles;
      ++n_item;
    }
  } else {
    // ------------------------------------------------------------------ epilogue: one key and half of the rows per thread
    const int quad = warp & 3, half = warp > kItProd + 4;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const int et = quad * 32 + lane;
    int kt = 0, n_item = 0;
    bool fail = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      if (!fail && !tc::mbar_wait(bar, parity, abort_flag)) fail = true;
      __syncwarp();
    };
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int c0 = half * 128 + et, i_row0 = item % row_tiles * RT, i_rows = min(RT, p.T - i_row0);
      const float wv = c0 < i_rows * HI ? p.w[(long)i_row0 * HI + c0] : 0.f;       // (on their way with the item's limits)
      const int nvv = c0 < i_rows ? p.nvalid[i_row0 + c0] : 0;
      const ItItem it = get(item);
      const int seg_end = min(it.key0 + per * kItKeys, min(p.key_hi, p.lds));
      // columns of the segment past the last tile with a valid key
      for (int r = half; r < it.nrows; r += 2)
        for (int k = it.key0 + it.tiles * kItKeys + et; k < seg_end; k += 128)
          p.scores[(long)(it.row0 + r) * p.lds + k] = -INFINITY;
      if (it.tiles == 0) continue;
      float* wt = wtab + (n_item & 1) * kItCols;
      int* nv = reinterpret_cast<int*>(wtab + 2 * kItCols) + (n_item & 1) * 32;      // valid keys of the rows
      wt[c0] = wv;
      if (c0 < RT) nv[c0] = nvv;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      ++n_item;
      for (int t = 0; t < it.tiles; ++t, ++kt) {
        const int s = kt & 1, k = it.key0 + t * kItKeys + et;
        const bool in = k < seg_end;
        wait(s_ready(s), (kt >> 1) & 1);
        tc::tc_fence_after();
        const uint32_t taddr = tmem_base + lane_off + s * kItCols + half * 128;
        float* out = p.scores + (long)(it.row0 + half * (RT / 2)) * p.lds + k;
        float acc = 0.f;
        uint32_t next[32];
        tc::tmem_ld32(taddr, next);
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          // the next 32 columns are on their way while these are summed
          uint32_t v[32];
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            asm volatile("" : "+r"(next[i]));          // not read ahead of the wait
            v[i] = next[i];
          }
          if (q < 3) {
            tc::tmem_ld32(taddr + (q + 1) * 32, next);
          } else {
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(s_free(s));
          }
          // The sums of all rows before the first store: a branch behind every row left each row's loads, sums and store
          // in one chain.
          constexpr int HG = HI < 32 ? HI : 32, G = 32 / HG;     // columns of one row inside a piece; rows of a piece
          float sum[G];
#pragma unroll
          for (int g = 0; g < G; ++g) {
            // four chains of eight terms at most: one chain over all heads rounds more (1.05e-7 of a score at 64 heads)
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
            for (int c = 0; c < HG; c += 4) {
              const float4 w4 = *reinterpret_cast<const float4*>(wt + half * 128 + q * 32 + g * HG + c);
              a0 = fmaf(fmaxf(__uint_as_float(v[g * HG + c]), 0.f), w4.x, a0);
              a1 = fmaf(fmaxf(__uint_as_float(v[g * HG + c + 1]), 0.f), w4.y, a1);
              a2 = fmaf(fmaxf(__uint_as_float(v[g * HG + c + 2]), 0.f), w4.z, a2);
              a3 = fmaf(fmaxf(__uint_as_float(v[g * HG + c + 3]), 0.f), w4.w, a3);
            }
            acc += (a0 + a1) + (a2 + a3);
            sum[g] = acc;
            if (HI <= 32) acc = 0.f;
          }
          if (HI <= 32 || (q & 1)) {                 // (64 heads: a row is two pieces)
            const int r0 = HI <= 32 ? q * G : q >> 1;            // among the rows of the half
#pragma unroll
            for (int g = 0; g < G; ++g) {
              const int r = half * (RT / 2) + r0 + g;
              if (in && r < it.nrows) out[(long)(r0 + g) * p.lds] = k < nv[r] ? sum[g] : -INFINITY;
            }
            acc = 0.f;
          }
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) tf_report(st, TF_TIMEOUT, 152, blockIdx.x, 0);
  if (warp == kItProd + 4) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, 512);
  }
}
