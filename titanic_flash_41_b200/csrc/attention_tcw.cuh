// Sparse attention of prefill rows on the tcgen05 tensor cores for 512-wide latent heads (up to 64 heads, one
// split).  Included by attention.cu inside its anonymous namespace, after attention_tc.cuh, whose row
// contract (sink, inverse rotation, finished rows) and role split it shares.
//
// A key row is 1 KB of f16, so the tiles of the narrow kernel do not fit: a chunk is 64 keys (64 KB, two in
// flight), Q is stored once (64 KB) and the second contraction is transposed, which uses all 128 rows of the MMA
// and leaves room in tensor memory for two S buffers:
//
//   S[head, key]    = Q[head, :] . K[key, :]         A = Q (64 rows; rows 64.. read what lies behind and only
//                                                     reach accumulator lanes nobody reads), B = key tile, K-major
//   O^T[dim, head] += sum_key K[key, dim] P[head, key]  A = the same tile MN-major, four blocks of 128 dims; B = P
//
//   warps 0-7   gather: four threads per key (128 dims each), the next chunk's bytes requested before this one
//               is converted
//   warps 8-11  warps 8, 9 softmax (one head per thread, stale reference maximum as in the narrow kernel);
//               all four own 32 lanes of O^T: they rescale it when the maximum moves (factors per
//               head through shared memory) and finish the row (neighbouring lanes hold a rotation pair)
//   warp 12     one thread issues the MMAs: QK of chunk c + 1 before PV of chunk c
//
// Shared memory would allow 2,300 cycles a chunk: with N = 64 an MMA step (128 x 64 x 16) reads 6 KB of operands, 48
// cycles at 128 bytes a cycle, for 32 cycles of math, and the gather writes 64 KB beside them.  Measured 7,000 - 8,000 (0.98 ms
// for 4,001 rows of 64 heads and up to 640 keys; tensor pipe 20 % active): bound by the chain of gather, QK, softmax and PV
// of the two chunks in flight.  The mma.sync kernel dequantised every key once per 16 heads and kept a
// transposed copy: 17.9 ms.
// Every wait is bounded as in the narrow kernel.
#pragma once

constexpr int kTwKeys = 64;
constexpr int kTwProd = 8;                          // gather warps: four threads per key
constexpr int kTwThreads = (kTwProd + 5) * 32;      // gather, 4 softmax / O^T, 1 MMA warp
constexpr int kTwSub = 8192;                        // [64 rows x 128 B]: 64 dims of the keys, of Q, or the keys of P
constexpr int kTwSubs = 8;                          // 512 dims
constexpr int kTwStage = kTwSubs * kTwSub;
constexpr int kTwQ = kTwSubs * kTwSub;
constexpr int kTwOps = kTwQ + 2 * kTwSub;           // Q, P x 2
constexpr int kTwSmem = kTwOps + 2 * kTwStage + 1024 + 1024;

// MN-major operand of 128-byte rows: next 64 columns one sub-tile further, next 8 k-rows 1,024 bytes
__device__ __forceinline__ uint64_t smem_desc_mn_w(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)(kTwSub >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__global__ void __launch_bounds__(kTwThreads, 1) sparse_attn_tcw_kernel(AttnParams p) {
  tf_pdl_sync();
  constexpr int DH = 512;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw0 = tc::smem_u32(smem_raw);
  const uint32_t base = (raw0 + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - raw0);
  const uint32_t q_s = base, p_s = base + kTwQ, st_s = base + kTwOps;
  uint8_t* q_g = aligned;
  uint8_t* p_g = aligned + kTwQ;
  uint8_t* st_g = aligned + kTwOps;
  const uint32_t bar0 = base + kTwOps + 2 * kTwStage;
  auto full = [&](int s) { return bar0 + 8u * s; };             // gather -> MMA             (8 warps)
  auto empty = [&](int s) { return bar0 + 8u * (2 + s); };      // PV done: stage free        (commit)
  auto s_ready = [&](int b) { return bar0 + 8u * (4 + b); };    // QK done                    (commit)
  auto s_free = [&](int b) { return bar0 + 8u * (6 + b); };     // softmax has read S         (2 warps)
  // the PV that read P[b] is done (commit); O is complete up to that chunk.  (A single barrier for "PV done" would be
  // ambiguous at the end of a row: while the PV before the last one still runs, the last one's parity is an older one's.)
  auto p_free = [&](int b) { return bar0 + 8u * (8 + b); };
  auto p_ready = [&](int b) { return bar0 + 8u * (10 + b); };   // P[b] written, O rescaled   (4 warps)
  const uint32_t o_free = bar0 + 96, q_ready = bar0 + 104, q_free = bar0 + 112;      // (4 warps), (8 warps), (commit)
  uint8_t* tail = st_g + 2 * kTwStage;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail + 128);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 136);
  volatile int* moved = reinterpret_cast<volatile int*>(tail + 144);       // [2 chunks][2 softmax warps]
  float* fac = reinterpret_cast<float*>(tail + 256);                       // [64] per-head factor
  float* fin = reinterpret_cast<float*>(tail + 512);                       // [64] per-head output scale

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(full(s), kTwProd);
      tc::mbar_init(empty(s), 1);
      tc::mbar_init(s_ready(s), 1);
      tc::mbar_init(s_free(s), 2);
      tc::mbar_init(p_ready(s), 4);
      tc::mbar_init(p_free(s), 1);
    }
    tc::mbar_init(o_free, 4);
    tc::mbar_init(q_ready, kTwProd);
    tc::mbar_init(q_free, 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == kTwProd + 4) tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS[2] = {tmem_base, tmem_base + 64u};
  const uint32_t tO = tmem_base + 128u;              // four blocks of 64 columns (heads), lane = dim of the block
  auto chunks_of = [&](int nkeys) { return max(1, (nkeys + kTwKeys - 1) / kTwKeys); };

  if (warp < kTwProd) {
    // ------------------------------------------------------------------ gather + convert
    const int key = threadIdx.x & (kTwKeys - 1), part = threadIdx.x >> 6;      // 128 dims of one key
    uint4 rawv[8];
    uint2 rsc;
    int it = 0, n_row = 0;
    bool ok = true;
    for (int r = blockIdx.x; r < p.T && ok; r += gridDim.x, ++n_row) {
      int nwin;
      const int nkeys = attn_row_keys(p, r, &nwin);
      const int nchunks = chunks_of(nkeys);
      const int pos = p.pos[r], reg = p.region[r];
      const uint8_t* win = p.win + (long)reg * p.win_region_stride;
      const uint8_t* comp = p.comp ? p.comp + (long)reg * p.comp_region_stride : nullptr;
      auto key_kind = [&](int c) -> int {             // 0 padding, 1 window slot, 2 compressed entry
        const int i = c * kTwKeys + key;
        return (c >= nchunks || i >= nkeys) ? 0 : (i < nwin ? 1 : 2);
      };
      auto key_val = [&](int c, int kind) -> int {
        const int i = c * kTwKeys + key;
        if (kind == 1) return (pos - nwin + 1 + i) % p.ring;
        if (kind == 2) return p.sel[(long)r * p.sel_stride + (i - nwin)];
        return 0;
      };
      auto load_raw = [&](int kind, int val) {
        if (kind == 1) {
          const uint8_t* row = win + (long)val * p.win_row;
#pragma unroll
          for (int j = 0; j < 8; ++j) rawv[j] = *reinterpret_cast<const uint4*>(row + part * 128 + j * 16);
          rsc.x = *reinterpret_cast<const uint32_t*>(row + DH + part * 4);           // one scale per 32 dims
        } else if (kind == 2) {
          int id = val;
          if (id < 0 || id >= p.maxC) {
            tf_report(p.st, TF_BAD_INDEX, 12, r, id);
            id = 0;
          }
          const uint8_t* row = comp + (long)id * p.comp_row;
#pragma unroll
          for (int j = 0; j < 4; ++j) rawv[j] = *reinterpret_cast<const uint4*>(row + part * 64 + j * 16);
          rsc = *reinterpret_cast<const uint2*>(row + DH / 2 + part * 8);            // one scale per 16 dims
        }
      };
      int kind_cur = key_kind(0), kind_next = key_kind(1);
      int val_cur = key_val(0, kind_cur), val_next = key_val(1, kind_next);
      load_raw(kind_cur, val_cur);
      // Q of this row, once the QK MMAs of the row before are done: 64 heads x 512 bf16 = 4,096 16-byte pieces
      if (!(ok = tc::mbar_wait(q_free, (n_row & 1) ^ 1, abort_flag))) break;
      {
        const uint4* qsrc = reinterpret_cast<const uint4*>(p.q + (long)r * p.Hl * DH);
#pragma unroll 4
        for (int j = 0; j < 16; ++j) {
          const int piece = (int)threadIdx.x + kTwProd * 32 * j;
          const int h = piece >> 6, c16 = piece & 63;           // 64 pieces per head row
          uint4 v = h < p.Hl ? qsrc[piece] : make_uint4(0u, 0u, 0u, 0u);
          uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
          for (int e = 0; e < 4; ++e) {                          // bf16 pair -> f16 pair (exact in range)
            const float2 f2 = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&vw[e]));
            vw[e] = pack_h2(f2.x, f2.y);
          }
          *reinterpret_cast<uint4*>(q_g + (c16 >> 3) * kTwSub + sw128(h, (c16 & 7) * 16)) = v;
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(q_ready);
      }
      for (int c = 0; c < nchunks; ++c, ++it) {
        const int s = it & 1;
        if (!(ok = tc::mbar_wait(empty(s), ((it >> 1) & 1) ^ 1, abort_flag))) break;
        uint8_t* kt = st_g + s * kTwStage + 2 * part * kTwSub;      // this thread's two sub-tiles
        auto put = [&](int seg, const uint32_t (&hv)[8]) {          // 16 dims = 32 bytes
          uint8_t* sub = kt + (seg >> 2) * kTwSub;
          const int cb = (seg & 3) * 32;
          *reinterpret_cast<uint4*>(sub + sw128(key, cb)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
          *reinterpret_cast<uint4*>(sub + sw128(key, cb + 16)) = make_uint4(hv[4], hv[5], hv[6], hv[7]);
        };
        if (kind_cur == 0) {
          const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
          for (int seg = 0; seg < 8; ++seg) put(seg, z);
        } else if (kind_cur == 1) {
#pragma unroll
          for (int seg = 0; seg < 8; ++seg) {
            uint32_t hv[8];
            const float sc = ue8m0_to_float((rsc.x >> (8 * (seg >> 1))) & 0xffu);
            const uint16_t* h = reinterpret_cast<const uint16_t*>(&rawv[seg]);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              uint32_t h2 = e4m3x2_to_h2(h[q]);
              const float2 v = __half22float2(*reinterpret_cast<__half2*>(&h2));
              hv[q] = pack_h2(v.x * sc, v.y * sc);
            }
            put(seg, hv);
          }
        } else {
          const __half2 k14 = __floats2half2_rn(16384.f, 16384.f);   // (the unpacked halves hold value * 2^-14)
#pragma unroll
          for (int seg = 0; seg < 8; ++seg) {
            uint32_t hv[8];
            const uint32_t sb = ((seg < 4 ? rsc.x : rsc.y) >> (8 * (seg & 3))) & 0xffu;
            const uint32_t sh = e4m3x2_to_h2((uint16_t)(sb | (sb << 8)));
            const __half2 sc2 = *reinterpret_cast<const __half2*>(&sh);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&rawv[seg >> 1]) + 2 * (seg & 1);
            e2m1x8_to_h2x4_scaled(w[0], hv);
            e2m1x8_to_h2x4_scaled(w[1], hv + 4);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const __half2 x = __hmul2(__hmul2(*reinterpret_cast<__half2*>(&hv[q]), k14), sc2);
              hv[q] = *reinterpret_cast<const uint32_t*>(&x);
            }
            put(seg, hv);
          }
        }
        kind_cur = kind_next;
        val_cur = val_next;
        load_raw(kind_cur, val_cur);
        kind_next = key_kind(c + 2);
        val_next = key_val(c + 2, kind_next);
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(full(s));
      }
    }
  } else if (warp == kTwProd + 4) {
    // ------------------------------------------------------------------ MMA issuer
    if (tc::elect_one()) {
      constexpr uint32_t idesc_qk = tc::instr_desc(0, 0, 128, 64);
      constexpr uint32_t idesc_pv = idesc_qk | (1u << 15);            // A (the key tile as V^T) MN-major
      int it = 0, n_row = 0;
      bool ok = true;
      auto qk = [&](int i) -> bool {
        const int s = i & 1;
        if (!tc::mbar_wait(full(s), (i >> 1) & 1, abort_flag)) return false;
        if (!tc::mbar_wait(s_free(s), ((i >> 1) & 1) ^ 1, abort_flag)) return false;
        tc::tc_fence_after();
#pragma unroll
        for (int j = 0; j < kTwSubs; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc::mma_f16(tS[s], tc::smem_desc_sw128(q_s + j * kTwSub) + 2 * k,
                        tc::smem_desc_sw128(st_s + s * kTwStage + j * kTwSub) + 2 * k, idesc_qk, (j | k) ? 1u : 0u);
        tc::mma_commit(s_ready(s));
        return true;
      };
      for (int r = blockIdx.x; r < p.T && ok; r += gridDim.x, ++n_row) {
        int nwin;
        const int nchunks = chunks_of(attn_row_keys(p, r, &nwin));
        if (!(ok = tc::mbar_wait(q_ready, n_row & 1, abort_flag))) break;
        if (!(ok = qk(it))) break;
        if (nchunks == 1) tc::mma_commit(q_free);
        for (int c = 0; c < nchunks; ++c, ++it) {
          if (c + 1 < nchunks) {
            if (!(ok = qk(it + 1))) break;
            if (c + 2 == nchunks) tc::mma_commit(q_free);
          }
          if (!(ok = tc::mbar_wait(p_ready(it & 1), (it >> 1) & 1, abort_flag))) break;
          if (c == 0 && !(ok = tc::mbar_wait(o_free, (n_row & 1) ^ 1, abort_flag))) break;
          tc::tc_fence_after();
          const uint32_t kt = st_s + (it & 1) * kTwStage;
          const uint64_t dp = tc::smem_desc_sw128(p_s + (it & 1) * kTwSub);
#pragma unroll
          for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tc::mma_f16(tO + 64 * b, smem_desc_mn_w(kt + 2 * b * kTwSub) + 128u * k, dp + 2 * k, idesc_pv,
                          (c | k) ? 1u : 0u);
          tc::mma_commit(empty(it & 1));
          tc::mma_commit(p_free(it & 1));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax (warps 8, 9), O^T (8-11)
    const int quad = warp - kTwProd;
    const bool sm = quad < 2;
    const int h = quad * 32 + lane;                   // head of a softmax thread
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    auto grp_bar = [&]() { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    // (after a time-out a warp stops waiting but keeps walking the named barriers with its partners)
    bool fail = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      if (!fail && !tc::mbar_wait(bar, parity, abort_flag)) fail = true;
      __syncwarp();
    };
    int it = 0, n_row = 0;
    for (int r = blockIdx.x; r < p.T; r += gridDim.x, ++n_row) {
      int nwin;
      const int nkeys = attn_row_keys(p, r, &nwin);
      const int nchunks = chunks_of(nkeys);
      float m = kNegBig, l = 0.f;
      for (int c = 0; c < nchunks; ++c, ++it) {
        const int sb = it & 1, valid = nkeys - c * kTwKeys;
        float cm = kNegBig, ls = 0.f;
        // exp2(s - m) of this thread's head into its row of P; cm = the chunk's largest score, ls = the sum
        auto expo = [&]() {
          cm = kNegBig;
          ls = 0.f;
          uint8_t* psub = p_g + sb * kTwSub;
#pragma unroll 1
          for (int q = 0; q < 2; ++q) {
            uint32_t v[32];
            tc::tmem_ld32(tS[sb] + lane_off + q * 32, v);
            tc::tmem_ld_wait();
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const bool in0 = q * 32 + 2 * i < valid, in1 = q * 32 + 2 * i + 1 < valid;
              const float x0 = in0 ? __uint_as_float(v[2 * i]) : kNegBig, x1 = in1 ? __uint_as_float(v[2 * i + 1]) : kNegBig;
              cm = fmaxf(cm, fmaxf(x0, x1));
              const float a = in0 ? exp2f(fmaf(x0, p.scale_log2, -m)) : 0.f;
              const float b = in1 ? exp2f(fmaf(x1, p.scale_log2, -m)) : 0.f;
              ls += a + b;
              pk[i] = pack_h2(a, b);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(psub + sw128(h, q * 64 + i * 16)) =
                  make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
          }
        };
        if (sm) {
          wait(s_ready(sb), (it >> 1) & 1);
          tc::tc_fence_after();
          if (c == 0) {
#pragma unroll 1
            for (int q = 0; q < 2; ++q) {
              uint32_t v[32];
              tc::tmem_ld32(tS[sb] + lane_off + q * 32, v);
              tc::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (q * 32 + i < valid) cm = fmaxf(cm, __uint_as_float(v[i]));
            }
            m = cm * p.scale_log2;
          }
          wait(p_free(sb), ((it >> 1) & 1) ^ 1);       // the PV that read this P buffer two chunks ago is done
          expo();
          const bool any = __any_sync(0xffffffffu, cm * p.scale_log2 > m + 8.f);
          if (lane == 0) moved[sb * 2 + quad] = any ? 1 : 0;
        }
        grp_bar();
        if (moved[sb * 2] | moved[sb * 2 + 1]) {
          // rare: the maximum moves; O^T columns (heads) are rescaled by all four warps
          if (sm) {
            const float nm = fmaxf(m, cm * p.scale_log2), f = exp2f(m - nm);
            m = nm;
            l *= f;
            fac[h] = f;
            expo();
          }
          grp_bar();
          if (c > 0) {
            wait(p_free((it - 1) & 1), ((it - 1) >> 1) & 1);        // the PV of the chunk before
            tc::tc_fence_after();
#pragma unroll 1
            for (int q = 0; q < 8; ++q) {
              uint32_t o[32];
              tc::tmem_ld32(tO + lane_off + q * 32, o);
              tc::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * fac[(q & 1) * 32 + i]);
              tmem_st32(tO + lane_off + q * 32, o);
            }
            tmem_st_wait_tc();
          }
        }
        l += ls;
        tc::tc_fence_before();
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (sm) tc::mbar_arrive(s_free(sb));
          tc::mbar_arrive(p_ready(sb));
        }
      }
      // ---- the row: sink as one more zero-valued logit, inverse rotation of the tail, f16 / bf16 row
      if (sm) {
        float scale_o = 0.f;
        if (l > 0.f) {
          const float lse = m + log2f(l);
          const float s2 = p.sink ? p.sink[min(h, p.Hl - 1)] * 1.4426950408889634f : kNegBig;
          const float mx = fmaxf(s2, lse);
          const float w = exp2f(lse - mx);
          scale_o = w / (w + (p.sink ? exp2f(s2 - mx) : 0.f)) / l;
        }
        fin[h] = scale_o;
      }
      grp_bar();
      wait(p_free((it - 1) & 1), ((it - 1) >> 1) & 1);              // the row's last PV
      tc::tc_fence_after();
      const int tail0 = DH - p.rope_dim, odd = lane & 1;
#pragma unroll 1
      for (int b = 0; b < 4; ++b) {
        const int d = b * 128 + quad * 32 + lane;
        float sn = 0.f, cs = 1.f;
        if (d >= tail0) {
          const float ang = (float)p.pos[r] * p.freqs[(d - tail0) >> 1];
          const double two_pi = 6.283185307179586476925286766559;
          sincosf((float)((double)ang - two_pi * floor((double)ang / two_pi)), &sn, &cs);
        }
        // an even lane finishes dims (d, d + 1) of head hh, its odd neighbour the same dims of head hh + 1
        const long orow = (long)r * p.ldo + (d & ~1);
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          uint32_t v[32];
          tc::tmem_ld32(tO + lane_off + b * 64 + q * 32, v);
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float own = __uint_as_float(odd ? v[i + 1] : v[i]);
            const float oth = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? v[i] : v[i + 1]), 1);
            const int hh = q * 32 + i + odd;
            const float sc = fin[hh];
            const float x = (odd ? oth : own) * sc, y = (odd ? own : oth) * sc;
            const float a = x * cs + y * sn, e = -x * sn + y * cs;       // angle -> -angle
            if (hh < p.Hl) {
              if (p.out16) *reinterpret_cast<uint32_t*>(p.out16 + orow + (long)hh * DH) = pack_h2(a, e);
              if (p.outb) *reinterpret_cast<uint32_t*>(p.outb + orow + (long)hh * DH) = pack_bf2(a, e);
            }
          }
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(o_free);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) tf_report(p.st, TF_TIMEOUT, 151, blockIdx.x, 0);
  if (warp == kTwProd + 4) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, 512);
  }
}
