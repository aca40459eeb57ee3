// Sparse attention of prefill rows on the tcgen05 tensor cores (head dim 128, up to 64 heads, one
// split).  Included by attention.cu inside its anonymous namespace (AttnParams, kNegBig).
//
// A persistent CTA takes one query row at a time.  All heads of the row read the same latent keys,
// so the heads are the M of both contractions and a chunk of 128 gathered keys is N of the first and
// K of the second:
//
//   S[head, key]  = Q[head, :] . K[key, :]        A = Q [ 64 x 128 dims]   B = key tile, K-major
//   O[head, dim] += P[head, key] * K[key, dim]     A = P [ 64 x 128 keys]   B = the same tile, MN-major
//                                                  (P in tensor memory, over the S it came from)
//
// Operands are f16 in shared memory with the 128-byte swizzle (two 64-column sub-tiles each): a latent
// value times its scale is exact in f16 (FP4 rows: five mantissa bits at most, FP8 rows: four), and
// Q is bf16 converted once per row.  The MMAs read 128 rows of A: rows 64.. lie in the shared memory behind
// and only reach accumulator lanes that nobody reads.
//
// Gather, softmax and MMAs of a chunk are chains of about the same length, so one CTA an SM with everything
// double-buffered took 2,540 cycles a chunk (388 us for 2,048 rows of 2,176 keys).  This form holds one Q, one
// S (and P) and one O and two key tiles, 81 KB of shared memory and 256 tensor-memory columns: two CTAs share an SM,
// and the chains of one row fill the waits of the other.  P as a tensor-memory operand takes a quarter of the
// MMAs' shared-memory reads away; with P in shared memory two CTAs gained nothing.  370 us; the one-CTA form, whose
// two softmax pairs need a P barrier per buffer to be sound, 400 - 412 us in the same run.
//
//   warps 0-3   gather: one thread per key of the chunk fetches its FP8 window row or FP4 compressed row (the next
//               chunk's bytes are requested when this one has been converted; ids are decoded a chunk after
//               they are loaded) and writes it as a row of the key tile; two tiles in flight
//   warps 4-5   softmax, one head per thread: base-2 online softmax with a stale reference maximum (O is
//               rescaled only when a score exceeds it by 2^8), P as f16 over the columns of S that have
//               been read; then the row: sink as an extra zero-valued logit, inverse
//               rotation of the tail, f16 / bf16 output
//   warp 6      one thread issues the MMAs: PV of chunk c and, once that is done, QK of chunk c + 1 (it overwrites S and P)
// Every mbarrier wait is bounded; on a time-out the CTA raises its abort flag, reports TF_TIMEOUT,
// frees its tensor memory and returns.
//
// Output: the finished rows, i.e. what the mma.sync kernel and attn_merge_kernel produce together with
// one split.
#pragma once
#include "tc.cuh"

constexpr int kTcKeys = 128;
constexpr int kTcProd = 4;                           // gather warps: one thread per key row
constexpr int kTcThreads = (kTcProd + 3) * 32;      // gather warps, 2 softmax warps, 1 MMA warp
constexpr int kTcSub = 16384;                       // one [128 rows x 128 B] sub-tile
constexpr int kTcHSub = 8192;                       // Q: 64 rows (the heads) of a sub-tile
constexpr int kTcStage = 2 * kTcSub;                // the key tile: two 64-dim sub-tiles of [128 keys x 128 B]
constexpr int kTcStages = 2;
constexpr int kTcOps = 2 * kTcHSub;                 // Q
constexpr int kTcSmem = kTcOps + kTcStages * kTcStage + 1024 + 256;

// byte offset of (row, byte column) inside a 128-byte-swizzled sub-tile
__device__ __forceinline__ uint32_t sw128(int row, int colb) {
  return (uint32_t)(row * 128 + ((((colb >> 4) ^ (row & 7)) << 4) | (colb & 15)));
}
__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t v[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
      "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
      "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t v[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: row i of A is lane i, two f16 per 32-bit column; ONE thread issues
__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// MN-major operand (the contiguous direction is M / N, here the 128 dims of a key row) in the same
// 128-byte-swizzled tile of 128-byte rows: 8 k-rows form a 1,024-byte group (stride offset), the
// second 64 columns live one sub-tile further (leading offset)
__device__ __forceinline__ uint64_t smem_desc_sw128_mn(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
  d |= (uint64_t)(kTcSub >> 4) << 16;              // leading byte offset: next 64 columns
  d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset: next 8 k-rows
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;                          // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ void tmem_st_wait_tc() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ int attn_row_keys(const AttnParams& p, int r, int* nwin_out) {
  const int pos = p.pos[r];
  const int nwin = min(pos + 1 - (p.min_pos ? p.min_pos[r] : 0), p.window);
  int nsel = 0;
  if (p.comp) {
    if (p.sel_count) nsel = p.sel_count[r];
    else {
      int lo = 0, hi = p.sel_stride;
      const int* s = p.sel + (long)r * p.sel_stride;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (s[mid] >= 0) lo = mid + 1; else hi = mid;
      }
      nsel = lo;
    }
  }
  *nwin_out = nwin;
  return nwin + nsel;
}

__global__ void __launch_bounds__(kTcThreads, 2) sparse_attn_tc_kernel(AttnParams p) {
  tf_pdl_sync();
  constexpr int DH = 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw0 = tc::smem_u32(smem_raw);
  const uint32_t base = (raw0 + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - raw0);
  const uint32_t q_s = base, st_s = base + kTcOps;
  uint8_t* q_g = aligned;
  uint8_t* st_g = aligned + kTcOps;
  const uint32_t bar0 = st_s + kTcStages * kTcStage;
  auto full = [&](int s) { return bar0 + 8u * s; };             // gather -> MMA             (4 warps)
  auto empty = [&](int s) { return bar0 + 16u + 8u * s; };      // PV done: stage free        (commit)
  const uint32_t s_ready = bar0 + 32;                           // QK done                    (commit)
  const uint32_t p_ready = bar0 + 48, o_ready = bar0 + 56;      // P written, O rescaled (2 warps); PV done (commit)
  const uint32_t o_free = bar0 + 64;                            // the row has been read from O (2 warps)
  const uint32_t q_ready = bar0 + 72, q_free = bar0 + 80;       // Q written (4 warps); the row's QK MMAs are done (commit)
  uint8_t* tail = st_g + kTcStages * kTcStage;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail + 96);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 104);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      tc::mbar_init(full(s), kTcProd);
      tc::mbar_init(empty(s), 1);
    }
    tc::mbar_init(s_ready, 1);
    tc::mbar_init(p_ready, 2);
    tc::mbar_init(o_ready, 1);
    tc::mbar_init(o_free, 2);
    tc::mbar_init(q_ready, kTcProd);
    tc::mbar_init(q_free, 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == kTcProd + 2) tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), 256);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tS = *tmem_slot, tO = tS + 128u;
  auto chunks_of = [&](int nkeys) { return max(1, (nkeys + kTcKeys - 1) / kTcKeys); };

  if (warp < kTcProd) {
    // ------------------------------------------------------------------ gather + convert
    const int key = threadIdx.x;
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
      // A key is (kind, value): kind 0 = padding, 1 = window ring slot, 2 = compressed entry id.  The
      // id is only looked at when its row is fetched, a chunk later: nothing waits for the id load.
      auto key_kind = [&](int c) -> int {
        const int i = c * kTcKeys + key;
        return (c >= nchunks || i >= nkeys) ? 0 : (i < nwin ? 1 : 2);
      };
      auto key_val = [&](int c, int kind) -> int {
        const int i = c * kTcKeys + key;
        if (kind == 1) return (pos - nwin + 1 + i) % p.ring;
        if (kind == 2) return p.sel[(long)r * p.sel_stride + (i - nwin)];
        return 0;
      };
      auto load_raw = [&](int kind, int val) {
        if (kind == 1) {
          const uint8_t* row = win + (long)val * p.win_row;
#pragma unroll
          for (int j = 0; j < 8; ++j) rawv[j] = *reinterpret_cast<const uint4*>(row + j * 16);
          rsc.x = *reinterpret_cast<const uint32_t*>(row + DH);               // one scale per 32 dims
        } else if (kind == 2) {
          int id = val;
          if (id < 0 || id >= p.maxC) {
            tf_report(p.st, TF_BAD_INDEX, 11, r, id);
            id = 0;
          }
          const uint8_t* row = comp + (long)id * p.comp_row;
#pragma unroll
          for (int j = 0; j < 4; ++j) rawv[j] = *reinterpret_cast<const uint4*>(row + j * 16);
          rsc = *reinterpret_cast<const uint2*>(row + DH / 2);                // one scale per 16 dims
        }
      };
      int kind_cur = key_kind(0), kind_next = key_kind(1);
      int val_cur = key_val(0, kind_cur), val_next = key_val(1, kind_next);
      load_raw(kind_cur, val_cur);
      // Q of this row, once the QK MMAs of the row before are done: 64 heads x 128 bf16 = 1,024 16-byte pieces
      if (!(ok = tc::mbar_wait(q_free, (n_row & 1) ^ 1, abort_flag))) break;
      {
        const uint4* qsrc = reinterpret_cast<const uint4*>(p.q + (long)r * p.Hl * DH);
#pragma unroll 4
        for (int j = 0; j < 1024 / (kTcProd * 32); ++j) {
          const int piece = (int)threadIdx.x + kTcProd * 32 * j;
          const int h = piece >> 4, c16 = piece & 15;           // 16 pieces per head row
          uint4 v = h < p.Hl ? qsrc[piece] : make_uint4(0u, 0u, 0u, 0u);
          uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
          for (int e = 0; e < 4; ++e) {                          // bf16 pair -> f16 pair (exact in range)
            const float2 f2 = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&vw[e]));
            vw[e] = pack_h2(f2.x, f2.y);
          }
          *reinterpret_cast<uint4*>(q_g + (c16 >> 3) * kTcHSub + sw128(h, (c16 & 7) * 16)) = v;
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(q_ready);
      }
      for (int c = 0; c < nchunks; ++c, ++it) {
        const int s = it & 1;
        if (!(ok = tc::mbar_wait(empty(s), ((it >> 1) & 1) ^ 1, abort_flag))) break;
        uint8_t* kt = st_g + s * kTcStage;
        // The key row as f16, sixteen values = one 32-byte piece at a time.  One branch per row kind, not per
        // piece: the FP4 body (all but the window rows) stays small.
        auto put = [&](int seg, const uint32_t (&hv)[8]) {
          uint8_t* ksub = kt + (seg >> 2) * kTcSub;
          *reinterpret_cast<uint4*>(ksub + sw128(key, (seg & 3) * 32)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
          *reinterpret_cast<uint4*>(ksub + sw128(key, (seg & 3) * 32 + 16)) = make_uint4(hv[4], hv[5], hv[6], hv[7]);
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
          // the unpacked halves hold value * 2^-14; two packed f16 multiplies (by 2^14, exact, then by
          // the group's e4m3 scale, exact) instead of a trip through fp32 and back
          const __half2 k14 = __floats2half2_rn(16384.f, 16384.f);
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
        // request the next chunk's rows and the ids of the chunk after it, then hand the stage over
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
  } else if (warp == kTcProd + 2) {
    // ------------------------------------------------------------------ MMA issuer
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::instr_desc(0, 0, 128, 128);      // f16 x f16, M 128, N 128, both K-major
      constexpr uint32_t idesc_pv = idesc | (1u << 16);               // B (the key tile as V) MN-major
      int it = 0, n_row = 0;
      bool ok = true;
      auto qk = [&](int i) -> bool {                                  // S = Q . Kt(stage i & 1)^T
        const int s = i & 1;
        if (!tc::mbar_wait(full(s), (i >> 1) & 1, abort_flag)) return false;
        // S lies over the P that the PV before reads: MMAs with different accumulators are not ordered among
        // themselves, so that PV has to be done, not only issued
        if (i > 0 && !tc::mbar_wait(o_ready, (i & 1) ^ 1, abort_flag)) return false;
        tc::tc_fence_after();
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc::mma_f16(tS, tc::smem_desc_sw128(q_s + j * kTcHSub) + 2 * k,
                        tc::smem_desc_sw128(st_s + s * kTcStage + j * kTcSub) + 2 * k, idesc, (j | k) ? 1u : 0u);
        tc::mma_commit(s_ready);
        return true;
      };
      for (int r = blockIdx.x; r < p.T && ok; r += gridDim.x, ++n_row) {
        int nwin;
        const int nchunks = chunks_of(attn_row_keys(p, r, &nwin));
        if (!(ok = tc::mbar_wait(q_ready, n_row & 1, abort_flag))) break;
        if (!(ok = qk(it))) break;
        if (nchunks == 1) tc::mma_commit(q_free);
        for (int c = 0; c < nchunks; ++c, ++it) {
          if (!(ok = tc::mbar_wait(p_ready, it & 1, abort_flag))) break;
          // the first PV of a row overwrites O: the row before must have been read
          if (c == 0 && !(ok = tc::mbar_wait(o_free, (n_row & 1) ^ 1, abort_flag))) break;
          tc::tc_fence_after();
          // B = the same key tile read MN-major (dims contiguous): 16 keys per step = 2,048 bytes, 8 columns of P
          const uint64_t dv = smem_desc_sw128_mn(st_s + (it & 1) * kTcStage);
#pragma unroll
          for (int k = 0; k < 8; ++k) mma_f16_ts(tO, tS + 8u * k, dv + 128u * k, idesc_pv, (c | k) ? 1u : 0u);
          tc::mma_commit(empty(it & 1));
          tc::mma_commit(o_ready);
          if (c + 1 < nchunks) {
            if (!(ok = qk(it + 1))) break;
            if (c + 2 == nchunks) tc::mma_commit(q_free);      // the row's last QK is issued
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: one head per thread
    const int quad = warp - kTcProd, h = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    // (after a time-out the warp stops waiting and runs out its loop: the launch's result is void)
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
        const int valid = nkeys - c * kTcKeys;           // columns >= valid are padding
        wait(s_ready, it & 1);
        tc::tc_fence_after();
        // The reference maximum m is the first chunk's; it moves only when some head finds a score
        // more than 2^8 above it (then O and l are rescaled).  Until then exp2(s - m) <= 256 is harmless in
        // f16 / fp32 and the ratio O / l does not depend on m.
        float c0 = kNegBig, c1 = kNegBig;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t v[32];
          tc::tmem_ld32(tS + lane_off + q * 32, v);
          tc::tmem_ld_wait();
          if (valid < kTcKeys) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (q * 32 + i >= valid) v[i] = __float_as_uint(kNegBig);
          }
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            c0 = fmaxf(c0, __uint_as_float(v[i]));
            c1 = fmaxf(c1, __uint_as_float(v[i + 1]));
          }
        }
        const float cm = fmaxf(c0, c1) * p.scale_log2;
        if (c == 0) {
          m = cm;
        } else if (__any_sync(0xffffffffu, cm > m + 8.f)) {
          // (QK of this chunk was issued when the PV before was done: O is complete)
          const float nm = fmaxf(m, cm), f = exp2f(m - nm);
          m = nm;
          l *= f;
          wait(o_ready, (it & 1) ^ 1);
          tc::tc_fence_after();
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            uint32_t o[32];
            tc::tmem_ld32(tO + lane_off + q * 32, o);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st32(tO + lane_off + q * 32, o);
          }
        }
        float l0 = 0.f, l1 = 0.f;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          uint32_t v[32];
          tc::tmem_ld32(tS + lane_off + q * 32, v);
          tc::tmem_ld_wait();
          if (valid < kTcKeys) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (q * 32 + i >= valid) v[i] = __float_as_uint(-INFINITY);
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a = exp2f(fmaf(__uint_as_float(v[2 * i]), p.scale_log2, -m));
            const float b = exp2f(fmaf(__uint_as_float(v[2 * i + 1]), p.scale_log2, -m));
            l0 += a;
            l1 += b;
            pk[i] = pack_h2(a, b);
          }
          tmem_st16(tS + lane_off + q * 16, pk);           // columns of S read by now
        }
        l += l0 + l1;
        tmem_st_wait_tc();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(p_ready);
      }
      // ---- the row: the sink is one more logit with a zero value: scaled by w / (w + w_sink) as the split merge
      // would.  Then the inverse rotation of the tail (the value shares the key's rotated latent) and
      // the f16 / bf16 row.  Lane j holds the sine and cosine of pair j of the tail.
      wait(o_ready, (it & 1) ^ 1);
      tc::tc_fence_after();
      float scale_o = 0.f;
      if (l > 0.f) {
        const float lse = m + log2f(l);
        const float s2 = p.sink ? p.sink[min(h, p.Hl - 1)] * 1.4426950408889634f : kNegBig;
        const float mx = fmaxf(s2, lse);
        const float w = exp2f(lse - mx);
        scale_o = w / (w + (p.sink ? exp2f(s2 - mx) : 0.f)) / l;
      }
      float sn = 0.f, cs = 1.f;
      if (lane < p.rope_dim / 2) {
        const float ang = (float)p.pos[r] * p.freqs[lane];
        const double two_pi = 6.283185307179586476925286766559;
        sincosf((float)((double)ang - two_pi * floor((double)ang / two_pi)), &sn, &cs);
      }
      const int tail0 = DH - p.rope_dim;
      const long orow = (long)r * p.ldo + (long)h * DH;
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        uint32_t v[32];
        tc::tmem_ld32(tO + lane_off + q * 32, v);
        tc::tmem_ld_wait();
        float o[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = __uint_as_float(v[i]) * scale_o;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const int d = q * 32 + i;
          const int j = (d - tail0) >> 1;                       // pair of the tail (uniform over the warp)
          const float sj = __shfl_sync(0xffffffffu, sn, j & 31), cj = __shfl_sync(0xffffffffu, cs, j & 31);
          if (d >= tail0) {
            const float a = o[i], b2 = o[i + 1];
            o[i] = a * cj + b2 * sj;                            // inverse rotation: angle -> -angle
            o[i + 1] = -a * sj + b2 * cj;
          }
        }
        if (h < p.Hl) {
          if (p.out16) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(p.out16 + orow + q * 32 + 8 * i) =
                  make_uint4(pack_h2(o[8 * i], o[8 * i + 1]), pack_h2(o[8 * i + 2], o[8 * i + 3]),
                             pack_h2(o[8 * i + 4], o[8 * i + 5]), pack_h2(o[8 * i + 6], o[8 * i + 7]));
          }
          if (p.outb) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(p.outb + orow + q * 32 + 8 * i) =
                  make_uint4(pack_bf2(o[8 * i], o[8 * i + 1]), pack_bf2(o[8 * i + 2], o[8 * i + 3]),
                             pack_bf2(o[8 * i + 4], o[8 * i + 5]), pack_bf2(o[8 * i + 6], o[8 * i + 7]));
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
  if (*abort_flag && threadIdx.x == 0) tf_report(p.st, TF_TIMEOUT, 150, blockIdx.x, 0);
  if (warp == kTcProd + 2) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tS, 256);
  }
}
