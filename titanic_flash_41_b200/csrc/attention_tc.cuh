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
// Q is bf16 converted once per row.  An MMA of 64 rows takes as long as one of 128 (64 cycles at N = 128, K = 16), so the
// heads are there twice: rows 64.. repeat them, and each copy does the softmax of 64 of a chunk's 128 keys.  That
// makes four softmax warps, one on each scheduler, out of two that shared two of them (128 exponentials a thread
// and chunk on one unit were 1,024 cycles, as long as the chunk's MMAs).  P holds zeros for the keys of the other copy, so
// lanes 0..63 of O are the sums over half of the keys, lanes 64.. over the other half; the row's end adds them.
//
// One Q, one S (and P over it) and one O, two key tiles, 108 KB of shared memory and 256 tensor-memory columns: two CTAs
// share an SM, and the chains of one row fill the waits of the other.  P as a tensor-memory operand takes a quarter of the
// MMAs' shared-memory reads away.
// 2,048 rows of 2,176 keys: 305 us; two softmax warps, one thread per key row, the row's end in the softmax warps: 346 (the MMAs
// alone: 130).  Inside a long prefill the clock follows the power limit (1.5 - 1.65 of 1.97 GHz) and the gain is smaller: four
// launches of 16,384 rows 8.4 -> 7.3 ms.  What bounds it now is the issue of 146 M warp instructions (a third of them the gather's
// conversion) at half of the slots, with scoreboard waits between; the tensor pipe is active half of the time.
//
//   warps 0-7   gather: four threads per key of the chunk fetch its FP8 window row or FP4 compressed row (the next
//               chunk's bytes are requested when this one has been converted; ids are decoded a chunk after
//               they are loaded) and write it as a row of the key tile; two tiles in flight.  Behind the first chunks
//               of a row they finish the row before: the halves exchange dims through shared memory (each finishes
//               64 of the 128), sink, inverse rotation of the tail, f16 / bf16 output
//   warps 8-11  softmax, one (head, half of the keys) per thread, its 64 scores in registers: base-2 online softmax
//               with a stale reference maximum (O is rescaled only when a score exceeds it by 2^8); they also write
//               the next row's Q while the last PV runs
//               One thread of warp 8 issues the MMAs: PV of chunk c and, once that is done, QK of chunk c + 1 (it
//               overwrites S and P).  The kernel is launched with 80 registers a thread; the gather gives up 16 (64), the
//               softmax takes 32 (112) for its scores and probabilities.
// Every mbarrier wait is bounded; on a time-out the CTA raises its abort flag, reports TF_TIMEOUT,
// frees its tensor memory and returns.
//
// Output: the finished rows, i.e. what the mma.sync kernel and attn_merge_kernel produce together with
// one split.
#pragma once
#include "tc.cuh"

constexpr int kTcKeys = 128;
constexpr int kTcProd = 8;                           // gather warps: four threads per key row
constexpr int kTcThreads = (kTcProd + 4) * 32;      // gather warps, softmax warps
constexpr int kTcGatherRegs = 64, kTcSoftmaxRegs = 112;       // of 80 a thread at launch: 2 x 64 + 112 = 3 x 80
constexpr int kTcSub = 16384;                       // one [128 rows x 128 B] sub-tile
constexpr int kTcStage = 2 * kTcSub;                // the key tile: two 64-dim sub-tiles of [128 keys x 128 B]
constexpr int kTcStages = 2;
constexpr int kTcOps = 2 * kTcSub;                  // Q, twice
constexpr int kTcMerge = 2048 + 512 + 2 * 4096;     // (maximum, sum) of each half, rotation, two rows; two times 8 dims of 64 heads each way
constexpr int kTcSmem = kTcOps + kTcStages * kTcStage + kTcMerge + 1024 + 256;

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
__device__ __forceinline__ void tmem_ld8_tc(uint32_t taddr, uint32_t v[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8_tc(uint32_t taddr, const uint32_t v[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
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
// two packed e2m1 values (low nibble first) -> f16x2, exact
__device__ __forceinline__ uint32_t e2m1x2_to_h2(uint32_t byte) {
  uint32_t r;
  asm("{\n\t.reg .b8 b, z0, z1, z2;\n\tmov.b32 {b, z0, z1, z2}, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, b;\n\t}" : "=r"(r) : "r"(byte));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
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

// What a role needs to know about a row, loaded a row ahead: nothing waits for these loads
struct RowMeta {
  int pos, min_pos, count, region;
};
__device__ __forceinline__ RowMeta row_meta(const AttnParams& p, int r) {
  RowMeta m = {0, 0, 0, 0};
  if (r >= p.T) return m;
  m.pos = p.pos[r];
  m.region = p.region[r];
  if (p.min_pos) m.min_pos = p.min_pos[r];
  if (p.comp && p.sel_count) m.count = p.sel_count[r];
  return m;
}
__device__ __forceinline__ int row_keys(const AttnParams& p, const RowMeta& m, int r, int* nwin_out) {
  if (p.comp && !p.sel_count) return attn_row_keys(p, r, nwin_out);
  *nwin_out = min(m.pos + 1 - m.min_pos, p.window);
  return *nwin_out + m.count;
}

// A finished row, by the eight gather warps (their tensor-memory lanes, warp % 4, are those of the softmax warps; warps 0-3
// take the first 32 dims of each half, 4-7 the others): both halves brought to one maximum; the sink is one more logit with
// a zero value: scaled by w / (w + w_sink) as the split merge would.  Then the inverse rotation of the tail (the value shares
// the key's rotated latent) and the f16 / bf16 row.  Lane j holds the sine and cosine of pair j of the tail (`rot`).
// The softmax warps are a chunk into the next row meanwhile: done by them, this was a fifth of their time.
// Four warps meet at an mbarrier (eight times a row): unlike bar.sync it has a bounded wait, should one of them have given up.
__device__ __forceinline__ bool finish_row(const AttnParams& p, int r, int warp, int lane, uint32_t tO, const float2* stat, const float2* rot,
                                           float* xch, uint32_t o_free, uint32_t meet, volatile int* abort_flag) {
  constexpr int DH = 128;
  const int quad = warp & 3, set = warp >> 2, hi = quad >> 1, h = (quad & 1) * 32 + lane;
  const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
  meet += 8u * set;
  xch += set * 1024;
  uint32_t met = 0;
  auto gather_sync = [&]() -> bool {
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(meet);
    return tc::mbar_wait(meet, met++ & 1, abort_flag);
  };
  const float2 own = stat[hi * 64 + h], other = stat[(hi ^ 1) * 64 + h];
  const float top = fmaxf(own.x, other.x);
  float f_own = exp2f(own.x - top), f_other = exp2f(other.x - top);
  const float l = hi ? fmaf(other.y, f_other, own.y * f_own) : fmaf(own.y, f_own, other.y * f_other);   // the same bits in both
  float scale_o = 0.f;
  if (l > 0.f) {
    const float lse = top + log2f(l);
    const float s2 = p.sink ? p.sink[min(h, p.Hl - 1)] * 1.4426950408889634f : kNegBig;
    const float mx = fmaxf(s2, lse);
    const float w = exp2f(lse - mx);
    scale_o = w / (w + (p.sink ? exp2f(s2 - mx) : 0.f)) / l;
  }
  f_own *= scale_o;
  f_other *= scale_o;
  const float sn = rot[lane].x, cs = rot[lane].y;
  const int tail0 = DH - p.rope_dim;
  const long orow = (long)r * p.ldo + (long)h * DH;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    // eight dims for the other half's threads, eight of their own finished here
    const int d0 = hi * 64 + set * 32 + q * 8;
    uint32_t give[8], keep[8];
    tmem_ld8_tc(tO + lane_off + (d0 ^ 64), give);
    tmem_ld8_tc(tO + lane_off + d0, keep);
    tc::tmem_ld_wait();
    if (q == 3) {                                             // O has been read
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(o_free);
    }
    if (q && !gather_sync()) return false;                    // the pieces before have been taken
#pragma unroll
    for (int i = 0; i < 8; ++i) xch[(hi ^ 1) * 512 + i * 64 + h] = __uint_as_float(give[i]);
    if (!gather_sync()) return false;
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = fmaf(__uint_as_float(keep[i]), f_own, xch[hi * 512 + i * 64 + h] * f_other);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const int d = d0 + i;
      const int j = (d - tail0) >> 1;                         // pair of the tail (uniform over the warp)
      const float sj = __shfl_sync(0xffffffffu, sn, j & 31), cj = __shfl_sync(0xffffffffu, cs, j & 31);
      if (d >= tail0) {
        const float a = o[i], b2 = o[i + 1];
        o[i] = a * cj + b2 * sj;                              // inverse rotation: angle -> -angle
        o[i + 1] = -a * sj + b2 * cj;
      }
    }
    if (h < p.Hl) {
      if (p.out16)
        *reinterpret_cast<uint4*>(p.out16 + orow + d0) =
            make_uint4(pack_h2(o[0], o[1]), pack_h2(o[2], o[3]), pack_h2(o[4], o[5]), pack_h2(o[6], o[7]));
      if (p.outb)
        *reinterpret_cast<uint4*>(p.outb + orow + d0) =
            make_uint4(pack_bf2(o[0], o[1]), pack_bf2(o[2], o[3]), pack_bf2(o[4], o[5]), pack_bf2(o[6], o[7]));
    }
  }
  return gather_sync();                                       // (the next row's first pieces)
}

__global__ void __launch_bounds__(kTcThreads, 2) sparse_attn_tc_kernel(const __grid_constant__ AttnParams p) {
  tf_pdl_sync();
  constexpr int DH = 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw0 = tc::smem_u32(smem_raw);
  const uint32_t base = (raw0 + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - raw0);
  const uint32_t q_s = base, st_s = base + kTcOps;
  uint8_t* q_g = aligned;
  uint8_t* st_g = aligned + kTcOps;
  float2* stat = reinterpret_cast<float2*>(st_g + kTcStages * kTcStage);     // [row parity][half][64 heads]: maximum, sum
  float2* rot = reinterpret_cast<float2*>(st_g + kTcStages * kTcStage + 2048);      // [row parity][32 pairs]: sine, cosine
  float* xch = reinterpret_cast<float*>(st_g + kTcStages * kTcStage + 2048 + 512);  // [set of warps][half of the reader][8 dims][64 heads]
  const uint32_t bar0 = st_s + kTcStages * kTcStage + kTcMerge;
  auto full = [&](int s) { return bar0 + 8u * s; };             // gather -> MMA             (8 warps)
  auto empty = [&](int s) { return bar0 + 16u + 8u * s; };      // PV done: stage free        (commit)
  const uint32_t s_ready = bar0 + 32;                           // QK done                    (commit)
  const uint32_t p_ready = bar0 + 48, o_ready = bar0 + 56;      // P written, O rescaled (4 warps); PV done (commit)
  const uint32_t o_free = bar0 + 64;                            // the row has been read from O (8 gather warps)
  const uint32_t q_ready = bar0 + 72;                           // Q written (4 warps)
  const uint32_t l_ready = bar0 + 88;                           // + 8 (row & 1): its maxima and sums are written (4 softmax warps)
  const uint32_t meet = bar0 + 104;                             // + 8 (warp / 4): the gather warps while they finish a row
  uint8_t* tail = st_g + kTcStages * kTcStage + kTcMerge;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail + 120);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 124);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      tc::mbar_init(full(s), kTcProd);
      tc::mbar_init(empty(s), 1);
    }
    tc::mbar_init(s_ready, 1);
    tc::mbar_init(p_ready, 4);
    tc::mbar_init(o_ready, 1);
    tc::mbar_init(o_free, kTcProd);
    tc::mbar_init(q_ready, 4);
    tc::mbar_init(l_ready, 4);
    tc::mbar_init(l_ready + 8, 4);
    tc::mbar_init(meet, 4);
    tc::mbar_init(meet + 8, 4);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == kTcProd) tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), 256);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tS = *tmem_slot, tO = tS + 128u;
  auto chunks_of = [&](int nkeys) { return max(1, (nkeys + kTcKeys - 1) / kTcKeys); };

  if (warp < kTcProd) {
    // ------------------------------------------------------------------ gather + convert
    // Four lanes share a key row, a lane takes 32 of its dims: a warp's load touches eight rows.  (One thread per row touched
    // 32 lines with every load.)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcGatherRegs));
    const int key0 = warp * 16 + (lane >> 2), piece = lane & 3;          // keys key0 and key0 + 8
    uint4 rawv[2];
    uint32_t rsc[2];
    int val_cur[2], val_next[2];
    int it = 0, n_row = 0;
    bool ok = true;
    int last_r = -1, last_it = 0;                // the row before, not yet finished, and its last chunk
    RowMeta meta = row_meta(p, blockIdx.x);
    for (int r = blockIdx.x; ok; r += gridDim.x, ++n_row) {
      const bool live = r < p.T;
      if (!live && last_r < 0) break;
      int nwin = 0;
      const int nkeys = live ? row_keys(p, meta, r, &nwin) : 0;
      const int nchunks = chunks_of(nkeys);
      const int pos = meta.pos, reg = meta.region;
      meta = row_meta(p, r + gridDim.x);
      const uint8_t* win = p.win + (long)reg * p.win_region_stride;
      const uint8_t* comp = p.comp ? p.comp + (long)reg * p.comp_region_stride : nullptr;
      const int* sel = p.sel + (long)r * p.sel_stride - nwin;
      // Kind of key k of the row: 0 = padding, 1 = window ring slot, 2 = compressed entry, whose id is only looked at when
      // its row is fetched, a chunk later: nothing waits for the id load.
      auto kind = [&](int k) -> int { return k >= nkeys ? 0 : (k < nwin ? 1 : 2); };
      // (both loads without a condition per key: a predicated load is merged with the register's old value, that is, waited for)
      const bool has_sel = nkeys > nwin;
      auto load_val = [&](int c, int (&val)[2]) {
        if (has_sel) {
#pragma unroll
          for (int i = 0; i < 2; ++i) val[i] = sel[min(max(c * kTcKeys + key0 + 8 * i, nwin), nkeys - 1)];
        }
      };
      auto load_raw = [&](int c) {
        if (has_sel) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            int id = val_cur[i];
            if (id < 0 || id >= p.maxC) {
              tf_report(p.st, TF_BAD_INDEX, 11, r, id);
              id = 0;
            }
            const uint8_t* row = comp + (long)id * p.comp_row;
            rawv[i] = *reinterpret_cast<const uint4*>(row + piece * 16);
            rsc[i] = *reinterpret_cast<const uint16_t*>(row + DH / 2 + piece * 2);          // one scale per 16 dims
          }
        }
      };
      if (live) {
        load_val(0, val_cur);
        load_val(1, val_next);
        load_raw(0);
      }
      for (int c = 0; c < nchunks; ++c) {
        if (live) {
          const int s = it & 1;
          if (!(ok = tc::mbar_wait(empty(s), ((it >> 1) & 1) ^ 1, abort_flag))) break;
          uint8_t* kt = st_g + s * kTcStage + (piece >> 1) * kTcSub;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int key = key0 + 8 * i, k = c * kTcKeys + key, kd = kind(k);
            // eight dims = one 16-byte piece of the f16 row at a time
            auto put = [&](int q, const uint32_t (&hv)[4]) {
              *reinterpret_cast<uint4*>(kt + sw128(key, (piece & 1) * 64 + q * 16)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
            };
            if (kd == 2) {
              // e2m1 values and their group's e4m3 scale are exact in f16, and so is the product
              const uint32_t w[4] = {rawv[i].x, rawv[i].y, rawv[i].z, rawv[i].w};
              const uint32_t slo = e4m3x2_to_h2((uint16_t)((rsc[i] & 0xffu) * 0x101u)), shi = e4m3x2_to_h2((uint16_t)((rsc[i] >> 8) * 0x101u));
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const __half2 sc2 = *reinterpret_cast<const __half2*>(q < 2 ? &slo : &shi);
                uint32_t hv[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const uint32_t v = e2m1x2_to_h2(w[q] >> (8 * e));
                  const __half2 x = __hmul2(*reinterpret_cast<const __half2*>(&v), sc2);
                  hv[e] = *reinterpret_cast<const uint32_t*>(&x);
                }
                put(q, hv);
              }
            } else if (kd == 1) {
              // (a window row is fetched here: a chunk of the row's seventeen, and the others keep their registers)
              const uint8_t* row = win + (long)((pos - nwin + 1 + k) % p.ring) * p.win_row;
              const float sc = ue8m0_to_float(row[DH + piece]);                             // one scale per 32 dims
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint2 raw = *reinterpret_cast<const uint2*>(row + piece * 32 + q * 8);
                uint32_t hv[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  uint32_t h2 = e4m3x2_to_h2((uint16_t)((e < 2 ? raw.x : raw.y) >> (16 * (e & 1))));
                  const float2 v = __half22float2(*reinterpret_cast<__half2*>(&h2));
                  hv[e] = pack_h2(v.x * sc, v.y * sc);
                }
                put(q, hv);
              }
            } else {
              const uint32_t z[4] = {0u, 0u, 0u, 0u};
#pragma unroll
              for (int q = 0; q < 4; ++q) put(q, z);
            }
          }
          tc::fence_proxy_async();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(full(s));
          // request the next chunk's rows and the ids of the chunk after it
#pragma unroll
          for (int i = 0; i < 2; ++i) val_cur[i] = val_next[i];
          load_raw(c + 1);
          load_val(c + 2, val_next);
          ++it;
        }
        // The row before is finished here, behind the first two chunks of this one: the stage after them is not
        // freed before the PV that waits for O to have been read
        if (last_r >= 0 && (c == 1 || nchunks == 1)) {
          const int n = n_row - 1;
          if (!(ok = tc::mbar_wait(l_ready + 8u * (n & 1), (n >> 1) & 1, abort_flag))) break;
          if (!(ok = tc::mbar_wait(o_ready, last_it & 1, abort_flag))) break;
          tc::tc_fence_after();
          if (!(ok = finish_row(p, last_r, warp, lane, tO, stat + (n & 1) * 128, rot + (n & 1) * 32, xch, o_free, meet, abort_flag))) break;
          last_r = -1;
        }
      }
      if (!live) break;
      last_r = r;
      last_it = it - 1;
    }
  } else {
    // ------------------------------------------------------------------ softmax: one head and 64 keys of a chunk per thread
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcSoftmaxRegs));
    const int quad = warp - kTcProd, hi = quad >> 1, h = (quad & 1) * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    // (after a time-out the warp stops waiting and runs out its loop: the launch's result is void)
    bool fail = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      if (!fail && !tc::mbar_wait(bar, parity, abort_flag)) fail = true;
      __syncwarp();
    };
    // ---- MMAs, by one thread of the first softmax warp: S is waited for by all four in any case
    constexpr uint32_t idesc = tc::instr_desc(0, 0, 128, 128);      // f16 x f16, M 128, N 128, both K-major
    constexpr uint32_t idesc_pv = idesc | (1u << 16);               // B (the key tile as V) MN-major
    auto qk = [&](int i, int n_row, bool first) {                    // S = Q . Kt(stage i & 1)^T
      const int s = i & 1;
      if (first && !fail && !tc::mbar_wait(q_ready, n_row & 1, abort_flag)) fail = true;
      if (!fail && !tc::mbar_wait(full(s), (i >> 1) & 1, abort_flag)) fail = true;
      // S lies over the P that the PV before reads: MMAs with different accumulators are not ordered among
      // themselves, so that PV has to be done, not only issued
      if (i > 0 && !fail && !tc::mbar_wait(o_ready, (i & 1) ^ 1, abort_flag)) fail = true;
      if (fail) return;
      tc::tc_fence_after();
      const uint64_t dq = tc::smem_desc_sw128(q_s), dk = tc::smem_desc_sw128(st_s + s * kTcStage);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          tc::mma_f16(tS, dq + (j * kTcSub >> 4) + 2 * k, dk + (j * kTcSub >> 4) + 2 * k, idesc, (j | k) ? 1u : 0u);
      tc::mma_commit(s_ready);
    };
    auto pv = [&](int i, int n_row, bool first) {
      if (!fail && !tc::mbar_wait(p_ready, i & 1, abort_flag)) fail = true;
      // the first PV of a row overwrites O: the row before must have been read
      if (first && !fail && !tc::mbar_wait(o_free, (n_row & 1) ^ 1, abort_flag)) fail = true;
      if (fail) return;
      tc::tc_fence_after();
      // B = the same key tile read MN-major (dims contiguous): 16 keys per step = 2,048 bytes, 8 columns of P
      const uint64_t dv = smem_desc_sw128_mn(st_s + (i & 1) * kTcStage);
#pragma unroll
      for (int k = 0; k < 8; ++k) mma_f16_ts(tO, tS + 8u * k, dv + 128u * k, idesc_pv, (!first || k) ? 1u : 0u);
      tc::mma_commit(empty(i & 1));
      tc::mma_commit(o_ready);
    };
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    // Q of a row, 64 heads x 128 bf16 = 1,024 16-byte pieces, as f16 and twice.  The QK MMAs of the row before are done
    // (their S has been waited for), and PV of its last chunk runs meanwhile.
    auto load_q = [&](int r) {
      const int tid = (int)threadIdx.x - kTcProd * 32;
      const uint4* qsrc = reinterpret_cast<const uint4*>(p.q + (long)r * p.Hl * DH);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int pc = tid + 128 * j, hd = pc >> 4, c16 = pc & 15;  // 16 pieces per head row
        uint4 v = hd < p.Hl ? qsrc[pc] : make_uint4(0u, 0u, 0u, 0u);
        uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {                              // bf16 pair -> f16 pair
          const float2 f2 = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&vw[e]));
          vw[e] = pack_h2(f2.x, f2.y);
        }
        uint8_t* dst = q_g + (c16 >> 3) * kTcSub + sw128(hd, (c16 & 7) * 16);
        *reinterpret_cast<uint4*>(dst) = v;
        *reinterpret_cast<uint4*>(dst + 64 * 128) = v;              // row h + 64: the same swizzle
      }
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(q_ready);
    };
    int it = 0, n_row = 0;
    RowMeta meta = row_meta(p, blockIdx.x);
    load_q(blockIdx.x);
    for (int r = blockIdx.x; r < p.T; r += gridDim.x, ++n_row) {
      int nwin;
      const int nkeys = row_keys(p, meta, r, &nwin);
      const int nchunks = chunks_of(nkeys);
      const int next = r + (int)gridDim.x, pos = meta.pos;
      meta = row_meta(p, next);
      float m = kNegBig;
      float2 l2 = make_float2(0.f, 0.f);
      for (int c = 0; c < nchunks; ++c, ++it) {
        const int valid = nkeys - c * kTcKeys - hi * 64; // columns >= valid of this half are padding
        if (quad == 0) {
          if (tc::elect_one()) qk(it, n_row, c == 0);
          __syncwarp();
        }
        wait(s_ready, it & 1);
        tc::tc_fence_after();
        uint32_t v[64];
        tc::tmem_ld32(tS + lane_off + hi * 64, *reinterpret_cast<uint32_t(*)[32]>(v));
        tc::tmem_ld32(tS + lane_off + hi * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
        tc::tmem_ld_wait();
        if (valid < 64) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (i >= valid) v[i] = __float_as_uint(-INFINITY);
        }
        // The reference maximum m is the first chunk's; it moves only when some head finds a score
        // more than 2^8 above it (then O and l are rescaled).  Until then exp2(s - m) <= 256 is harmless in
        // f16 / fp32 and the ratio O / l does not depend on m.
        float cm[4] = {kNegBig, kNegBig, kNegBig, kNegBig};
#pragma unroll
        for (int i = 0; i < 64; ++i) cm[i & 3] = fmaxf(cm[i & 3], __uint_as_float(v[i]));
        const float top = fmaxf(fmaxf(cm[0], cm[1]), fmaxf(cm[2], cm[3])) * p.scale_log2;
        if (c == 0) {
          m = top;
        } else if (__any_sync(0xffffffffu, top > m + 8.f)) {
          // (QK of this chunk was issued when the PV before was done: O is complete)
          const float nm = fmaxf(m, top), f = exp2f(m - nm);
          m = nm;
          l2.x *= f;
          l2.y *= f;
          wait(o_ready, (it & 1) ^ 1);
          tc::tc_fence_after();
#pragma unroll 1
          for (int q = 0; q < 16; ++q) {
            uint32_t o[8];
            tmem_ld8_tc(tO + lane_off + q * 8, o);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st8_tc(tO + lane_off + q * 8, o);
          }
        }
        const float2 nm2 = make_float2(-m, -m);
        uint32_t pk[32];
        // A chunk's sum is closed before it is added to the row's: one chain through a row of 8,192 keys gathers up to 2.7e-5 of
        // the sum (an addend whose last bits round the same way every time), chains of 32 and one addition a chunk 9e-7.
        float2 lc = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float2 x = fma2(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sc2, nm2);
          const float2 e = make_float2(exp2f(x.x), exp2f(x.y));
          lc = add2(lc, e);
          pk[i] = pack_h2(e.x, e.y);
        }
        l2 = add2(l2, lc);
        // P over the columns of S that this thread holds in registers; zeros for the other half's keys
        tmem_st32(tS + lane_off + hi * 32, pk);
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = 0u;
        tmem_st32(tS + lane_off + (hi ^ 1) * 32, pk);
        tmem_st_wait_tc();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(p_ready);
        if (quad == 0) {
          if (tc::elect_one()) pv(it, n_row, c == 0);
          __syncwarp();
        }
      }
      stat[(n_row & 1) * 128 + hi * 64 + h] = make_float2(m, l2.x + l2.y);
      if (quad == 3) {
        float sn = 0.f, cs = 1.f;
        if (lane < p.rope_dim / 2) {
          const float ang = (float)pos * p.freqs[lane];
          const double two_pi = 6.283185307179586476925286766559;
          sincosf((float)((double)ang - two_pi * floor((double)ang / two_pi)), &sn, &cs);
        }
        rot[(n_row & 1) * 32 + lane] = make_float2(sn, cs);
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(l_ready + 8u * (n_row & 1));
      if (next < p.T) load_q(next);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) tf_report(p.st, TF_TIMEOUT, 150, blockIdx.x, 0);
  if (warp == kTcProd) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tS, 256);
  }
}
