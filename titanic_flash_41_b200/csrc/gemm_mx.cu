// Block-scaled tensor-core GEMM for sm_100a (prefill rows):
//
//   C[M, N] = (A * sfa) (B * sfb)^T      A [M, K] e4m3 (MXFP8 activations)
//                                         B [N, K] e4m3, or packed e2m1 (MXFP4 experts, K/2 bytes per row)
//                                         sfa / sfb: one UE8M0 scale per (row, 32 k)
//
// `tcgen05.mma kind::mxf8f6f4.block_scale` applies both scale vectors inside the tensor core, so a
// whole K runs into ONE accumulator in tensor memory: no per-128-k promotion through registers
// (which holds the fp32-scaled form at about half the FP8 rate) and no conversion pass for MXFP4
// weights (TMA expands the nibbles to the padded shared-memory form the instruction reads).
//
// A pair of CTAs (two SMs, `cta_group::2`) works on one tile, and the WEIGHTS are the M side of the instruction: 256
// output features (128 a CTA) by up to 256 activation rows, 32 at a time.  Why:
//   - One SM alone (128 rows x 256 features) reads 48 KB from L2 per 512 cycles of MMAs, 94 bytes a cycle: more than
//     an SM gets.  In a pair each CTA brings its own 128 features and HALF of the rows: 62 bytes a cycle (47 with
//     FP4 weights).
//   - The rows of an expert are whatever the router gave it.  On the N side a tile is as wide as its rows (a multiple
//     of 32), on the M side every tile was 128 rows: at 6 rows an expert 122 of them were padding that was
//     multiplied and, worse, fetched (as many bytes as the weights themselves), at 384 rows one sixth.
//   - The instruction's time is the N side's: measured 128 cycles at N = 256, 64 at 128, 46 from 64 down.
// The copies and MMAs are issued by an elected thread (`elect.sync`): under `lane == 0` the compiler wraps every one of them in
// a loop over the lanes that might be active, and four MMAs and a commit took 390 cycles to issue instead of 100.
// Measured (bf16 out, cold L2; the one-SM form of 128 rows x 256 features before): 16384 x 9984 x 4096 542 -> 433 us
// (3.09 PFLOP/s), 16384 x 4096 x 8192 462 -> 358, 4001 x 9984 x 4096 148 -> 116, 197 x 4096 x 8192 41 -> 26,
// 197 x 4096 x 2048 21.5 -> 15.4.  A k block of a 256-row tile takes 565 cycles: 512 of MMAs, the rest is the drain of the
// accumulator once a tile.  Tiles of 192 rows with two accumulators: 460 and 370 us (more L2 bytes a flop).
//
// Scale layout in global memory ("units"): 128 bytes hold the scales of 32 consecutive rows x 128 k,
// byte (row % 32) * 4 + (k / 32) % 4; units are ordered [k / 128][row / 32].  The scales a tile
// needs for one 128-deep k block are then contiguous (512 B for 128 features, 1 KB for 256 rows): one bulk copy
// each per stage, and a warp moves them to tensor memory with one 4-byte shared load per lane and column
// (tcgen05.st; columns j = rows 32j..32j+31, byte = which 32-k group).  Expert scales are read as stored instead
// (row-major, 16 bytes = 512 k of 128 rows a TMA box): their re-ordering was 5 % of a short prefill.
//
// Persistent CTA pairs; in each CTA:
//   warp 0       TMA producer of the operands (its 128 features, its half of the tile's rows); warp 14 of the scales.
//                One thread that issued all of a k block's copies took 720 - 770 cycles for it, more than the MMAs.
//   warp 1       owns the tensor memory; in the first CTA of the pair one thread issues the MMAs of both
//   warps 2-5    scale movers: shared memory -> tensor memory, one per 32-lane quadrant; they arrive at the first CTA's
//                barrier.  The operand tiles of both CTAs complete on the first CTA's barrier by themselves.
//   warps 6-13   epilogue: tensor memory -> registers -> bf16 / f32; a lane is a feature, a register a row, so a
//                warp stores 64 (128) contiguous bytes of one row
// Stages and accumulators follow the tile: as many stages as 227 KB hold (6 at 256 rows, 9 at 32), two accumulators
// where tensor memory has room for two (up to 192 rows).  With one, the epilogue takes all of its columns into registers
// (bf16: packed) before it stores, so that the next tile's MMAs wait for the drain only.
// Grouped form (routed experts): a list of tiles, each with its expert, first row and rows; B holds the experts' matrices
// one after another (rows [e * N, (e + 1) * N)).
// Every mbarrier wait is bounded: on a time-out the CTA raises its abort flag, reports TF_TIMEOUT, lets
// copies in flight land, frees its tensor memory and returns.
//
// The same kernel without scales (MX = 0) multiplies bf16 x bf16 (64 k a block, the vision tower and the router logits of
// gemm_tc.cu): no scale movers, and two accumulators always fit.
// 8192^3: 1.59 PFLOP/s (1.35 by the one-SM form of gemm_tc.cu).
//
// Reference behaviour: block-scaled dense and expert GEMMs of the prefill path
// (src/blockscaled.rs:21-87 scale format; src/fp8_linear.rs:122 call site; the b12x
// `gemm.dense` / `moe.grouped` bundles).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "gemm_pair.h"
#include "tc.cuh"

namespace {

constexpr int BF = 256, BK = 128;                              // features of a pair's tile, k block
constexpr int kMaxRows = 256;                                  // rows of a tile
constexpr int kMaxStages = 12;
constexpr int kGroupRows = 8;                                  // row tiles of a dense matrix walked together
constexpr int kSfwBytes = 512;                                 // scales of 128 features
constexpr int kSfSlots = 4, kSfSlotBytes = 3072;               // ring of row-major expert scales: 512 k of 128 features
constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + 4 + kEpiWarps + 1) * 32;
constexpr int kSfCols = 16;                                    // per stage: 4 (features) + 8 (rows), padded
constexpr int kTmemCols = 512;
constexpr int kTailBytes = 512;                                // barriers, tensor-memory address, abort flag
constexpr int kSmemMax = 232448;

struct MxGemmParams {
  int M, N, K;               // N: features of one matrix
  int mats;                  // 2: a second matrix of the same shape follows (columns N .. 2N of C)
  int b_fp4;                 // B is packed e2m1
  int sf_kind;               // weight scales: 0 units, 1 row-major (K / 32 % 16 == 0), 2 row-major (K / 32 % 16 == 8)
  const uint8_t* sfa;        // units [K/128][sfa_units]
  const uint8_t* sfb;        // units [K/128][sfb_units] (sf_kind 0)
  const uint8_t* sfb2;
  int sfa_units, sfb_units;  // units per k block (rows / 32, padded)
  void* C;
  int ldc;
  int tile_n;                // dense: rows of a tile; grouped: the most rows of one
  int box_rows;              // rows of one TMA load of A
  int stages, stage_bytes, bufs;
  const int* tile_expert;    // grouped form (null: dense)
  const int* tile_row0;      // first row of a tile (null: 128 * tile)
  const int* tile_rows;      // rows of a tile that count (null: 128); the others are not stored
  const int* num_tiles;
  int max_tiles;             // room of the lists
  TfStatusWord* status;
};

__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t v[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t v[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t v[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

// ---- a pair of CTAs
__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the barrier at the same offset of the pair's first CTA
__device__ __forceinline__ uint32_t of_first(uint32_t bar) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(bar));
  return r;
}
// A tile of this CTA whose bytes complete on a barrier of the pair's first CTA: the operands of both CTAs announce themselves to
// the thread that issues the MMAs of both, with no thread of the second CTA in between.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t first_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(first_bar)
      : "memory");
}
// Arrival at a barrier of the pair's first CTA, and the wait for it.  All that they order is tensor memory (scale columns
// written, accumulators read), between the tcgen05 fences on both sides: relaxed, at cluster scope.  With .release.cluster and
// .acquire.cluster every k block paid two memory barriers, about 2,000 cycles.
__device__ __forceinline__ void arrive_first(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(of_first(bar)) : "memory");
}
__device__ __forceinline__ bool pair_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded like tc::mbar_wait
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (pair_try(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (pair_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > 2000000000LL) {
      *abort_flag = 1;
      return false;
    }
  }
}
// one arrival at this barrier of BOTH CTAs when every MMA issued so far by this thread has completed
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}

// D[tmem of both CTAs] (+)= (A * sfa) (B * sfb)^T, scales read from tensor memory; ONE thread of the first CTA issues
__device__ __forceinline__ void mma_mx(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa,
                                       uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// block-scaled instruction descriptor: A (the weights) e4m3 (0) or e2m1 (5), B (the rows) e4m3, both K-major, UE8M0 scales,
// M = 256; + `sf` in both scale-id fields: which byte of the 32-bit scale columns this 32-k step uses
__device__ __forceinline__ uint32_t idesc_mx(uint32_t afmt, uint32_t rows) {
  return (afmt << 7) | ((rows >> 3) << 17) | (1u << 23) | ((uint32_t)(BF >> 4) << 24);
}

struct MxTile {
  int row0, rows, n;         // first row, rows that count and that C has (0 or less: none), columns of the MMA (a multiple of 32)
  int f0;                    // first feature inside its matrix
  int wrow;                  // the same as a row of B
  int mat;
};

template <int OUT_F32, int MX>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_mx_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapW,
               const __grid_constant__ CUtensorMap mapW2, const __grid_constant__ CUtensorMap mapS,
               const __grid_constant__ CUtensorMap mapS2, const __grid_constant__ CUtensorMap mapSo,
               const __grid_constant__ CUtensorMap mapSo2, const MxGemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;            // swizzled tiles need 1024-byte alignment
  uint8_t* aligned = smem_raw + (base - raw);
  const int stages = p.stages, stage_bytes = p.stage_bytes;
  const uint32_t sfs0 = base + stages * stage_bytes;       // ring of row-major scales
  const uint32_t bar0 = sfs0 + (p.sf_kind ? kSfSlots * kSfSlotBytes : 0);
  auto full = [&](int s) { return bar0 + 8u * s; };                             // of the first CTA: operands of both
  auto empty = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
  auto sc_full = [&](int s) { return bar0 + 8u * (2 * kMaxStages + s); };        // this CTA's scales in shared memory
  auto sf_full = [&](int s) { return bar0 + 8u * (3 * kMaxStages + s); };        // of the first CTA: those of both in tensor memory
  auto tfull = [&](int b) { return bar0 + 8u * (4 * kMaxStages + b); };
  auto tempty = [&](int b) { return bar0 + 8u * (4 * kMaxStages + 2 + b); };     // of the first CTA
  auto sfs_full = [&](int b) { return bar0 + 8u * (4 * kMaxStages + 4 + b); };
  auto sfs_empty = [&](int b) { return bar0 + 8u * (4 * kMaxStages + 4 + kSfSlots + b); };
  constexpr int kBars = 4 * kMaxStages + 4 + 2 * kSfSlots;
  static_assert(8 * kBars + 8 <= kTailBytes, "");
  uint8_t* tail = aligned + (bar0 - base) + 8 * kBars;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)pair_rank();
  constexpr int BKE = MX ? BK : 64;                        // elements of a 128-byte k block
  const int kblocks = p.K / BKE;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      tc::mbar_init(full(s), 1);
      tc::mbar_init(empty(s), 1);
      tc::mbar_init(sc_full(s), 1);
      tc::mbar_init(sf_full(s), 8);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(tfull(b), 1);
      tc::mbar_init(tempty(b), 2 * kEpiWarps);
    }
    for (int b = 0; b < kSfSlots; ++b) {
      tc::mbar_init(sfs_full(b), 1);
      tc::mbar_init(sfs_empty(b), 4);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc::tc_fence_before();
  __syncthreads();
  pair_sync();                                              // the other CTA's barriers are set up
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t sf_base = tmem_base + kTmemCols - stages * kSfCols;      // scale columns behind the accumulators
  // set-up done: wait for the kernel before this one (operands and tile lists are its outputs)
  tf_pdl_sync();
  const int fb1 = (p.N + BF - 1) / BF, fbs = fb1 * p.mats;  // feature blocks of one matrix, of all
  const int rt = p.tile_expert ? min(*p.num_tiles, p.max_tiles) : (p.M + p.tile_n - 1) / p.tile_n;
  const int items = rt * fbs;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  // Order of the tiles.  The pairs running at one time should share their operands: experts take all feature
  // blocks of a row tile before the next one (256 experts of one tile, N 2048, K 4096, with the row tiles first:
  // the rows of all experts were fetched again for every block), dense matrices eight row tiles by as many feature
  // blocks as there are pairs.
  auto tile_of = [&](int item) {
    MxTile t;
    int ri, fb;
    if (p.tile_expert) {
      ri = item / fbs;
      fb = item - ri * fbs;
      t.row0 = p.tile_row0 ? p.tile_row0[ri] : 128 * ri;
      t.rows = min(p.tile_rows ? p.tile_rows[ri] : 128, p.M - t.row0);
    } else {
      const int g = item / (kGroupRows * fbs), r = item - g * kGroupRows * fbs, gm = min(kGroupRows, rt - g * kGroupRows);
      ri = g * kGroupRows + r % gm;
      fb = r / gm;
      t.row0 = ri * p.tile_n;
      t.rows = min(p.tile_n, p.M - t.row0);
    }
    t.rows = min(t.rows, p.tile_n);
    t.n = (max(t.rows, 1) + 31) & ~31;                      // (an empty tile is walked like one of a row; nothing is stored)
    t.mat = fb >= fb1;
    t.f0 = (fb - (t.mat ? fb1 : 0)) * BF;
    t.wrow = t.f0 + (p.tile_expert ? p.tile_expert[ri] * p.N : 0) + rank * 128;
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: operand tiles
    if (tc::elect_one()) {
      tc::prefetch_tmap(&mapX);
      tc::prefetch_tmap(&mapW);
      const int wbytes = p.b_fp4 ? 128 * 64 : 128 * 128, box_bytes = p.box_rows * 128;
      const uint32_t first_full = of_first(full(0));
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int item = first; item < items && ok; item += step) {
        const MxTile t = tile_of(item);
        const CUtensorMap* mw = t.mat ? &mapW2 : &mapW;
        const int half = t.n >> 1, xrow = t.row0 + rank * half, loads = (half + p.box_rows - 1) / p.box_rows;
        const uint32_t tx = 2 * (wbytes + loads * box_bytes);             // both CTAs' (parts of a box out of range count too)
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!(ok = tc::mbar_wait(empty(s), ph ^ 1, abort_flag))) break;
          // (the second CTA's bytes may come before the first has set its count: the phase cannot end before that arrival,
          // nor can it be an older one, whose MMAs have freed this stage)
          if (rank == 0) tc::mbar_expect_tx(full(s), tx);
          const uint32_t sa = base + s * stage_bytes, sx = sa + 128 * 128, bar = first_full + 8u * s;
          tma_load_pair(sa, mw, kb * BKE, t.wrow, bar);
          tma_load_pair(sx, &mapX, kb * BKE, xrow, bar);
          for (int i = 1; i < loads; ++i) tma_load_pair(sx + i * box_bytes, &mapX, kb * BKE, xrow + i * p.box_rows, bar);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
      // the last commits arrive at this CTA's barriers before it may leave
      for (int i = 0; i < stages && ok; ++i) {
        ok = tc::mbar_wait(empty(s), ph ^ 1, abort_flag);
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000) {}       // copies in flight land before the smem goes back
      }
    }
  } else if (warp == kThreads / 32 - 1) {
    // ------------------------------------------------------------------ TMA producer: scales
    if (MX && tc::elect_one()) {
      int s = 0, b = 0;
      uint32_t ph = 0, bph = 0;
      bool ok = true;
      for (int item = first; item < items && ok; item += step) {
        const MxTile t = tile_of(item);
        const uint8_t* sfw = (t.mat ? p.sfb2 : p.sfb) + (long)(t.wrow >> 5) * 128;
        const uint8_t* sfx = p.sfa + (long)(t.row0 >> 5) * 128;
        const uint32_t xbytes = t.n * 4;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (p.sf_kind && (kb & 3) == 0) {
            if (!(ok = tc::mbar_wait(sfs_empty(b), bph ^ 1, abort_flag))) break;
            const uint32_t d = sfs0 + b * kSfSlotBytes;
            const int x = kb * 4;
            if (p.sf_kind == 1) {
              tc::mbar_expect_tx(sfs_full(b), 2048);
              tc::tma_load_2d(d, t.mat ? &mapS2 : &mapS, x, t.wrow, sfs_full(b));
            } else {
              // rows of K / 32 = 8 (mod 16) bytes, seen as pairs: the even row at x, the odd one 8 bytes off the grain
              tc::mbar_expect_tx(sfs_full(b), 3072);
              tc::tma_load_2d(d, t.mat ? &mapS2 : &mapS, x, t.wrow >> 1, sfs_full(b));
              tc::tma_load_2d(d + 1024, t.mat ? &mapSo2 : &mapSo, (p.K >> 5) - 8 + x, t.wrow >> 1, sfs_full(b));
            }
            if (++b == kSfSlots) { b = 0; bph ^= 1; }
          }
          if (!(ok = tc::mbar_wait(empty(s), ph ^ 1, abort_flag))) break;
          const uint32_t sc = base + (s + 1) * stage_bytes - 2048;
          tc::mbar_expect_tx(sc_full(s), xbytes + (p.sf_kind ? 0 : kSfwBytes));
          tc::bulk_g2s(sc + kSfwBytes, sfx, xbytes, sc_full(s));
          if (!p.sf_kind) tc::bulk_g2s(sc, sfw, kSfwBytes, sc_full(s));
          sfx += (long)p.sfa_units * 128;
          sfw += (long)p.sfb_units * 128;
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000) {}       // copies in flight land before the smem goes back
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (rank == 0 && tc::elect_one()) {
      int s = 0, ab = 0;
      uint32_t ph = 0, aph = 0;
      bool ok = true;
      for (int item = first; item < items && ok; item += step) {
        const uint32_t n = (uint32_t)tile_of(item).n, id = MX ? idesc_mx(p.b_fp4 ? 5u : 0u, n) : tc::instr_desc(1, 1, BF, n);
        const uint32_t td = tmem_base + ab * p.tile_n;
        if (!(ok = pair_wait(tempty(ab), aph ^ 1, abort_flag))) break;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (MX && !(ok = pair_wait(sf_full(s), ph, abort_flag))) break;
          if (!(ok = tc::mbar_wait(full(s), ph, abort_flag))) break;
          tc::tc_fence_after();
          const uint32_t sa = base + s * stage_bytes;
          const uint64_t da = tc::smem_desc_sw128(sa), db = tc::smem_desc_sw128(sa + 128 * 128);
          const uint32_t sfw = sf_base + s * kSfCols, sfx = sfw + 4;
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k) {
            if (MX) mma_mx(td, da + 2 * k, db + 2 * k, id | (k << 4) | (k << 29), sfw, sfx, (kb | k) ? 1u : 0u);
            else mma_bf16(td, da + 2 * k, db + 2 * k, id, (kb | k) ? 1u : 0u);
          }
          commit_pair(empty(s));             // frees the stage and, with it, the stage's scale columns
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (ok) commit_pair(tfull(ab));
        if (++ab == p.bufs) { ab = 0; aph ^= 1; }
      }
    }
  } else if (!MX && warp < 6) {
    // ------------------------------------------------------------------ (no scales to move)
  } else if (warp < 6) {
    // ------------------------------------------------------------------ scale movers
    // When sc_full(s) completes for lap r of the ring, the MMAs that read scale columns s in lap r - 1 are
    // done (the producer refilled the stage only after their commit): the columns are free.
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    int s = 0, b = 0;
    uint32_t ph = 0, bph = 0;
    bool ok = true;
    uint4 w[4];                              // row-major scales of feature rows lane + 32 j, 512 k
    for (int item = first; item < items && ok; item += step) {
      for (int kb = 0; kb < kblocks; ++kb) {
        if (p.sf_kind && (kb & 3) == 0) {
          if (!(ok = tc::mbar_wait(sfs_full(b), bph, abort_flag))) break;
          const uint8_t* sl = aligned + stages * stage_bytes + b * kSfSlotBytes;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = lane + 32 * j;
            if (p.sf_kind == 1) {
              w[j] = *reinterpret_cast<const uint4*>(sl + r * 16);
            } else {
              const uint2* src = reinterpret_cast<const uint2*>((r & 1) ? sl + 1024 + (r >> 1) * 32 + 8 : sl + (r >> 1) * 16);
              const uint2 lo = src[0], hi = src[1];
              w[j] = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(sfs_empty(b));
          if (++b == kSfSlots) { b = 0; bph ^= 1; }
        }
        if (!(ok = tc::mbar_wait(sc_full(s), ph, abort_flag))) break;
        const uint8_t* sf = aligned + s * stage_bytes + stage_bytes - 2048;
        uint32_t vw[4], vx[8];
        if (p.sf_kind) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            vw[j] = w[j].x;                  // this block's word; the next one moves up
            w[j] = make_uint4(w[j].y, w[j].z, w[j].w, 0u);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) vw[j] = *reinterpret_cast<const uint32_t*>(sf + j * 128 + lane * 4);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) vx[j] = *reinterpret_cast<const uint32_t*>(sf + kSfwBytes + j * 128 + lane * 4);
        const uint32_t t = sf_base + lane_base + s * kSfCols;
        tmem_st4(t, vw);
        tmem_st8(t + 4, vx);
        tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_first(sf_full(s));
        if (++s == stages) { s = 0; ph ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int quad = warp & 3;                 // TMEM lanes this warp may touch: [32*quad, 32*quad+32)
    const int half = (warp - 6) >> 2;          // which half of the tile's columns
    int ab = 0;
    uint32_t aph = 0;
    bool ok = true;
    for (int item = first; item < items && ok; item += step) {
      const MxTile t = tile_of(item);
      const int cols = t.n >> 1, c0 = half * cols;             // a multiple of 16
      const int f = t.f0 + rank * 128 + quad * 32 + lane;      // this lane's feature
      const int live = f < p.N ? min(cols, t.rows - c0) : 0;   // columns of this warp's half that are stored
      const long off = (long)(t.row0 + c0) * p.ldc + (t.mat ? p.N : 0) + f;
      if (!(ok = tc::mbar_wait(tfull(ab), aph, abort_flag))) break;
      tc::tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + ab * p.tile_n + c0;
      auto release = [&]() {
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_first(tempty(ab));
      };
      if (OUT_F32) {
        float* dst = reinterpret_cast<float*>(p.C) + off;
#pragma unroll 1
        for (int c = 0; c < cols; c += 32) {
          uint32_t v[32];
          tmem_ld16(taddr + c, v);
          if (c + 16 < cols) tmem_ld16(taddr + c + 16, v + 16);
          tc::tmem_ld_wait();
          if (c + 32 >= cols) release();
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (c + i < live) *dst = __uint_as_float(v[i]);
            dst += p.ldc;
          }
        }
      } else {
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + off;
        uint32_t pk[64];
#pragma unroll
        for (int c = 0; c < 128; c += 32) {
          if (c < cols) {
            uint32_t v[32];
            tmem_ld16(taddr + c, v);
            if (c + 16 < cols) tmem_ld16(taddr + c + 16, v + 16);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
              pk[c / 2 + i] = *reinterpret_cast<const uint32_t*>(&h);
            }
          }
        }
        release();
#pragma unroll
        for (int c = 0; c < 128; c += 2) {
          if (c < live) reinterpret_cast<uint16_t*>(dst)[0] = (uint16_t)pk[c / 2];
          if (c + 1 < live) reinterpret_cast<uint16_t*>(dst)[p.ldc] = (uint16_t)(pk[c / 2] >> 16);
          dst += 2 * p.ldc;
        }
      }
      if (++ab == p.bufs) { ab = 0; aph ^= 1; }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) tf_report(p.status, TF_TIMEOUT, MX ? 140 : 141, blockIdx.x, p.b_fp4);
  __syncwarp();
  pair_sync();                                 // nobody leaves while the other CTA may still arrive at its barriers
  if (warp == 1) {
    tc::tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// MXFP8 quantiser of activation rows with the scales in the unit layout.
// One thread per (row, 32 inputs).  dst row = pair_dst[r] when given (expert-sorted padded rows),
// source row = r / x_div.
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ int mx_exponent(float amax) {
  // smallest power of two >= amax / 448 (so the scaled values fit e4m3)
  if (!(amax > 0.f)) return -127;
  int e2;
  const float m = frexpf(amax * (1.f / 448.f), &e2);       // value = m * 2^e2, m in [0.5, 1)
  return max(-127, min(127, (m == 0.5f) ? e2 - 1 : e2));
}

template <typename T>
__global__ void __launch_bounds__(128) quant_rows_mx_units_kernel(const T* __restrict__ x, int ldx, int x_div,
                                                                  const int* __restrict__ pair_dst,
                                                                  uint8_t* __restrict__ q, uint8_t* __restrict__ sf,
                                                                  int sf_units, int rows, int K) {
  tf_pdl_sync();
  const int ks = K / 32;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)rows * ks) return;
  const int r = (int)(i / ks), b = (int)(i % ks);
  const int dst = pair_dst ? pair_dst[r] : r;
  if (dst < 0) return;
  const T* src = x + (long)(r / x_div) * ldx + b * 32;
  // 32 inputs = 64 (or 128) contiguous bytes, 16-byte aligned (ldx is a multiple of 8 elements)
  constexpr int kVec = 16 / sizeof(T);
  T raw[32];
#pragma unroll
  for (int j = 0; j < 32 / kVec; ++j)
    *reinterpret_cast<uint4*>(raw + j * kVec) = *reinterpret_cast<const uint4*>(src + j * kVec);
  float v[32];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    v[j] = to_f<T>(raw[j]);
    amax = fmaxf(amax, fabsf(v[j]));
  }
  const int ex = mx_exponent(amax);
  const float inv = exp2f((float)-ex);
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] * inv, v[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi =
        __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] * inv, v[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    o[j] = lo | (hi << 16);
  }
  uint4* out = reinterpret_cast<uint4*>(q + (long)dst * K + b * 32);
  out[0] = make_uint4(o[0], o[1], o[2], o[3]);
  out[1] = make_uint4(o[4], o[5], o[6], o[7]);
  sf[((long)(b >> 2) * sf_units + (dst >> 5)) * 128 + (dst & 31) * 4 + (b & 3)] = (uint8_t)(ex + 127);
}

// Clamped SwiGLU of [rows, 2I] bf16 (gate | up) -> MXFP8 rows [rows, I] + unit-layout scales.
// One thread per (row, 32 outputs).  `num_rows` (device, optional) bounds the rows at run time, `tile_rows` (optional)
// the rows of each 128-row tile; with `row_of` (optional) row i of the launch is row_of[i] (< 0: none).
__global__ void __launch_bounds__(128) swiglu_rows_mx_units_kernel(const __nv_bfloat16* __restrict__ y, int ldy,
                                                                   uint8_t* __restrict__ q, uint8_t* __restrict__ sf,
                                                                   int sf_units, int rows, int I, float limit,
                                                                   const int* __restrict__ num_rows,
                                                                   const int* __restrict__ tile_rows,
                                                                   const int* __restrict__ row_of) {
  tf_pdl_sync();
  const int ks = I / 32;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int live = num_rows ? min(rows, *num_rows) : rows;
  if (i >= (long)live * ks) return;
  const int b = (int)(i % ks), r = row_of ? row_of[i / ks] : (int)(i / ks);
  if (r < 0) return;
  if (tile_rows && (r & 127) >= tile_rows[r >> 7]) return;           // padding
  const __nv_bfloat16* g = y + (long)r * ldy + b * 32;
  const __nv_bfloat16* u = g + I;
  __nv_bfloat16 gr[32], ur[32];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<uint4*>(gr + 8 * j) = *reinterpret_cast<const uint4*>(g + 8 * j);
    *reinterpret_cast<uint4*>(ur + 8 * j) = *reinterpret_cast<const uint4*>(u + 8 * j);
  }
  float v[32];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    float gate = __bfloat162float(gr[j]), up = __bfloat162float(ur[j]);
    if (limit > 0.f) {
      gate = fminf(gate, limit);
      up = fminf(fmaxf(up, -limit), limit);
    }
    v[j] = gate / (1.f + __expf(-gate)) * up;
    amax = fmaxf(amax, fabsf(v[j]));
  }
  const int ex = mx_exponent(amax);
  const float inv = exp2f((float)-ex);
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] * inv, v[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi =
        __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] * inv, v[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    o[j] = lo | (hi << 16);
  }
  uint4* out = reinterpret_cast<uint4*>(q + (long)r * I + b * 32);
  out[0] = make_uint4(o[0], o[1], o[2], o[3]);
  out[1] = make_uint4(o[4], o[5], o[6], o[7]);
  sf[((long)(b >> 2) * sf_units + (r >> 5)) * 128 + (r & 31) * 4 + (b & 3)] = (uint8_t)(ex + 127);
}

// row-major UE8M0 scales [rows, K/32] -> unit layout [K/128][units][128].  Seen as 4-byte words (the four
// scales of a 128-deep k block) this is the transpose of a [rows][K/128] matrix: word (kb, row) lands at
// kb * units * 32 + row.  Bound by HBM, so a CTA moves 128 rows x 32 words through shared memory and
// both sides are whole 128-byte lines (a 33-word pitch keeps the column reads free of bank conflicts).
// 524,288 rows of K = 4096 (134 MB moved): 272 us with one thread per byte scattered over 512-byte strides, 58 us
// in this form, 20 us in 16-byte pieces (sf_to_units_vec_kernel below), which K / 128 of a multiple of eight takes; this
// form serves the other widths and addresses off the 16-byte grain.  `s` or `out` off a 4-byte boundary: byte by byte.
constexpr int kTrRows = 128, kTrWords = 32;
__global__ void __launch_bounds__(256) sf_to_units_kernel(const uint8_t* __restrict__ s, uint8_t* __restrict__ out,
                                                          long rows, int kb_n, int units, int words) {
  tf_pdl_sync();
  __shared__ uint32_t tile[kTrRows][kTrWords + 1];
  const long r0 = (long)blockIdx.x * kTrRows;
  const int k0 = blockIdx.y * kTrWords, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = k0 + lane;
#pragma unroll
  for (int i = 0; i < kTrRows / 8; ++i) {
    const long r = r0 + warp + 8 * i;
    uint32_t v = 0;
    if (r < rows && k < kb_n) {
      const uint8_t* src = s + (r * kb_n + k) * 4;
      if (words) v = *reinterpret_cast<const uint32_t*>(src);
      else v = src[0] | (src[1] << 8) | (src[2] << 16) | ((uint32_t)src[3] << 24);
    }
    tile[warp + 8 * i][lane] = v;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kTrWords * kTrRows / 256; ++i) {
    const int j = i * 256 + threadIdx.x, kk = j / kTrRows, rr = j % kTrRows;
    if (k0 + kk >= kb_n || r0 + rr >= rows) continue;
    uint8_t* dst = out + ((long)(k0 + kk) * units * 32 + r0 + rr) * 4;
    const uint32_t v = tile[rr][kk];
    if (words) *reinterpret_cast<uint32_t*>(dst) = v;
    else
      for (int b = 0; b < 4; ++b) dst[b] = (uint8_t)(v >> (8 * b));
  }
}

// The same transpose in 16-byte pieces on both sides (rows of a multiple of W words, 16-byte aligned): a CTA
// moves 4096 / W rows x W words.  Word (w, r) sits at w * rows + (r ^ (w / 4) * (128 / W)): the four
// scattered stores of a piece and the 16-byte reads are free of bank conflicts.
template <int W>
__global__ void __launch_bounds__(256) sf_to_units_vec_kernel(const uint8_t* __restrict__ s, uint8_t* __restrict__ out,
                                                              long rows, int kb_n, int units) {
  tf_pdl_sync();
  constexpr int ROWS = 4096 / W;
  __shared__ __align__(16) uint32_t tile[4096];
  const long r0 = (long)blockIdx.x * ROWS;
  const int k0 = blockIdx.y * W;
  uint4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = threadIdx.x + 256 * i, r = p / (W / 4), q = p % (W / 4);
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (r0 + r < rows) v[i] = __ldg(reinterpret_cast<const uint4*>(s + ((r0 + r) * kb_n + k0) * 4) + q);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = threadIdx.x + 256 * i, q = p % (W / 4);
    uint32_t* d = tile + 4 * q * ROWS + ((p / (W / 4)) ^ (q * (128 / W)));
    d[0] = v[i].x;
    d[ROWS] = v[i].y;
    d[2 * ROWS] = v[i].z;
    d[3 * ROWS] = v[i].w;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = threadIdx.x + 256 * i, w = p / (ROWS / 4), r = p % (ROWS / 4) * 4;
    const uint4 o = *reinterpret_cast<const uint4*>(tile + w * ROWS + (r ^ ((w >> 2) * (128 / W))));
    uint8_t* dst = out + ((long)(k0 + w) * units * 32 + r0 + r) * 4;
    if (r0 + r + 3 < rows) {
      *reinterpret_cast<uint4*>(dst) = o;
    } else {
      const uint32_t e[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (r0 + r + j < rows) reinterpret_cast<uint32_t*>(dst)[j] = e[j];
    }
  }
}

// fp32 power-of-two scales per 128 x 128 block [rows/128, K/128] -> unit layout (every 32 x 32
// sub-block of a block carries the block's exponent).  `bad` counts scales that are not powers of two
// in the UE8M0 range.
__global__ void __launch_bounds__(256) block_scales_to_units_kernel(const float* __restrict__ s, int lds,
                                                                    uint8_t* __restrict__ out, long rows, int kb_n,
                                                                    int units, int* __restrict__ bad) {
  tf_pdl_sync();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;      // (row, k block)
  if (i >= rows * kb_n) return;
  const long r = i / kb_n;
  const int kb = (int)(i % kb_n);
  const float v = s[(r >> 7) * lds + kb];
  int e2;
  const float m = frexpf(v, &e2);                                  // v = m * 2^e2
  int ex = e2 - 1;
  if (!(v > 0.f) || m != 0.5f || ex < -127 || ex > 127) {
    if (bad) atomicAdd(bad, 1);
    ex = -127;
  }
  const uint32_t byte = (uint32_t)(ex + 127);
  *reinterpret_cast<uint32_t*>(out + ((long)kb * units + (r >> 5)) * 128 + (r & 31) * 4) = byte * 0x01010101u;
}

int g_sms = 0;

inline bool make_map_fp4(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K) {
  auto fn = tc::encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 31) || ((K / 2) & 31) || (K & 127)) return false;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K / 2};
  cuuint32_t box[2] = {128, 128};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Rows of a dense matrix's tiles: the least estimated time over the tile widths.  Per k block a tile takes its MMAs
// (2 cycles a row) or its L2 bytes (128 features + its rows at 64 bytes a cycle), whichever is longer, and
// the tiles run in waves of one per pair.
inline int dense_rows(int M, int fbs, int pairs, int b_fp4) {
  int best = 32;
  long best_cost = 0;
  for (int n = 32; n <= kMaxRows; n += 32) {
    const long tiles = (long)((M + n - 1) / n) * fbs, waves = (tiles + pairs - 1) / pairs;
    const long cost = waves * (2 * n > (b_fp4 ? 128 : 256) + n ? 2 * n : (b_fp4 ? 128 : 256) + n);
    if (n == 32 || cost <= best_cost) {
      best = n;
      best_cost = cost;
    }
    if (n >= M) break;
  }
  return best;
}

struct MxCall {
  int mx;                    // 0: bf16 x bf16
  const void *A, *B, *B2;
  long lda, ldb, b_rows;
  int b_fp4, sfa_units, sfb_units, sf_rows;
  const void *sfa, *sfb, *sfb2;
  void* C;
  int ldc, out_kind, M, N, K;
  const int *tile_expert, *tile_row0, *tile_rows, *num_tiles;
  int tile_max, max_tiles;
};

int launch_mx(const MxCall& a, void* status, cudaStream_t st) {
  if (!g_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  auto kernel = a.mx ? (a.out_kind == 0 ? gemm_mx_kernel<1, 1> : gemm_mx_kernel<0, 1>)
                     : (a.out_kind == 0 ? gemm_mx_kernel<1, 0> : gemm_mx_kernel<0, 0>);
  static unsigned long long limit_set[4] = {0, 0, 0, 0};
  if (tf_smem_limit((const void*)kernel, kSmemMax, &limit_set[(a.out_kind == 0) + 2 * (a.mx != 0)]) != cudaSuccess) return -2;
  const int pairs = g_sms / 2, mats = a.B2 ? 2 : 1, fbs = (a.N + BF - 1) / BF * mats;
  MxGemmParams p;
  p.tile_n = a.tile_expert ? (a.tile_max + 31) / 32 * 32 : dense_rows(a.M, fbs, pairs, a.b_fp4);
  // one load where all tiles are alike; an expert's rows come 32 at a time, as many as there are
  p.box_rows = a.tile_expert ? 32 : p.tile_n / 2;
  const int x_rows = (p.tile_n / 2 + 31) / 32 * 32;
  p.stage_bytes = 128 * 128 + x_rows * 128 + 2048;
  p.sf_kind = !a.sf_rows ? 0 : a.K / 32 % 16 == 0 ? 1 : 2;
  const int room = kSmemMax - 1024 - kTailBytes - (p.sf_kind ? kSfSlots * kSfSlotBytes : 0);
  p.stages = room / p.stage_bytes < kMaxStages ? room / p.stage_bytes : kMaxStages;
  p.bufs = 2 * p.tile_n + (a.mx ? p.stages * kSfCols : 0) <= kTmemCols ? 2 : 1;
  CUtensorMap mX, mW, mW2, mS, mS2, mSo, mSo2;
  const CUtensorMapDataType dt = a.mx ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int es = a.mx ? 1 : 2;
  if (!tc::make_map_2d(&mX, a.A, dt, es, a.M, a.K, a.lda, p.box_rows)) return -4;
  auto weights = [&](CUtensorMap* m, const void* B) {
    return a.b_fp4 ? a.ldb == a.K / 2 && make_map_fp4(m, B, a.b_rows, a.K)
                   : tc::make_map_2d(m, B, dt, es, a.b_rows, a.K, a.ldb, 128);
  };
  if (!weights(&mW, a.B) || (a.B2 && !weights(&mW2, a.B2))) return -4;
  if (!a.B2) mW2 = mW;
  mS = mS2 = mSo = mSo2 = mX;
  const uint64_t pitch = a.K / 32;
  auto scales = [&](CUtensorMap* m, CUtensorMap* mo, const void* s) {
    if (p.sf_kind == 1) return tc::make_map_2d_plain(m, s, a.b_rows, pitch, pitch, 16, 128);
    return tc::make_map_2d_plain(m, s, a.b_rows / 2, 2 * pitch, 2 * pitch, 16, 64) &&
           tc::make_map_2d_plain(mo, s, a.b_rows / 2, 2 * pitch, 2 * pitch, 32, 64);
  };
  if (p.sf_kind && (!scales(&mS, &mSo, a.sfb) || (a.B2 && !scales(&mS2, &mSo2, a.sfb2)))) return -4;
  p.M = a.M; p.N = a.N; p.K = a.K; p.mats = mats; p.b_fp4 = a.b_fp4 ? 1 : 0;
  p.sfa = reinterpret_cast<const uint8_t*>(a.sfa);
  p.sfb = reinterpret_cast<const uint8_t*>(a.sfb); p.sfb2 = reinterpret_cast<const uint8_t*>(a.B2 ? a.sfb2 : a.sfb);
  p.sfa_units = a.sfa_units; p.sfb_units = a.sfb_units;
  p.C = a.C; p.ldc = a.ldc;
  p.tile_expert = a.tile_expert; p.tile_row0 = a.tile_row0; p.tile_rows = a.tile_rows; p.num_tiles = a.num_tiles;
  p.max_tiles = a.max_tiles;
  p.status = reinterpret_cast<TfStatusWord*>(status);
  const long tiles = (a.tile_expert ? a.max_tiles : (a.M + p.tile_n - 1) / p.tile_n) * (long)fbs;
  const int grid = 2 * (int)(tiles < pairs ? tiles : pairs);
  tf_launch(kernel, dim3(grid), dim3(kThreads), kSmemMax, st, mX, mW, mW2, mS, mS2, mSo, mSo2, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace

int tf_gemm_pair_bf16(const void* A, long lda, const void* B, long ldb, void* C, int ldc, int out_kind, int M, int N, int K,
                      void* status, cudaStream_t st) {
  MxCall a = {};
  a.A = A; a.B = B; a.lda = 2 * lda; a.ldb = 2 * ldb; a.b_rows = N;
  a.C = C; a.ldc = ldc; a.out_kind = out_kind; a.M = M; a.N = N; a.K = K;
  return launch_mx(a, status, st);
}

// Scale units needed for `rows` rows that tiles of `tile_rows` rows may touch (whole tiles).
TF_API long tf_mx_sf_units(long rows, int tile_rows) {
  return (rows + tile_rows - 1) / tile_rows * tile_rows / 32;
}

// C[M, N] (ldc elements per row; out_kind 0 = f32, 2 = bf16) = A (e4m3 [M, K], row pitch lda bytes) x
// B^T.  B: e4m3 [b_rows, K] (row pitch ldb bytes) or, with b_fp4, packed e2m1 [b_rows, K / 2].
// sfa / sfb: unit-layout scales with sfa_units / sfb_units units per 128-deep k block
// (tf_mx_sf_units(M, 128) and tf_mx_sf_units(b_rows, 256) or more).  Grouped form: A rows are expert-sorted in segments
// of whole 128-row tiles, tile_expert / num_m_tiles as in tf_gemm_tc, b_rows = experts * N, N a multiple of 256.
// tile_rows (grouped form, optional): rows of every tile that count; padding is not stored.
TF_API int tf_gemm_mx_rows(const void* A, long lda, const void* B, long ldb, long b_rows, int b_fp4, const void* sfa,
                           int sfa_units, const void* sfb, int sfb_units, void* C, int ldc, int out_kind, int M, int N,
                           int K, const int* tile_expert, const int* num_m_tiles, const int* tile_rows, void* status,
                           cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0 || K % BK || N % 8 || (out_kind != 0 && out_kind != 2)) return -1;
  if (!A || !B || !sfa || !sfb || !C) return -1;
  if (tile_expert && (N % BF || !num_m_tiles)) return -1;
  const long m_tiles = (M + 127) / 128, f_tiles = (N + BF - 1) / BF;
  if (sfa_units < m_tiles * 4) return -1;
  if (sfb_units < (tile_expert ? b_rows / 32 : f_tiles * (BF / 32))) return -1;
  if ((reinterpret_cast<uintptr_t>(sfa) & 15) || (reinterpret_cast<uintptr_t>(sfb) & 15)) return -1;
  if ((reinterpret_cast<uintptr_t>(C) & 15) || (ldc * (out_kind == 0 ? 4 : 2)) % 16) return -1;
  const MxCall a = {1, A, B, nullptr, lda, ldb, b_rows, b_fp4, sfa_units, sfb_units, 0, sfa, sfb, nullptr, C, ldc, out_kind,
                    M, N, K, tile_expert, nullptr, tile_expert ? tile_rows : nullptr, num_m_tiles, 128, (int)m_tiles};
  return launch_mx(a, status, st);
}

// Experts' form: MXFP4 weights and scales as stored.  B (and, optional, B2: a second matrix of the same shape whose columns
// follow at C + N) packed e2m1 [b_rows, K / 2], sb / sb2 row-major UE8M0 [b_rows, K / 32] (b_rows = experts * N, N a
// multiple of 256, K of 256).  Tile t: rows [tile_row0[t], tile_row0[t] + tile_rows[t]) of A, tile_rows[t] <= tile_max
// <= 256, tile_row0 a multiple of 32; A holds M rows and sfa their units (sfa_units >= M / 32).
TF_API int tf_gemm_mx_experts(const void* A, const void* sfa, int sfa_units, const void* B, const void* B2, const void* sb,
                              const void* sb2, long b_rows, void* C, int ldc, int out_kind, int M, int N, int K,
                              const int* tile_expert, const int* tile_row0, const int* tile_rows, const int* num_tiles,
                              int tile_max, int max_tiles, void* status, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 256 || N % BF || b_rows % N || (out_kind != 0 && out_kind != 2)) return -1;
  if (!A || !B || !sfa || !sb || !C || (B2 && !sb2) || !tile_expert || !tile_row0 || !tile_rows || !num_tiles) return -1;
  if (tile_max < 1 || tile_max > kMaxRows || max_tiles < 1 || M % 32 || sfa_units < M / 32) return -1;
  if (reinterpret_cast<uintptr_t>(sfa) & 15) return -1;
  if ((reinterpret_cast<uintptr_t>(C) & 15) || (ldc * (out_kind == 0 ? 4 : 2)) % 16) return -1;
  const MxCall a = {1, A, B, B2, K, K / 2, b_rows, 1, sfa_units, 0, 1, sfa, sb, sb2, C, ldc, out_kind,
                    M, N, K, tile_expert, tile_row0, tile_rows, num_tiles, tile_max, max_tiles};
  return launch_mx(a, status, st);
}

TF_API int tf_gemm_mx(const void* A, long lda, const void* B, long ldb, long b_rows, int b_fp4, const void* sfa,
                      int sfa_units, const void* sfb, int sfb_units, void* C, int ldc, int out_kind, int M, int N,
                      int K, const int* tile_expert, const int* num_m_tiles, void* status, cudaStream_t st) {
  return tf_gemm_mx_rows(A, lda, B, ldb, b_rows, b_fp4, sfa, sfa_units, sfb, sfb_units, C, ldc, out_kind, M, N, K,
                         tile_expert, num_m_tiles, nullptr, status, st);
}

// x [rows / x_div source rows, K] (xkind 0 f32, 1 f16, 2 bf16; row pitch ldx elements) -> q e4m3
// [dst rows, K] + unit-layout scales.  pair_dst (optional): destination row of every source pair.
TF_API int tf_quant_rows_mx_units(const void* x, int xkind, int ldx, int x_div, const int* pair_dst, void* q, void* sf,
                                  int sf_units, int rows, int K, cudaStream_t st) {
  if (rows <= 0 || K % 128 || x_div <= 0 || !x || !q || !sf || ldx % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) return -1;
  const long n = (long)rows * (K / 32);
  const dim3 grid((unsigned)((n + 127) / 128));
  uint8_t* qq = reinterpret_cast<uint8_t*>(q);
  uint8_t* ss = reinterpret_cast<uint8_t*>(sf);
  if (xkind == 0)
    tf_launch(quant_rows_mx_units_kernel<float>, grid, dim3(128), 0, st, reinterpret_cast<const float*>(x), ldx, x_div,
              pair_dst, qq, ss, sf_units, rows, K);
  else if (xkind == 1)
    tf_launch(quant_rows_mx_units_kernel<__half>, grid, dim3(128), 0, st, reinterpret_cast<const __half*>(x), ldx,
              x_div, pair_dst, qq, ss, sf_units, rows, K);
  else if (xkind == 2)
    tf_launch(quant_rows_mx_units_kernel<__nv_bfloat16>, grid, dim3(128), 0, st,
              reinterpret_cast<const __nv_bfloat16*>(x), ldx, x_div, pair_dst, qq, ss, sf_units, rows, K);
  else
    return -1;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

TF_API int tf_swiglu_rows_mx_units(const void* y, int ldy, void* q, void* sf, int sf_units, int rows, int I,
                                   float limit, const int* num_rows, const int* tile_rows, cudaStream_t st) {
  if (rows <= 0 || I % 128 || !y || !q || !sf || ldy % 8 || (reinterpret_cast<uintptr_t>(y) & 15)) return -1;
  const long n = (long)rows * (I / 32);
  tf_launch(swiglu_rows_mx_units_kernel, dim3((unsigned)((n + 127) / 128)), dim3(128), 0, st,
            reinterpret_cast<const __nv_bfloat16*>(y), ldy, reinterpret_cast<uint8_t*>(q),
            reinterpret_cast<uint8_t*>(sf), sf_units, rows, I, limit, num_rows, tile_rows, (const int*)nullptr);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// The same for the rows pair_dst[0 .. pairs) of y and q (negative: skipped)
TF_API int tf_swiglu_pairs_mx_units(const void* y, int ldy, void* q, void* sf, int sf_units, const int* pair_dst, int pairs,
                                    int I, float limit, cudaStream_t st) {
  if (pairs <= 0 || I % 128 || !y || !q || !sf || !pair_dst || ldy % 8 || (reinterpret_cast<uintptr_t>(y) & 15)) return -1;
  const long n = (long)pairs * (I / 32);
  tf_launch(swiglu_rows_mx_units_kernel, dim3((unsigned)((n + 127) / 128)), dim3(128), 0, st,
            reinterpret_cast<const __nv_bfloat16*>(y), ldy, reinterpret_cast<uint8_t*>(q),
            reinterpret_cast<uint8_t*>(sf), sf_units, pairs, I, limit, (const int*)nullptr, (const int*)nullptr, pair_dst);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// row-major UE8M0 scales [rows, K / 32] -> unit layout (`out` holds K / 128 * units * 128 bytes, zeroed by the caller)
TF_API int tf_mx_sf_to_units(const void* s, void* out, long rows, int K, int units, cudaStream_t st) {
  if (rows <= 0 || K % 128 || units * 32L < rows) return -1;
  const uintptr_t both = reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(out);
  const int W = K / 128 % 32 == 0 ? 32 : K / 128 % 16 == 0 ? 16 : K / 128 % 8 == 0 ? 8 : 0;
  if (W && !(both & 15)) {
    auto kernel = W == 32 ? sf_to_units_vec_kernel<32> : W == 16 ? sf_to_units_vec_kernel<16> : sf_to_units_vec_kernel<8>;
    const int tr = 4096 / W;
    tf_launch(kernel, dim3((unsigned)((rows + tr - 1) / tr), K / 128 / W), dim3(256), 0, st,
              reinterpret_cast<const uint8_t*>(s), reinterpret_cast<uint8_t*>(out), rows, K / 128, units);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  const int words = !(both & 3);
  tf_launch(sf_to_units_kernel, dim3((unsigned)((rows + kTrRows - 1) / kTrRows), (K / 128 + kTrWords - 1) / kTrWords),
            dim3(256), 0, st, reinterpret_cast<const uint8_t*>(s), reinterpret_cast<uint8_t*>(out), rows, K / 128,
            units, words);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// fp32 scales per 128 x 128 block (row pitch lds) -> unit layout; *bad (device, optional) counts
// scales that are not exact powers of two in range (such a matrix cannot take this path)
TF_API int tf_mx_block_scales_to_units(const float* s, int lds, void* out, long rows, int K, int units, int* bad,
                                       cudaStream_t st) {
  if (rows <= 0 || K % 128 || units * 32L < rows) return -1;
  const long n = rows * (K / 128);
  tf_launch(block_scales_to_units_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, s, lds,
            reinterpret_cast<uint8_t*>(out), rows, K / 128, units, bad);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
