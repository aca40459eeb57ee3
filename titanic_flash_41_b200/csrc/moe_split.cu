// Routed-expert GEMV of decode rows with f16 activations on the block-scaled tensor cores.
//
// The experts are MXFP4 (packed e2m1, one UE8M0 scale per 32 inputs).  Where the activations stay f16, the register-fed kernel
// of smallm_gemm.cu unpacks every nibble on the CUDA cores and runs at half of the HBM rate.  An f16 number is the sum of
// six e4m3 numbers with block scales of their own, so six rows of `tcgen05.mma kind::mxf8f6f4.block_scale` replace one f16 row:
//
//   x = p0 + p1 + .. + p5      p_i: e4m3, UE8M0 scale per 32 inputs of the remainder x - p0 .. - p_{i-1}
//
// Each piece takes four significant bits of an element near the maximum of what its block still holds, and all bits above 2^-9 of
// its scale of the others; the maximum falls by 16 or more from piece to piece.  Three pieces hold the eleven bits of every
// element above 2^-14 of its block's maximum, six those of any finite f16 numbers in one block (the largest is 2^40 times the
// smallest; with three, four, five pieces up to 2^-27, 2^-32, 2^-37 of the maximum were left).  Products of e2m1 and e4m3 are exact and
// sums are fp32; the pieces' sums are added in fp32, the smallest first.  Error against fp64 sums of the same 5,120 f16 inputs, mean of
// twelve draws (f16 x f16 mma.sync form beside it): normal 3.9e-8 (2.0e-7), magnitudes spread over e^normal 6.3e-8 (5.6e-7), over
// e^(2 normal) 1.05e-6 (1.50e-6), SwiGLU products 9.6e-8 (7.7e-7).
//
// An accumulator has 16 columns: two rows of an expert (six columns each).  An expert with more rows takes another pass over
// its weights, out of L2; decode blocks give an expert one or two.
//
//   split_rows_kernel  the activations of every (row, expert) pair, in the order of the groups, as six rows
//   moe_split_kernel   persistent CTAs, one per SM; work item = (expert, 128 features of w1 and of w3) or
//                      (expert, 256 features of w2); FC1 writes FC2's input (clamped SwiGLU, rounded to f16, six pieces)
//     warp 0    TMA producer of the tiles, warp 1 MMA issuer, warps 2-5 scale movers and epilogue, warp 6 TMA producer of the
//               scales (512 inputs at a time: row-major as stored, 16 bytes a row)
// The structure of a CTA is that of moe_mx.cu; here K may end inside 512 inputs, and rows of scales may be 8 bytes off the
// 16-byte grain (K = 2,304: 72 bytes), which two boxes over pairs of rows fetch.
// 24 rows x 6 of 384 experts, 5,120 -> 2,304 -> 5,120, seven launches of a decode step (two of 24 rows, five of 4): FC1 1,437 (unpacked) ->
// 730 us, FC2 783 -> 386 (three pieces: 685 and 374).  24 experts of one row: 53 us, 5.7 TB/s of weights, and 33 us, 4.6 (ncu).
//
// Every wait is bounded: on a time-out the CTA raises its abort flag, reports TF_TIMEOUT, frees its tensor memory and returns.
//
// Reference behaviour: the routed-expert decode path of the reference's MoE kernels (runtime/kernels/moe: grouped MXFP4 expert
// matvec with clamped SwiGLU, f16 activations).
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "tc.cuh"

namespace {

constexpr int kThreads = 7 * 32;
constexpr int kTile = 128;          // features of a matrix tile
constexpr int kCols = 16;           // accumulator columns of a matrix
constexpr int kPieces = 6, kItemRows = kCols / kPieces;
constexpr int kBK = 128;            // inputs per stage
constexpr int kStages = 6;
constexpr int kStageBytes = 2 * kTile * 128 + kCols * 128;
constexpr int kSfsSlots = 3;        // staged scales: 512 inputs of 2 x 128 features and 16 rows
constexpr int kSfsMat = 3072, kSfsBytes = 2 * kSfsMat + kCols * 16;
constexpr int kSfBufs = 4;          // scale slots in tensor memory
constexpr int kAccCols = 2 * 2 * kCols;                  // two items x two matrices
constexpr int kSfaCol = kAccCols, kSfbCol = kAccCols + kSfBufs * 32, kTmemCols = 256;
constexpr int kSplitSmem = kStages * kStageBytes + kSfsSlots * kSfsBytes + 1024 + 512;

struct SplitParams {
  const int* g_expert;
  const int* g_start;
  const int* g_count;
  const int* n_groups;
  const int* sorted_pairs;
  void* out;                        // plain form: f32 rows by pair
  uint8_t* q_out;                   // fused form: pieces [6 pairs][N] and their scales [6 pairs][q_pitch]
  uint8_t* q_scale;
  int q_pitch, ldo, N, K, off_grain;       // off_grain: rows of weight scales 8 bytes off the 16-byte grain
  float limit;
  TfStatusWord* status;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t v[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
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
// D[tmem] (+)= (A * scale_A) (B * scale_B)^T, scales read from tensor memory; ONE thread issues
__device__ __forceinline__ void mma_mx(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa,
                                       uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// A = e2m1 (5), B = e4m3 (0), both K-major, UE8M0 scales, `sf`: byte of the 32-bit scale columns
__device__ __forceinline__ uint32_t idesc_mx(uint32_t sf) {
  return (sf << 4) | (5u << 7) | ((uint32_t)(kCols >> 3) << 17) | (1u << 23) | ((uint32_t)(kTile >> 4) << 24) | (sf << 29);
}
// smallest power of two >= amax / 448 (so the scaled values fit e4m3), as an exponent
__device__ __forceinline__ int mx_exponent(float amax) {
  if (!(amax > 0.f)) return -127;
  int e2;
  const float m = frexpf(amax * (1.f / 448.f), &e2);       // value = m * 2^e2, m in [0.5, 1)
  return max(-127, min(127, (m == 0.5f) ? e2 - 1 : e2));
}
// e4m3 has a NaN and no infinity: one in a row, or a product beyond f16, goes on as NaN, and with it every sum over the row (as a
// saturated 448 times the block's scale it came out as a plausible number)
__device__ __forceinline__ float finite_or_nan(float x) { return fmaf(x, 0.f, x); }
__device__ __forceinline__ uint8_t to_e4m3(float x) { return (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3); }

// DUAL 1: w1 and w3 tiles + SwiGLU; 0: two adjacent tiles of one matrix
template <int DUAL>
__global__ void __launch_bounds__(kThreads, 1)
moe_split_kernel(const __grid_constant__ CUtensorMap mapW1, const __grid_constant__ CUtensorMap mapW3,
                 const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapS1,
                 const __grid_constant__ CUtensorMap mapS3, const __grid_constant__ CUtensorMap mapO1,
                 const __grid_constant__ CUtensorMap mapO3, const __grid_constant__ CUtensorMap mapSX, const SplitParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - raw);
  const uint32_t sfs0 = base + kStages * kStageBytes, bar0 = sfs0 + kSfsSlots * kSfsBytes;
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
  auto sf_full = [&](int b) { return bar0 + 8u * (2 * kStages + b); };
  auto sf_empty = [&](int b) { return bar0 + 8u * (2 * kStages + kSfBufs + b); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * kStages + 2 * kSfBufs + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kStages + 2 * kSfBufs + 2 + b); };
  auto sfs_full = [&](int b) { return bar0 + 8u * (2 * kStages + 2 * kSfBufs + 4 + b); };
  auto sfs_empty = [&](int b) { return bar0 + 8u * (2 * kStages + 2 * kSfBufs + 4 + kSfsSlots + b); };
  uint8_t* tail = aligned + kStages * kStageBytes + kSfsSlots * kSfsBytes + 8 * (2 * kStages + 2 * kSfBufs + 4 + 2 * kSfsSlots);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kItemN = DUAL ? kTile : 2 * kTile;
  const int tiles_n = p.N / kItemN, kchunks = p.K / kBK, nsuper = (kchunks + 3) / 4;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(full(s), 1);
      tc::mbar_init(empty(s), 1);
    }
    for (int b = 0; b < kSfBufs; ++b) {
      tc::mbar_init(sf_full(b), 4);
      tc::mbar_init(sf_empty(b), 1);
    }
    for (int b = 0; b < kSfsSlots; ++b) {
      tc::mbar_init(sfs_full(b), 1);
      tc::mbar_init(sfs_empty(b), 4);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(acc_full(b), 1);
      tc::mbar_init(acc_empty(b), 4);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  tf_pdl_sync();
  const int items = *p.n_groups * tiles_n;
  // One step of a role: two rows of one expert against one item's features
  struct Step {
    int item, g, n0, start, count, c0;       // group, first feature, first pair and pairs of the group, first pair of the step
  };
  auto open = [&](Step& s) {
    if (s.item >= items) return;
    s.g = s.item / tiles_n;
    s.n0 = (s.item - s.g * tiles_n) * kItemN;
    s.start = p.g_start[s.g];
    s.count = p.g_count[s.g];
    s.c0 = 0;
  };
  auto advance = [&](Step& s) {
    s.c0 += kItemRows;
    if (s.c0 >= s.count) {
      s.item += gridDim.x;
      open(s);
    }
  };
  Step step = {(int)blockIdx.x, 0, 0, 0, 0, 0};
  open(step);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: tiles
    if (tc::elect_one()) {
      tc::prefetch_tmap(&mapW1);
      tc::prefetch_tmap(&mapX);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (; step.item < items && ok; advance(step)) {
        const int wrow = p.g_expert[step.g] * p.N + step.n0, xrow = kPieces * (step.start + step.c0);
        for (int kc = 0; kc < kchunks; ++kc) {
          if (!(ok = tc::mbar_wait(empty(s), ph ^ 1, abort_flag))) break;
          tc::mbar_expect_tx(full(s), 2 * kTile * 64 + kCols * 128);         // (packed bytes of the e2m1 boxes)
          const uint32_t sa = base + s * kStageBytes;
          tc::tma_load_2d(sa, &mapW1, kc * kBK, wrow, full(s));
          if (DUAL) tc::tma_load_2d(sa + kTile * 128, &mapW3, kc * kBK, wrow, full(s));
          else tc::tma_load_2d(sa + kTile * 128, &mapW1, kc * kBK, wrow + kTile, full(s));
          tc::tma_load_2d(sa + 2 * kTile * 128, &mapX, kc * kBK, xrow, full(s));
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000) {}       // copies in flight land before the smem goes back
      }
    }
  } else if (warp == 6) {
    // ------------------------------------------------------------------ TMA producer: scales
    if (tc::elect_one()) {
      const int pitch = p.K >> 5;
      int b = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (; step.item < items && ok; advance(step)) {
        const int wrow = p.g_expert[step.g] * p.N + step.n0, xrow = kPieces * (step.start + step.c0);
        for (int sc = 0; sc < nsuper; ++sc) {
          if (!(ok = tc::mbar_wait(sfs_empty(b), ph ^ 1, abort_flag))) break;
          tc::mbar_expect_tx(sfs_full(b), (p.off_grain ? 2 * 3072 : 2 * 2048) + kCols * 16);
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const uint32_t d = sfs0 + b * kSfsBytes + m * kSfsMat;
            const int row = wrow + (!DUAL && m ? kTile : 0);
            const CUtensorMap* ms = DUAL && m ? &mapS3 : &mapS1;
            if (!p.off_grain) {
              tc::tma_load_2d(d, ms, sc * 16, row, sfs_full(b));
            } else {
              // pairs of rows: the even one at 16 sc, the odd one 8 bytes off the grain
              tc::tma_load_2d(d, ms, sc * 16, row >> 1, sfs_full(b));
              tc::tma_load_2d(d + 1024, DUAL && m ? &mapO3 : &mapO1, pitch - 8 + sc * 16, row >> 1, sfs_full(b));
            }
          }
          tc::tma_load_2d(sfs0 + b * kSfsBytes + 2 * kSfsMat, &mapSX, sc * 16, xrow, sfs_full(b));
          if (++b == kSfsSlots) { b = 0; ph ^= 1; }
        }
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (tc::elect_one()) {
      int s = 0, sb = 0, ab = 0;
      uint32_t ph = 0, sph = 0, aph = 0;
      bool ok = true;
      for (; step.item < items && ok; advance(step)) {
        if (!(ok = tc::mbar_wait(acc_empty(ab), aph ^ 1, abort_flag))) break;
        const uint32_t td = tmem_base + ab * 2 * kCols;
        for (int sc = 0; sc < nsuper && ok; ++sc) {
          if (!(ok = tc::mbar_wait(sf_full(sb), sph, abort_flag))) break;
          tc::tc_fence_after();
          const uint32_t sfa = tmem_base + kSfaCol + sb * 32, sfb = tmem_base + kSfbCol + sb * 16;
          const int nc = min(4, kchunks - 4 * sc);
          for (int c = 0; c < nc; ++c) {
            if (!(ok = tc::mbar_wait(full(s), ph, abort_flag))) break;
            tc::tc_fence_after();
            const uint32_t sa = base + s * kStageBytes;
            const uint64_t da1 = tc::smem_desc_sw128(sa), da3 = tc::smem_desc_sw128(sa + kTile * 128),
                           db = tc::smem_desc_sw128(sa + 2 * kTile * 128);
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
              const uint32_t acc = (sc | c | (int)k) ? 1u : 0u, id = idesc_mx(k);
              mma_mx(td, da1 + 2 * k, db + 2 * k, id, sfa + c * 4, sfb + c * 4, acc);
              mma_mx(td + kCols, da3 + 2 * k, db + 2 * k, id, sfa + 16 + c * 4, sfb + c * 4, acc);
            }
            tc::mma_commit(empty(s));
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
          if (ok) tc::mma_commit(sf_empty(sb));
          if (++sb == kSfBufs) { sb = 0; sph ^= 1; }
        }
        if (ok) tc::mma_commit(acc_full(ab));
        if (++ab == 2) { ab = 0; aph ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ scale movers + epilogue
    // The epilogue of a step runs after the first scales of the next one have been delivered: the MMAs never wait for it.
    const int quad = warp & 3;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    auto epilogue = [&](const Step& st, int opair, int ab, uint32_t aph) -> bool {
      if (!tc::mbar_wait(acc_full(ab), aph, abort_flag)) return false;
      tc::tc_fence_after();
      uint32_t a1[kCols], a3[kCols];
      tmem_ld16(tmem_base + lane_base + ab * 2 * kCols, a1);
      tmem_ld16(tmem_base + lane_base + ab * 2 * kCols + kCols, a3);
      tc::tmem_ld_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(acc_empty(ab));
      const int n = st.n0 + quad * 32 + lane, rows = min(kItemRows, st.count - st.c0);
#pragma unroll
      for (int r = 0; r < kItemRows; ++r) {
        if (r >= rows) break;
        float o1 = __uint_as_float(a1[kPieces * r + kPieces - 1]), o3 = __uint_as_float(a3[kPieces * r + kPieces - 1]);
#pragma unroll
        for (int i = kPieces - 2; i >= 0; --i) {
          o1 += __uint_as_float(a1[kPieces * r + i]);
          o3 += __uint_as_float(a3[kPieces * r + i]);
        }
        if (DUAL) {
          float gate = o1, up = o3;
          if (p.limit > 0.f) {                 // (comparisons, not fminf: a NaN is not clamped away)
            gate = gate > p.limit ? p.limit : gate;
            up = up > p.limit ? p.limit : up < -p.limit ? -p.limit : up;
          }
          float rest = finite_or_nan(__half2float(__float2half(gate / (1.f + __expf(-gate)) * up)));
          // the warp's 32 features are one scale group of the second GEMV's input
#pragma unroll
          for (int i = 0; i < kPieces; ++i) {
            const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, rest == rest ? __float_as_uint(fabsf(rest)) : 0u));
            const int ex = mx_exponent(amax);
            const uint8_t q = to_e4m3(rest * exp2f((float)-ex));
            const long row = kPieces * (long)(st.start + st.c0 + r) + i;
            p.q_out[row * p.N + n] = q;
            if (lane == 0) p.q_scale[row * p.q_pitch + n / 32] = (uint8_t)(ex + 127);
            rest -= e4m3_to_float(q) * exp2f((float)ex);
          }
        } else {
          const int pair = __shfl_sync(0xffffffffu, opair, r);
          float* dst = reinterpret_cast<float*>(p.out) + (long)pair * p.ldo + n;
          dst[0] = o1;
          dst[kTile] = o3;
        }
      }
      return true;
    };
    int f = 0, sb = 0, b = 0, ab = 0, opair = 0, pend_pair = 0;
    uint32_t sph = 0, bph = 0, aph = 0;
    bool ok = true, pending = false;
    Step pend = step;
    for (; step.item < items && ok; advance(step)) {
      for (int sc = 0; sc < nsuper && ok; ++sc, ++f) {
        if (!(ok = tc::mbar_wait(sfs_full(b), bph, abort_flag))) break;
        // rows lane, lane + 32, lane + 64, lane + 96 of each matrix: 16 scale bytes = four 128-input words
        const uint8_t* sl = aligned + kStages * kStageBytes + b * kSfsBytes;
        uint4 w[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = lane + 32 * j;
            if (!p.off_grain) {
              w[m][j] = *reinterpret_cast<const uint4*>(sl + m * kSfsMat + r * 16);
            } else {
              const uint2* src = reinterpret_cast<const uint2*>(sl + m * kSfsMat + ((r & 1) ? 1024 + (r >> 1) * 32 + 8 : (r >> 1) * 16));
              const uint2 lo = src[0], hi = src[1];
              w[m][j] = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
          }
        const uint4 xa = *reinterpret_cast<const uint4*>(sl + 2 * kSfsMat + (lane & (kCols - 1)) * 16);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(sfs_empty(b));
        if (++b == kSfsSlots) { b = 0; bph ^= 1; }
        if (!(ok = tc::mbar_wait(sf_empty(sb), sph ^ 1, abort_flag))) break;
        tc::tc_fence_after();
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint32_t v[16];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            v[0 + j] = w[m][j].x;       // inputs   0..127 of this block: column j = rows 32j..32j+31
            v[4 + j] = w[m][j].y;       // inputs 128..255
            v[8 + j] = w[m][j].z;
            v[12 + j] = w[m][j].w;
          }
          tmem_st16(tmem_base + lane_base + kSfaCol + sb * 32 + m * 16, v);
        }
        {
          uint32_t v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0;
          v[0] = xa.x; v[4] = xa.y; v[8] = xa.z; v[12] = xa.w;
          tmem_st16(tmem_base + lane_base + kSfbCol + sb * 16, v);
        }
        tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(sf_full(sb));
        if (++sb == kSfBufs) { sb = 0; sph ^= 1; }
        if (sc == 0) {
          if (pending) {
            if (!(ok = epilogue(pend, pend_pair, ab, aph))) break;
            if (++ab == 2) { ab = 0; aph ^= 1; }
          }
          // output rows of this step, looked up while its MMAs run
          if (!DUAL) opair = p.sorted_pairs[step.start + min(step.c0 + min(lane, kItemRows - 1), step.count - 1)];
        }
      }
      pend = step;
      pend_pair = opair;
      pending = true;
    }
    if (ok && pending) epilogue(pend, pend_pair, ab, aph);
  }
  tc::tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) tf_report(p.status, TF_TIMEOUT, 145 + DUAL, blockIdx.x, items);
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// x [rows, K] f16 -> pieces of the rows of the sorted pairs: q [6 pairs][K], s [6 pairs][pitch].  One thread per (pair, 32 inputs).
__global__ void __launch_bounds__(128) split_rows_kernel(const __half* __restrict__ x, int ldx, const int* __restrict__ sorted_pairs,
                                                         const int* __restrict__ n_local, int topk, uint8_t* __restrict__ q,
                                                         uint8_t* __restrict__ s, int pitch, int pairs, int K) {
  tf_pdl_sync();
  const int ks = K / 32, i = blockIdx.x * blockDim.x + threadIdx.x, pr = i / ks, b = i - pr * ks;
  if (pr >= min(pairs, *n_local)) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + (long)(sorted_pairs[pr] / topk) * ldx + b * 32);
  float v[32];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 u = src[j];
    const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __half22float2(h[e]);
      v[8 * j + 2 * e] = finite_or_nan(f.x);
      v[8 * j + 2 * e + 1] = finite_or_nan(f.y);
    }
  }
#pragma unroll 1
  for (int piece = 0; piece < kPieces; ++piece) {
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) amax = fmaxf(amax, fabsf(v[j]));          // (of the numbers: fmaxf passes a NaN by)
    const int ex = mx_exponent(amax);
    const float inv = exp2f((float)-ex), scale = exp2f((float)ex);
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint32_t word = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint8_t c = to_e4m3(v[4 * j + e] * inv);
        word |= (uint32_t)c << (8 * e);
        v[4 * j + e] -= e4m3_to_float(c) * scale;
      }
      o[j] = word;
    }
    const long row = kPieces * (long)pr + piece;
    uint4* dst = reinterpret_cast<uint4*>(q + row * K + b * 32);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    s[row * pitch + b] = (uint8_t)(ex + 127);
  }
}

int g_split_sms = 0;

inline bool make_map_fp4(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K) {
  auto fn = tc::encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 31) || ((K / 2) & 31) || (K & 127)) return false;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K / 2};
  cuuint32_t box[2] = {128, (cuuint32_t)kTile};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Rows of a split buffer for one f16 row
TF_API int tf_moe_split_pieces() { return kPieces; }

// Bytes between the scale rows of a split buffer of K inputs (K / 32, rounded up to whole 16 bytes)
TF_API int tf_moe_split_pitch(int K) { return (K / 32 + 15) / 16 * 16; }

// x [rows, K] f16 (16-byte aligned rows) -> q [6 * pairs, K] e4m3, s [6 * pairs, tf_moe_split_pitch(K)] UE8M0: the six pieces of the
// row of every sorted pair (rows sorted_pairs[i] / topk, i < *n_local <= pairs).
TF_API int tf_moe_split_rows(const void* x, int ldx, const int* sorted_pairs, const int* n_local, int topk, int pairs, void* q,
                             void* s, int K, cudaStream_t st) {
  if (pairs <= 0 || K % 32 || ldx % 8 || topk <= 0 || !x || !sorted_pairs || !n_local || !q || !s || (reinterpret_cast<uintptr_t>(x) & 15)) return -1;
  const long n = (long)pairs * (K / 32);
  tf_launch(split_rows_kernel, dim3((unsigned)((n + 127) / 128)), dim3(128), 0, st, reinterpret_cast<const __half*>(x), ldx, sorted_pairs,
            n_local, topk, reinterpret_cast<uint8_t*>(q), reinterpret_cast<uint8_t*>(s), tf_moe_split_pitch(K), pairs, K);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Routed experts over the groups of tf_route_group with split f16 rows (x, sx: tf_moe_split_rows or the fused form's outputs,
// 6 * pairs rows in sorted order).  With w3: clamped SwiGLU of w1 / w3, rounded to f16, as pieces q_out [6 * pairs, N] and
// q_scale [6 * pairs, tf_moe_split_pitch(N)], in sorted order; N a multiple of 128.  Without: f32 out rows by pair; N of 256.
// w [experts, N, K / 2] packed e2m1, s [experts, N, K / 32] UE8M0; K a multiple of 256.
TF_API int tf_moe_gemv_split(const void* w1, const void* w3, const void* s1, const void* s3, int experts, const void* x,
                             const void* sx, int pairs, void* out, int ldo, void* q_out, void* q_scale, int N, int K,
                             const int* g_expert, const int* g_start, const int* g_count, const int* n_groups,
                             const int* sorted_pairs, int max_groups, float limit, void* status, cudaStream_t st) {
  const bool dual = w3 != nullptr;
  if (experts <= 0 || pairs <= 0 || max_groups <= 0 || N <= 0 || K <= 0 || K % 256 || N % (dual ? kTile : 2 * kTile)) return -1;
  if (!w1 || !s1 || !x || !sx || (dual ? !s3 || !q_out || !q_scale : !out) || !g_expert || !g_start || !g_count || !n_groups ||
      !sorted_pairs)
    return -1;
  if (!g_split_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_split_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const uint64_t rows = (uint64_t)experts * N, pitch = K / 32;
  const int off = pitch % 16 != 0;
  CUtensorMap m1, m3, mx, ms1, ms3, mo1, mo3, msx;
  if (!make_map_fp4(&m1, w1, rows, K) || !make_map_fp4(&m3, dual ? w3 : w1, rows, K)) return -4;
  if (!tc::make_map_2d(&mx, x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)kPieces * pairs, K, K, kCols)) return -4;
  if (!tc::make_map_2d_plain(&msx, sx, (uint64_t)kPieces * pairs, tf_moe_split_pitch(K), tf_moe_split_pitch(K), 16, kCols)) return -4;
  auto scales = [&](CUtensorMap* m, CUtensorMap* mo, const void* s) {
    if (!off) {
      const bool ok = tc::make_map_2d_plain(m, s, rows, pitch, pitch, 16, kTile);
      *mo = *m;
      return ok;
    }
    return tc::make_map_2d_plain(m, s, rows / 2, 2 * pitch, 2 * pitch, 16, kTile / 2) &&
           tc::make_map_2d_plain(mo, s, rows / 2, 2 * pitch, 2 * pitch, 32, kTile / 2);
  };
  if (!scales(&ms1, &mo1, s1) || !scales(&ms3, &mo3, dual ? s3 : s1)) return -4;
  SplitParams p;
  p.g_expert = g_expert; p.g_start = g_start; p.g_count = g_count; p.n_groups = n_groups; p.sorted_pairs = sorted_pairs;
  p.out = out; p.ldo = ldo;
  p.q_out = reinterpret_cast<uint8_t*>(q_out); p.q_scale = reinterpret_cast<uint8_t*>(q_scale);
  p.q_pitch = tf_moe_split_pitch(N); p.N = N; p.K = K; p.off_grain = off; p.limit = limit;
  p.status = reinterpret_cast<TfStatusWord*>(status);
  const long items = (long)max_groups * (N / (dual ? kTile : 2 * kTile));
  const int grid = (int)(items < g_split_sms ? items : g_split_sms);
  auto kernel = dual ? moe_split_kernel<1> : moe_split_kernel<0>;
  static unsigned long long limit_set[2] = {0, 0};
  if (tf_smem_limit((const void*)kernel, kSplitSmem, &limit_set[dual]) != cudaSuccess) return -2;
  tf_launch(kernel, dim3(grid), dim3(kThreads), kSplitSmem, st, m1, m3, mx, ms1, ms3, mo1, mo3, msx, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
