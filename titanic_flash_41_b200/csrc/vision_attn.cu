// Dense attention of the vision tower on the tcgen05 tensor cores (head dim 64, no mask but the length).
//
//   S[row, key]  = Q[row, :] . K[key, :]          A = Q [128 x 64]  B = K tile [128 x 64], K-major
//   O[row, dim] += P[row, key] * V[key, dim]      A = P [128 x 128] in tensor memory, B = V tile, MN-major
//
// A CTA takes 128 query rows of one head and walks the keys in tiles of 128; scores and probabilities
// never leave the SM.  Four softmax warps (one accumulator lane = one query row per thread) turn S
// into bf16 probabilities that go back to tensor memory as the A operand of PV; the reference maximum is the
// first tile's and moves (O rescaled) only when a score exceeds it by 2^8.  A row of S is read into
// registers at once, so QK of tile j + 1 runs under the exponentials of tile j.  One thread issues TMA (K and V rings of two tiles), one the MMAs: QK of tile j + 1 before
// PV of tile j.  256 tensor-memory columns (S 128, P 64, O 64) and 81 KB of shared memory: two CTAs share an SM,
// and one's exponentials run while the other waits for its MMAs.
//
// Bound by the exponentials: 128 x 128 of them take 1,024 cycles of the SM's special function units
// against 512 cycles of MMAs (2.1 M multiply-adds of a tile pair at 4,096 a cycle).  The products went through
// HBM before (fp32 scores and bf16 probabilities of one head at a time): 4.1 ms a layer of 8,580 patches x
// 16 heads.
//
// Every mbarrier wait is bounded; on a time-out the CTA raises its abort flag, reports TF_TIMEOUT, lets
// copies in flight land, frees its tensor memory and returns.
// (reference: src/vision.rs:481 encode, attention of kernels/vision.cu.)
#include "tc.cuh"

namespace {

constexpr int kTile = 128;                          // query rows of a CTA and keys of a tile
constexpr int kTileBytes = kTile * 128;             // 128 rows of 64 bf16
constexpr int kRing = 2;
constexpr int kVaThreads = 6 * 32;                  // 4 softmax warps, MMA warp, TMA warp
constexpr int kVaSmem = kTileBytes * (1 + 2 * kRing) + 1024 + 256;
constexpr int kVaCols = 256;
constexpr float kVaNeg = -1e30f;

struct VisAttnParams {
  __nv_bfloat16* out;
  int n, n_pad, ldo;
  float scale_log2;
  TfStatusWord* st;
};

__device__ __forceinline__ void tmem_st_x32(uint32_t taddr, const uint32_t v[32]) {
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t v[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t v[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// V tile as the MN-major B operand: 64 dims = the 128 swizzled bytes of a row, 8 keys = one 1,024-byte group
__device__ __forceinline__ uint64_t v_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
// D[tmem] (+)= A[tmem] * B[smem]: row i of A is lane i, two bf16 per 32-bit column; ONE thread issues
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__global__ void __launch_bounds__(kVaThreads, 2)
vis_attn_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                const __grid_constant__ CUtensorMap mapV, const VisAttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* tail = smem_raw + (base - raw) + kTileBytes * (1 + 2 * kRing);
  const uint32_t q_s = base, k_s = base + kTileBytes, v_s = k_s + kRing * kTileBytes;
  const uint32_t bar0 = v_s + kRing * kTileBytes;
  const uint32_t q_full = bar0, s_ready = bar0 + 8, p_ready = bar0 + 16, o_done = bar0 + 24, s_free = bar0 + 112;
  auto k_full = [&](int s) { return bar0 + 32u + 8u * s; };
  auto k_empty = [&](int s) { return bar0 + 48u + 8u * s; };
  auto v_full = [&](int s) { return bar0 + 64u + 8u * s; };
  auto v_empty = [&](int s) { return bar0 + 80u + 8u * s; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail + 96);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 104);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tc::mbar_init(q_full, 1);
    tc::mbar_init(s_ready, 1);
    tc::mbar_init(p_ready, 4);
    tc::mbar_init(s_free, 4);
    tc::mbar_init(o_done, 1);
    for (int s = 0; s < kRing; ++s) {
      tc::mbar_init(k_full(s), 1);
      tc::mbar_init(k_empty(s), 1);
      tc::mbar_init(v_full(s), 1);
      tc::mbar_init(v_empty(s), 1);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 4) tc::tmem_alloc(tc::smem_u32(const_cast<uint32_t*>(tmem_slot)), kVaCols);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tS = *tmem_slot, tP = tS + 128u, tO = tS + 192u;
  tf_pdl_sync();
  const int row0 = blockIdx.x * kTile, hrow = blockIdx.y * p.n_pad;
  const int tiles = (p.n + kTile - 1) / kTile;

  if (warp == 5) {
    // ------------------------------------------------------------------ TMA producer
    if (tc::elect_one()) {
      tc::mbar_expect_tx(q_full, kTileBytes);
      tc::tma_load_2d(q_s, &mapQ, 0, hrow + row0, q_full);
      for (int j = 0; j < tiles; ++j) {
        const int s = j % kRing;
        const uint32_t ph = ((j / kRing) & 1) ^ 1;
        if (!tc::mbar_wait(k_empty(s), ph, abort_flag)) break;
        tc::mbar_expect_tx(k_full(s), kTileBytes);
        tc::tma_load_2d(k_s + s * kTileBytes, &mapK, 0, hrow + j * kTile, k_full(s));
        if (!tc::mbar_wait(v_empty(s), ph, abort_flag)) break;
        tc::mbar_expect_tx(v_full(s), kTileBytes);
        tc::tma_load_2d(v_s + s * kTileBytes, &mapV, 0, hrow + j * kTile, v_full(s));
      }
    }
  } else if (warp == 4) {
    // ------------------------------------------------------------------ MMA issuer
    if (tc::elect_one()) {
      constexpr uint32_t idesc_qk = tc::instr_desc(1, 1, 128, 128);
      constexpr uint32_t idesc_pv = tc::instr_desc(1, 1, 128, 64) | (1u << 16);       // B MN-major
      auto qk = [&](int j) -> bool {
        const int s = j % kRing;
        if (!tc::mbar_wait(k_full(s), (j / kRing) & 1, abort_flag)) return false;
        tc::tc_fence_after();
        const uint64_t da = tc::smem_desc_sw128(q_s), db = tc::smem_desc_sw128(k_s + s * kTileBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k) tc::mma_f16(tS, da + 2 * k, db + 2 * k, idesc_qk, k ? 1u : 0u);
        tc::mma_commit(s_ready);
        tc::mma_commit(k_empty(s));
        return true;
      };
      bool ok = tc::mbar_wait(q_full, 0, abort_flag) && qk(0);
      for (int j = 0; j < tiles && ok; ++j) {
        const int s = j % kRing;
        // S of tile j has been read: QK of the next tile; then PV once P of tile j is in tensor memory
        if (j + 1 < tiles && !(ok = tc::mbar_wait(s_free, j & 1, abort_flag) && qk(j + 1))) break;
        if (!(ok = tc::mbar_wait(p_ready, j & 1, abort_flag))) break;
        if (!(ok = tc::mbar_wait(v_full(s), (j / kRing) & 1, abort_flag))) break;
        tc::tc_fence_after();
        const uint64_t dv = v_desc(v_s + s * kTileBytes);
#pragma unroll
        for (int k = 0; k < 8; ++k) mma_ts(tO, tP + 8 * k, dv + 128u * k, idesc_pv, (j | k) ? 1u : 0u);
        tc::mma_commit(o_done);
        tc::mma_commit(v_empty(s));
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: one row per thread
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    bool fail = false;
    // after a time-out the warp stops waiting and runs out its loop: the launch's result is void
    auto wait = [&](uint32_t bar, uint32_t parity) {
      if (!fail && !tc::mbar_wait(bar, parity, abort_flag)) fail = true;
      __syncwarp();
    };
    float m = kVaNeg, l = 0.f;
    for (int j = 0; j < tiles; ++j) {
      const int valid = p.n - j * kTile;
      wait(s_ready, j & 1);
      tc::tc_fence_after();
      // The whole row of S comes into registers at once, so QK of the next tile can overwrite it while this
      // one is exponentiated.
      uint32_t v[128];
#pragma unroll
      for (int q = 0; q < 4; ++q) tc::tmem_ld32(tS + lane_off + q * 32, v + q * 32);
      tc::tmem_ld_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(s_free);
      if (valid < kTile) {
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i >= valid) v[i] = __float_as_uint(-INFINITY);
      }
      float c0 = kVaNeg, c1 = kVaNeg, c2 = kVaNeg, c3 = kVaNeg;
#pragma unroll
      for (int i = 0; i < 128; i += 4) {
        c0 = fmaxf(c0, __uint_as_float(v[i]));
        c1 = fmaxf(c1, __uint_as_float(v[i + 1]));
        c2 = fmaxf(c2, __uint_as_float(v[i + 2]));
        c3 = fmaxf(c3, __uint_as_float(v[i + 3]));
      }
      const float cm = fmaxf(fmaxf(c0, c1), fmaxf(c2, c3)) * p.scale_log2;
      if (j == 0) {
        m = cm;
      } else if (__any_sync(0xffffffffu, cm > m + 8.f)) {
        // rare: the maximum moves; O and l are rescaled once the PV before is done
        const float nm = fmaxf(m, cm), f = exp2f(m - nm);
        m = nm;
        l *= f;
        wait(o_done, (j & 1) ^ 1);
        tc::tc_fence_after();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint32_t o[8];
          tmem_ld8(tO + lane_off + q * 8, o);
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          tmem_st8(tO + lane_off + q * 8, o);
        }
      }
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float x0 = __uint_as_float(v[q * 64 + 2 * i]), x1 = __uint_as_float(v[q * 64 + 2 * i + 1]);
          const float a = exp2f(fmaf(x0, p.scale_log2, -m)), b = exp2f(fmaf(x1, p.scale_log2, -m));
          ls[(2 * i) & 3] += a;
          ls[(2 * i + 1) & 3] += b;
          pk[i] = pack_bf16(a, b);
        }
        // P may be overwritten once the PV before has read it
        if (q == 0 && j > 0) wait(o_done, (j & 1) ^ 1);
        tmem_st_x32(tP + lane_off + q * 32, pk);
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      tmem_st_done();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(p_ready);
    }
    wait(o_done, (tiles - 1) & 1);
    tc::tc_fence_after();
    const int row = row0 + warp * 32 + lane;
    const float inv = 1.f / l;
    __nv_bfloat16* dst = p.out + (long)row * p.ldo + blockIdx.y * 64;
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      uint32_t o[32];
      tc::tmem_ld32(tO + lane_off + q * 32, o);
      tc::tmem_ld_wait();
      if (row < p.n) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            w[e] = pack_bf16(__uint_as_float(o[8 * i + 2 * e]) * inv, __uint_as_float(o[8 * i + 2 * e + 1]) * inv);
          *reinterpret_cast<uint4*>(dst + q * 32 + i * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // whichever role gave up (the producer may have issued its last copy and left before): copies in flight land
    // before the shared memory goes back
    const long long t0 = clock64();
    while (clock64() - t0 < 400000) {}
    if (threadIdx.x == 0) tf_report(p.st, TF_TIMEOUT, 160, blockIdx.x, blockIdx.y);
  }
  if (warp == 4) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tS, kVaCols);
  }
}

}  // namespace

// q, k, v [heads][n_pad][64] bf16 (16-byte aligned; n_pad a multiple of 128; rows n.. of k and v finite)
// -> out[row, head * 64 + c] (bf16, ldo elements per row, a multiple of 8) = softmax(scale q k^T) v for row < n
TF_API int tf_vis_attention(const void* q, const void* k, const void* v, void* out, int n, int n_pad, int heads, int ldo,
                            float scale, void* status, cudaStream_t st) {
  if (n <= 0 || heads <= 0 || heads > 65535 || n_pad % kTile || n > n_pad || ldo % 8 || !q || !k || !v || !out ||
      (reinterpret_cast<uintptr_t>(out) & 15))
    return -1;
  CUtensorMap mq, mk, mv;
  const uint64_t rows = (uint64_t)heads * n_pad;
  if (!tc::make_map_2d(&mq, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, 64, 128, kTile) ||
      !tc::make_map_2d(&mk, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, 64, 128, kTile) ||
      !tc::make_map_2d(&mv, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, 64, 128, kTile))
    return -4;
  static unsigned long long limit_set = 0;
  if (tf_smem_limit((const void*)vis_attn_kernel, kVaSmem, &limit_set) != cudaSuccess) return -2;
  VisAttnParams p = {(__nv_bfloat16*)out, n, n_pad, ldo, scale * 1.4426950408889634f, (TfStatusWord*)status};
  tf_launch(vis_attn_kernel, dim3((n + kTile - 1) / kTile, heads), dim3(kVaThreads), kVaSmem, st, mq, mk, mv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
