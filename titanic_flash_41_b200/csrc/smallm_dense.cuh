// Dense form of the weight-streaming GEMM (FP8 with 128 x 128 block scales, or bf16; up to 32 rows), included by
// smallm_gemm.cu inside its anonymous namespace.  Fragments and per-block promotion are those described
// there (a lane's 16-byte weight load IS its part of the A fragment); what differs is how the stream is kept
// full:
//
//   * weights go through shared memory with 16-byte asynchronous copies.  Every lane copies exactly the
//     bytes it will read itself, so a stage needs no barrier, only the lane's own wait, and the ring (three 4 KB
//     stages a warp, two CTAs of eight warps an SM) holds 192 KB of requests an SM.  Held in registers the
//     same prefetch cost 228 of them: one CTA an SM and 4.0 TB/s on the FP8 head (129,280 x 4096, 132 us)
//     against 6.6 TB/s here (80 us); 4096 x 8192 for four rows: 11.2 -> 8.0 us.
//   * CTAs are persistent: the copies run ahead across output tiles, so neither the reduction over the
//     K-splitting warps nor the start of the next tile stops the stream.
//   * K blocks are dealt to the eight warps in turn (block b to warp b % 8): adjacent 128-byte pieces of a row are
//     requested together and a K of few blocks still keeps the warps even.
//   * up to four 8-row activation tiles per pass: 17 to 32 rows read the weights once, not twice.
//   * the dual (SwiGLU) form takes 16 features of both matrices as its two tiles.
//
// Grid: one CTA per tile up to the number of resident CTAs (two an SM for 16 rows or fewer, one beyond, where the
// accumulators of four row tiles need the registers); more tiles are walked with that stride.
struct DenseParams {
  const uint8_t *W, *W3;
  const float *S, *S3;       // FP8 block scales [N / 128][lds]
  int ldw, lds;
  const __half* X;           // f16 (bf16 for bf16 weights)
  int ldx;
  void* Y;
  int ldy, out_kind;
  int N, K, M, tiles;
  float swiglu_limit;
  int x_group_n;             // block-diagonal form: features [g x_group_n, (g + 1) x_group_n) read the K activations
  int x_group_stride;        // that start at column g x_group_stride (0: one group)
};

constexpr int kDenseWarps = 8;
constexpr int kDenseStage = 4096;                    // bytes of a warp's stage: 32 weight rows x 128 bytes

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int KIND, int MT, bool DUAL, int STAGES>
__global__ void __launch_bounds__(kDenseWarps * 32, MT <= 2 ? 2 : 1) smallm_dense_kernel(const DenseParams p) {
  constexpr int KB = KIND == 0 ? 128 : 64;           // k per 128-byte block
  constexpr int FT = DUAL ? 16 : 32;                 // features per tile
  constexpr int XV = KIND == 0 ? 2 : 1;              // 16-byte activation pieces per 64 bytes of weights
  extern __shared__ __align__(16) uint8_t dense_smem[];
  float* red = reinterpret_cast<float*>(dense_smem + kDenseWarps * STAGES * kDenseStage);   // [warp][tile][m][32][4]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint8_t* ring = dense_smem + warp * STAGES * kDenseStage + lane * 16;
  const uint32_t ring_s = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
  const int nb = p.K / KB;
  const int count = nb > warp ? (nb - warp + kDenseWarps - 1) / kDenseWarps : 0;     // this warp's blocks of a tile

  // ---- copies run ahead of the math: (i_tile, i_blk) is the next block to request
  int i_tile = blockIdx.x, i_blk = 0, i_stage = 0;
  auto issue = [&]() {
    if (count > 0 && i_tile < p.tiles) {
      const long row = (long)(i_tile * FT + g) * p.ldw + (warp + kDenseWarps * i_blk) * 128 + t * 16;
      const uint8_t* a = p.W + row;
      const uint8_t* b = DUAL ? p.W3 + row : a + 16L * p.ldw;
      const long r8 = 8L * p.ldw;
      const uint32_t dst = ring_s + i_stage * kDenseStage;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        cp_async16(dst + (s * 4 + 0) * 512, a + s * 64);
        cp_async16(dst + (s * 4 + 1) * 512, a + r8 + s * 64);
        cp_async16(dst + (s * 4 + 2) * 512, b + s * 64);
        cp_async16(dst + (s * 4 + 3) * 512, b + r8 + s * 64);
      }
      if (++i_blk == count) {
        i_blk = 0;
        i_tile += gridDim.x;
      }
    }
    cp_async_commit();                               // (an empty group keeps the count of groups uniform)
    i_stage = i_stage + 1 == STAGES ? 0 : i_stage + 1;
  };
#pragma unroll
  for (int s = 0; s < STAGES; ++s) issue();
  tf_pdl_sync();                                     // activations are the output of the kernel before this one

  const __half* xrow[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) xrow[m] = p.X + (long)min(m * 8 + g, p.M - 1) * p.ldx + t * (KIND == 0 ? 16 : 8);

  int c_stage = 0;
  for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    const int n0 = tile * FT;
    const int x0 = p.x_group_n ? n0 / p.x_group_n * p.x_group_stride : 0;
    float acc[2][MT][4];
#pragma unroll
    for (int ti = 0; ti < 2; ++ti)
#pragma unroll
      for (int m = 0; m < MT; ++m) acc[ti][m][0] = acc[ti][m][1] = acc[ti][m][2] = acc[ti][m][3] = 0.f;
    const float* S = KIND == 0 ? p.S + (long)(n0 >> 7) * p.lds : nullptr;
    const float* S3 = KIND == 0 && DUAL ? p.S3 + (long)(n0 >> 7) * p.lds : nullptr;
    for (int j = 0; j < count; ++j) {
      const int blk = warp + kDenseWarps * j, kb = blk * KB;
      uint4 xv[2][MT][XV];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int e = 0; e < XV; ++e)
            xv[s][m][e] = *reinterpret_cast<const uint4*>(xrow[m] + x0 + kb + s * (KB / 2) + e * 8);
      float sc = 1.f, sc3 = 1.f;
      if (KIND == 0) {
        sc = __ldg(S + blk);
        sc3 = DUAL ? __ldg(S3 + blk) : sc;
      }
      cp_async_wait<STAGES - 1>();
      const uint8_t* st = ring + c_stage * kDenseStage;
      float part[2][MT][4];
      if (KIND == 0) {
#pragma unroll
        for (int ti = 0; ti < 2; ++ti)
#pragma unroll
          for (int m = 0; m < MT; ++m) part[ti][m][0] = part[ti][m][1] = part[ti][m][2] = part[ti][m][3] = 0.f;
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
#pragma unroll
        for (int ti = 0; ti < 2; ++ti) {
          const uint4 w0 = *reinterpret_cast<const uint4*>(st + (s * 4 + ti * 2) * 512);
          const uint4 w8 = *reinterpret_cast<const uint4*>(st + (s * 4 + ti * 2 + 1) * 512);
          const uint32_t a0w[4] = {w0.x, w0.y, w0.z, w0.w}, a8w[4] = {w8.x, w8.y, w8.z, w8.w};
          if (KIND == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t a[4];
              a[0] = e4m3x2_to_h2((uint16_t)(a0w[q] & 0xffffu));
              a[1] = e4m3x2_to_h2((uint16_t)(a8w[q] & 0xffffu));
              a[2] = e4m3x2_to_h2((uint16_t)(a0w[q] >> 16));
              a[3] = e4m3x2_to_h2((uint16_t)(a8w[q] >> 16));
#pragma unroll
              for (int m = 0; m < MT; ++m) {
                const uint4 x = xv[s][m][(q >> 1) % XV];
                const uint32_t b[2] = {(q & 1) ? x.z : x.x, (q & 1) ? x.w : x.y};
                mma_f16_16816(part[ti][m], a, b);
              }
            }
          } else {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const uint32_t a[4] = {a0w[2 * q], a8w[2 * q], a0w[2 * q + 1], a8w[2 * q + 1]};
#pragma unroll
              for (int m = 0; m < MT; ++m) {
                const uint4 x = xv[s][m][0];
                const uint32_t b[2] = {q ? x.z : x.x, q ? x.w : x.y};
                mma_bf16_16816(acc[ti][m], a, b);
              }
            }
          }
        }
      }
      if (KIND == 0) {
#pragma unroll
        for (int ti = 0; ti < 2; ++ti)
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[ti][m][i] = fmaf(ti ? sc3 : sc, part[ti][m][i], acc[ti][m][i]);
      }
      c_stage = c_stage + 1 == STAGES ? 0 : c_stage + 1;
      issue();                                       // refills the stage just read
    }
    // ---- fixed-order reduction over the K-splitting warps, then the epilogue
#pragma unroll
    for (int ti = 0; ti < 2; ++ti)
#pragma unroll
      for (int m = 0; m < MT; ++m)
        *reinterpret_cast<float4*>(red + (((warp * 2 + ti) * MT + m) * 32 + lane) * 4) =
            make_float4(acc[ti][m][0], acc[ti][m][1], acc[ti][m][2], acc[ti][m][3]);
    __syncthreads();
    constexpr int kSlots = (DUAL ? 1 : 2) * MT * 128;
#pragma unroll 1
    for (int s = threadIdx.x; s < kSlots; s += kDenseWarps * 32) {
      const int i = s & 3, ln = (s >> 2) & 31, m = (s >> 7) % MT, ti = (s >> 7) / MT;
      float v = 0.f, v3 = 0.f;
#pragma unroll
      for (int w = 0; w < kDenseWarps; ++w) {
        v += red[(((w * 2 + ti) * MT + m) * 32 + ln) * 4 + i];
        if (DUAL) v3 += red[(((w * 2 + 1) * MT + m) * 32 + ln) * 4 + i];
      }
      // C fragment: weight row = g (+8 for i >= 2); activation row = 2t + (i & 1)
      const int n = n0 + 16 * ti + (ln >> 2) + ((i & 2) ? 8 : 0), r = m * 8 + 2 * (ln & 3) + (i & 1);
      if (r < p.M && n < p.N) {
        float o = v;
        if (DUAL) {
          float gate = v, up = v3;
          if (p.swiglu_limit > 0.f) {
            gate = fminf(gate, p.swiglu_limit);
            up = fminf(fmaxf(up, -p.swiglu_limit), p.swiglu_limit);
          }
          o = gate / (1.f + __expf(-gate)) * up;
        }
        const long off = (long)r * p.ldy + n;
        if (p.out_kind == 0) reinterpret_cast<float*>(p.Y)[off] = o;
        else if (p.out_kind == 1) reinterpret_cast<__half*>(p.Y)[off] = __float2half(o);
        else reinterpret_cast<__nv_bfloat16*>(p.Y)[off] = __float2bfloat16(o);
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
}

template <int KIND, int MT, bool DUAL>
cudaError_t launch_dense_mt(const DenseParams& p, int sms, cudaStream_t st) {
  constexpr int STAGES = MT <= 2 ? 3 : 5;
  constexpr int smem = kDenseWarps * STAGES * kDenseStage + kDenseWarps * 2 * MT * 512;
  auto kernel = smallm_dense_kernel<KIND, MT, DUAL, STAGES>;
  static unsigned long long limit_set = 0;
  const cudaError_t e = tf_smem_limit((const void*)kernel, smem, &limit_set);
  if (e != cudaSuccess) return e;
  const int resident = sms * (MT <= 2 ? 2 : 1);
  tf_launch(kernel, dim3(p.tiles < resident ? p.tiles : resident), dim3(kDenseWarps * 32), smem, st, p);
  return cudaGetLastError();
}

template <int KIND, bool DUAL>
cudaError_t launch_dense(DenseParams p, cudaStream_t st) {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  p.tiles = p.N / (DUAL ? 16 : 32);
  if (p.M <= 8) return launch_dense_mt<KIND, 1, DUAL>(p, sms, st);
  if (p.M <= 16) return launch_dense_mt<KIND, 2, DUAL>(p, sms, st);
  if (p.M <= 24) return launch_dense_mt<KIND, 3, DUAL>(p, sms, st);
  return launch_dense_mt<KIND, 4, DUAL>(p, sms, st);
}
