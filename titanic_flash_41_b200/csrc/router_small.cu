// Router logits of the decode step: logits[r, e] = sum_k x[r, k] * gate[e, k] for a few rows.
//
// The gate matrix is small (experts x hidden bf16, 2 MB at 256 x 4096), so the generic
// weight-streaming GEMV, which gives one CTA 32 output features, would run it on 8 CTAs and wait
// on memory latency.  Here one CTA owns two expert rows and its eight warps an eighth of the inputs
// each: every lane walks its part in 16-byte steps with one accumulator per expert and activation row (the rows
// come out of L1 / L2, once for both experts), the warps' partial sums meet in shared memory and
// are added by pairs.  Fixed summation order: bitwise reproducible.  Row counts up to 4 and 8 have
// forms of their own: with sixteen accumulators (and sixteen clamped loads) for any count, one expert
// and four warps a CTA, one row took 11 us and sixteen 12.4 us.
//
// Reference behaviour: router scores of kernels/moe_frontend.cuh (`ca_route_topk` takes these
// logits); the top-k itself stays in tf_router_topk.
#include <cuda_bf16.h>

#include "common.cuh"

namespace {

constexpr int kRouterWarps = 8, kRouterExperts = 2;

template <int ROWS>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_logits_small_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const __nv_bfloat16* __restrict__ gate,
                           float* __restrict__ out, int ldo, int T, int E, int d) {
  __shared__ float red[kRouterWarps][kRouterExperts][ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e0 = blockIdx.x * kRouterExperts;
  const uint4* wrow[kRouterExperts];
#pragma unroll
  for (int q = 0; q < kRouterExperts; ++q) wrow[q] = reinterpret_cast<const uint4*>(gate + (long)min(e0 + q, E - 1) * d);
  const int steps = d / 8;                                   // 16-byte steps of a row
  const int per = (steps + kRouterWarps - 1) / kRouterWarps, k_lo = warp * per, k_hi = min(steps, k_lo + per);
  // the first gate vectors (immutable) are requested before waiting for the kernel that writes x
  uint4 wnext[kRouterExperts];
#pragma unroll
  for (int q = 0; q < kRouterExperts; ++q)
    wnext[q] = k_lo + lane < k_hi ? __ldg(wrow[q] + k_lo + lane) : make_uint4(0u, 0u, 0u, 0u);
  tf_pdl_sync();
  for (int t0 = 0; t0 < T; t0 += ROWS) {
    float acc[kRouterExperts][ROWS];
#pragma unroll
    for (int q = 0; q < kRouterExperts; ++q)
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc[q][r] = 0.f;
    for (int k8 = k_lo + lane; k8 < k_hi; k8 += 32) {
      uint4 xv[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        xv[r] = __ldg(reinterpret_cast<const uint4*>(x + (long)min(t0 + r, T - 1) * ldx) + k8);
      float2 wf[kRouterExperts][4];
      const int kn = k8 + 32 < k_hi ? k8 + 32 : k_lo + lane;     // next step, or the first one for the next rows
#pragma unroll
      for (int q = 0; q < kRouterExperts; ++q) {
        const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wnext[q]);
#pragma unroll
        for (int j = 0; j < 4; ++j) wf[q][j] = __bfloat1622float2(wp[j]);
        wnext[q] = __ldg(wrow[q] + kn);
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&xv[r]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 xf = __bfloat1622float2(xp[j]);
#pragma unroll
          for (int q = 0; q < kRouterExperts; ++q) {
            acc[q][r] = fmaf(wf[q][j].x, xf.x, acc[q][r]);
            acc[q][r] = fmaf(wf[q][j].y, xf.y, acc[q][r]);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kRouterExperts; ++q)
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float v = warp_sum(acc[q][r]);
        if (lane == 0) red[warp][q][r] = v;
      }
    __syncthreads();
    if (threadIdx.x < kRouterExperts * ROWS) {
      const int q = threadIdx.x / ROWS, r = threadIdx.x % ROWS;
      if (t0 + r < T && e0 + q < E) {
        // by pairs: a chain over eight warps rounds more than one over four
        float v[kRouterWarps];
#pragma unroll
        for (int w = 0; w < kRouterWarps; ++w) v[w] = red[w][q][r];
#pragma unroll
        for (int o = kRouterWarps / 2; o > 0; o >>= 1)
#pragma unroll
          for (int w = 0; w < o; ++w) v[w] += v[w + o];
        out[(long)(t0 + r) * ldo + e0 + q] = v[0];
      }
    }
    __syncthreads();
  }
}

}  // namespace

// x [T, d] bf16 (row pitch ldx elements), gate [E, d] bf16, out [T, E] f32 (row pitch ldo)
TF_API int tf_router_logits_small(const void* x, int ldx, const void* gate, void* out, int ldo, int T, int E, int d,
                                  cudaStream_t st) {
  if (T <= 0 || d % 8 || ldx % 8) return -1;
  auto kernel = T <= 4 ? router_logits_small_kernel<4> : T <= 8 ? router_logits_small_kernel<8> : router_logits_small_kernel<16>;
  tf_launch(kernel, dim3((E + kRouterExperts - 1) / kRouterExperts), dim3(kRouterWarps * 32), 0, st,
            reinterpret_cast<const __nv_bfloat16*>(x), ldx, reinterpret_cast<const __nv_bfloat16*>(gate),
            reinterpret_cast<float*>(out), ldo, T, E, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
