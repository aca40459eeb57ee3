// Sublayer boundary of decode rows with its neighbours folded in: one launch does
//   [combine]  delta[r, :] = sum_j wts[r, j] * y_pair[r * topk + j, :] (experts of this rank, in
//              slot order) + shared[r, :]                 -- what tf_moe_combine would have written
//   [residual] x[r, :] = bf16(x[r, :] + delta[r, :])
//   [norm]     v = bf16(x * rsqrt(mean(x^2) + eps) * w)   -> f16 and / or bf16 copies
//   [mx8]      the MXFP8 form of v (e4m3 + one UE8M0 scale per 32) for the block-scaled expert GEMV
// The arithmetic is that of tf_moe_combine + tf_add_norm + tf_quant_rows_mx8 run one after the
// other (same order of additions, same roundings), so results are bit-identical; what goes away
// is two launches and two dependent-launch gaps per layer of a captured decode step.
//
// Reference behaviour: the FFN sum with the shared expert (kernels/ffn_sum_shared.cuh:7-33), the
// residual RMSNorm (kernels/core.cu:851 ca_rms_bf16) and the MXFP8 K32 activation quantisation of
// the MoE front-end (kernels/moe_frontend.cuh).
#include <limits.h>

#include "rownorm.cuh"

namespace {

struct FusedNormParams {
  __nv_bfloat16* x;            // [T, d] residual stream, updated in place
  const float* delta;          // [T, d] fp32 or null
  const float* y_pair;         // combine source (null: use delta)
  const int* ids;
  const float* wts;
  const float* shared_y;       // may be null
  int topk, e_lo, e_hi;
  const __nv_bfloat16* w;      // [d]
  __half* h16;
  __nv_bfloat16* hb;
  uint8_t* x8;                 // [T, d] e4m3 or null
  uint8_t* x8s;                // [T, d / 32] UE8M0
  int d;
  float eps;
};

__global__ void __launch_bounds__(1024) fused_norm_kernel(const FusedNormParams p) {
  tf_pdl_sync();
  extern __shared__ float row[];            // d floats
  __shared__ float scratch[32];
  const int r = blockIdx.x, d = p.d;
  __nv_bfloat16* xr = p.x + (long)r * d;
  float ss = 0.f;
  // four consecutive elements per thread and step: 16-byte loads of the expert outputs, all
  // independent, so a row's 7 x 16 KB of inputs are in flight at once
  for (int i = threadIdx.x * 4; i < d; i += blockDim.x * 4) {
    const uint2 xraw = *reinterpret_cast<const uint2*>(xr + i);
    const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&xraw);
    const float2 x01 = __bfloat1622float2(xb[0]), x23 = __bfloat1622float2(xb[1]);
    float v[4] = {x01.x, x01.y, x23.x, x23.y};
    bool add = false;
    float dv[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.y_pair) {
      for (int j = 0; j < p.topk; ++j) {
        const int e = p.ids[r * p.topk + j];
        if (e >= p.e_lo && e < p.e_hi) {
          const float wj = p.wts[r * p.topk + j];
          const float4 y = *reinterpret_cast<const float4*>(p.y_pair + (long)(r * p.topk + j) * d + i);
          dv[0] = fmaf(wj, y.x, dv[0]);
          dv[1] = fmaf(wj, y.y, dv[1]);
          dv[2] = fmaf(wj, y.z, dv[2]);
          dv[3] = fmaf(wj, y.w, dv[3]);
        }
      }
      if (p.shared_y) {
        const float4 y = *reinterpret_cast<const float4*>(p.shared_y + (long)r * d + i);
        dv[0] += y.x; dv[1] += y.y; dv[2] += y.z; dv[3] += y.w;
      }
      add = true;
    } else if (p.delta) {
      const float4 y = *reinterpret_cast<const float4*>(p.delta + (long)r * d + i);
      dv[0] = y.x; dv[1] = y.y; dv[2] = y.z; dv[3] = y.w;
      add = true;
    }
    if (add) {
#pragma unroll
      for (int c = 0; c < 4; ++c) v[c] = bf16_round(v[c] + dv[c]);
      __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
      *reinterpret_cast<uint2*>(xr + i) = *reinterpret_cast<uint2*>(o);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      row[i + c] = v[c];
      ss += v[c] * v[c];
    }
  }
  ss = block_sum(ss, scratch);
  row_norm_store(row, d, ss, p.eps, p.w, p.h16, p.hb, p.x8, p.x8s, r);
}

// The same for d <= 4096: one piece of four consecutive elements per thread, kept in registers from the residual to the MXFP8
// row (32 inputs = eight neighbouring threads).  Bound by the latency of its dependent loads: the expert ids and
// weights of a row are requested together and then all its expert rows, the norm's weight before the wait for the
// kernel before, and nothing goes through shared memory but the sum of squares.  With the loads one behind the other
// and 32-lane reductions of four groups in turn a decode row of 4096 took 5.7 us.  Same arithmetic, same order.
constexpr int kNormTopk = 8;                 // experts whose rows are in flight at once
__global__ void __launch_bounds__(1024) fused_norm_row_kernel(const FusedNormParams p) {
  const int i = threadIdx.x * 4;
  const uint2 wraw = __ldg(reinterpret_cast<const uint2*>(p.w + i));
  tf_pdl_sync();
  __shared__ float scratch[32];
  const long r = blockIdx.x;
  const int d = p.d;
  __nv_bfloat16* xr = p.x + r * d;
  const uint2 xraw = *reinterpret_cast<const uint2*>(xr + i);
  float dv[4] = {0.f, 0.f, 0.f, 0.f};
  const bool add = p.y_pair || p.delta;
  if (p.y_pair) {
    float4 sh = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.shared_y) sh = *reinterpret_cast<const float4*>(p.shared_y + r * d + i);
    for (int j0 = 0; j0 < p.topk; j0 += kNormTopk) {
      int e[kNormTopk];
      float w[kNormTopk];
      float4 y[kNormTopk];
#pragma unroll
      for (int j = 0; j < kNormTopk; ++j) {
        const bool in = j0 + j < p.topk;
        e[j] = in ? p.ids[r * p.topk + j0 + j] : -1;
        w[j] = in ? p.wts[r * p.topk + j0 + j] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < kNormTopk; ++j) {
        const bool in = j0 + j < p.topk && e[j] >= p.e_lo && e[j] < p.e_hi;
        if (in) y[j] = *reinterpret_cast<const float4*>(p.y_pair + (r * p.topk + j0 + j) * d + i);
        else e[j] = INT_MIN;
      }
#pragma unroll
      for (int j = 0; j < kNormTopk; ++j)
        if (e[j] != INT_MIN) {
          dv[0] = fmaf(w[j], y[j].x, dv[0]);
          dv[1] = fmaf(w[j], y[j].y, dv[1]);
          dv[2] = fmaf(w[j], y[j].z, dv[2]);
          dv[3] = fmaf(w[j], y[j].w, dv[3]);
        }
    }
    if (p.shared_y) {
      dv[0] += sh.x; dv[1] += sh.y; dv[2] += sh.z; dv[3] += sh.w;
    }
  } else if (p.delta) {
    const float4 y = *reinterpret_cast<const float4*>(p.delta + r * d + i);
    dv[0] = y.x; dv[1] = y.y; dv[2] = y.z; dv[3] = y.w;
  }
  const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&xraw);
  const float2 x01 = __bfloat1622float2(xb[0]), x23 = __bfloat1622float2(xb[1]);
  float v[4] = {x01.x, x01.y, x23.x, x23.y};
  if (add) {
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = bf16_round(v[c] + dv[c]);
    __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
    *reinterpret_cast<uint2*>(xr + i) = *reinterpret_cast<uint2*>(o);
  }
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) ss += v[c] * v[c];
  ss = block_sum(ss, scratch);
  const float inv = rsqrtf(ss / (float)d + p.eps);
  const __nv_bfloat162* wb = reinterpret_cast<const __nv_bfloat162*>(&wraw);
  const float2 w01 = __bfloat1622float2(wb[0]), w23 = __bfloat1622float2(wb[1]);
  const float g[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
  for (int c = 0; c < 4; ++c) v[c] = bf16_round(v[c] * inv * g[c]);
  __half hv[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) hv[c] = __float2half(v[c]);
  if (p.h16) *reinterpret_cast<uint2*>(p.h16 + r * d + i) = *reinterpret_cast<uint2*>(hv);
  if (p.hb) {
    __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
    *reinterpret_cast<uint2*>(p.hb + r * d + i) = *reinterpret_cast<uint2*>(o);
  }
  if (p.x8) {
    float amax = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      v[c] = __half2float(hv[c]);                        // values as the f16 copy holds them
      amax = fmaxf(amax, fabsf(v[c]));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    int ex = -127;
    if (amax > 0.f) {
      int e2;
      const float m = frexpf(amax * (1.f / 448.f), &e2);
      ex = max(-127, min(127, (m == 0.5f) ? e2 - 1 : e2));
    }
    const float q = exp2f((float)-ex);
    uint32_t b = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      b |= (uint32_t)__nv_cvt_float_to_fp8(v[c] * q, __NV_SATFINITE, __NV_E4M3) << (8 * c);
    *reinterpret_cast<uint32_t*>(p.x8 + r * d + i) = b;
    if ((threadIdx.x & 7) == 0) p.x8s[r * (d / 32) + i / 32] = (uint8_t)(ex + 127);
  }
}

// RMSNorm of R columns of a projection's rows (fp32 or bf16) -> f16 rows [T, R].  One CTA per row; the row is
// read twice (the second time from L1).  Replaces seven elementwise library launches.
template <typename P>
__global__ void __launch_bounds__(256) rms_cols_kernel(const P* __restrict__ x, long ldx, const __nv_bfloat16* __restrict__ w,
                                                       __half* __restrict__ out, int R, float eps) {
  tf_pdl_sync();
  __shared__ float scratch[32];
  const P* row = x + (long)blockIdx.x * ldx;
  float ss = 0.f;
  for (int i = threadIdx.x; i < R; i += blockDim.x) {
    const float v = (float)row[i];
    ss += v * v;
  }
  const float inv = rsqrtf(block_sum(ss, scratch) / (float)R + eps);
  for (int i = threadIdx.x; i < R; i += blockDim.x)
    out[(long)blockIdx.x * R + i] = __float2half((float)row[i] * inv * __bfloat162float(w[i]));
}

// out = bf16(x + delta): the finished residual rows (eight elements a thread)
__global__ void __launch_bounds__(256) residual_rows_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ delta,
                                                            __nv_bfloat16* __restrict__ out, long n) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  const uint4 raw = *reinterpret_cast<const uint4*>(x + i);
  const float4 a = *reinterpret_cast<const float4*>(delta + i), b = *reinterpret_cast<const float4*>(delta + i + 4);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  const float2 x0 = __bfloat1622float2(h[0]), x1 = __bfloat1622float2(h[1]), x2 = __bfloat1622float2(h[2]), x3 = __bfloat1622float2(h[3]);
  __nv_bfloat162 o[4] = {__floats2bfloat162_rn(x0.x + a.x, x0.y + a.y), __floats2bfloat162_rn(x1.x + a.z, x1.y + a.w),
                         __floats2bfloat162_rn(x2.x + b.x, x2.y + b.y), __floats2bfloat162_rn(x3.x + b.z, x3.y + b.w)};
  *reinterpret_cast<uint4*>(out + i) = *reinterpret_cast<uint4*>(o);
}

}  // namespace

// x [T rows of R columns, pitch ldx elements] (x_kind 0 fp32, 2 bf16), w [R] bf16 -> out [T, R] f16
TF_API int tf_rms_cols(const void* x, int x_kind, long ldx, const void* w, void* out, int T, int R, float eps,
                       cudaStream_t st) {
  if (T <= 0 || R <= 0 || !x || !w || !out) return T <= 0 ? 0 : -1;
  if (x_kind == 0) tf_launch(rms_cols_kernel<float>, dim3(T), dim3(256), 0, st, (const float*)x, ldx, (const __nv_bfloat16*)w, (__half*)out, R, eps);
  else if (x_kind == 2) tf_launch(rms_cols_kernel<__nv_bfloat16>, dim3(T), dim3(256), 0, st, (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, (__half*)out, R, eps);
  else return -1;
  return (int)cudaGetLastError();
}

// out[i] = bf16(x[i] + delta[i]), i < n (a multiple of 8; 16-byte aligned)
TF_API int tf_residual_rows(const void* x, const float* delta, void* out, long n, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8 || (((uintptr_t)x | (uintptr_t)delta | (uintptr_t)out) & 15)) return -1;
  tf_launch(residual_rows_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, st, (const __nv_bfloat16*)x, delta,
            (__nv_bfloat16*)out, n);
  return (int)cudaGetLastError();
}

// Exactly one of (delta) / (y_pair, ids, wts[, shared_y]) / neither feeds the residual add.
TF_API int tf_add_norm_fused(void* x, const void* delta, const void* y_pair, const int* ids, const void* wts,
                             const void* shared_y, int topk, int e_lo, int e_hi, const void* w, void* h16, void* hb,
                             void* x8, void* x8s, int T, int d, float eps, cudaStream_t st) {
  if (d % 128 || T <= 0 || (y_pair && (!ids || !wts || topk <= 0)) || (x8 && !x8s)) return -1;
  FusedNormParams p;
  p.x = (__nv_bfloat16*)x; p.delta = (const float*)delta; p.y_pair = (const float*)y_pair; p.ids = ids;
  p.wts = (const float*)wts; p.shared_y = (const float*)shared_y; p.topk = topk; p.e_lo = e_lo; p.e_hi = e_hi;
  p.w = (const __nv_bfloat16*)w; p.h16 = (__half*)h16; p.hb = (__nv_bfloat16*)hb; p.x8 = (uint8_t*)x8;
  p.x8s = (uint8_t*)x8s; p.d = d; p.eps = eps;
  const uintptr_t a16 = (uintptr_t)delta | (uintptr_t)y_pair | (uintptr_t)shared_y;
  const uintptr_t a8 = (uintptr_t)x | (uintptr_t)w | (uintptr_t)h16 | (uintptr_t)hb;
  if (d <= 4096 && !(a16 & 15) && !(a8 & 7) && !((uintptr_t)x8 & 3)) {
    tf_launch(fused_norm_row_kernel, dim3(T), dim3(d / 4), 0, st, p);
    return (int)cudaGetLastError();
  }
  tf_launch(fused_norm_kernel, dim3(T), dim3(d >= 4096 ? 1024 : 256), d * sizeof(float), st, p);
  return (int)cudaGetLastError();
}
