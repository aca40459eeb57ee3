// mHC boundary (multi-stream residual with hc_mult = H copies), H <= 4.
//
//   tf_hc_prepare   the H*(2+H) mixes of the flattened H x d row against `fn`
//                   (fp32 weights), all scaled by rsqrt(mean(x^2) + rms_eps); then
//                   pre_h = sigmoid(m_h*s0 + b_h) + eps, post_h = 2*sigmoid(m_{H+h}*s1 + b_{H+h}),
//                   comb = Sinkhorn(row-softmax + eps) (column step first, then iters-1 row/column
//                   pairs); finally the collapsed input v = sum_h pre_h * x_h (sequential fp32
//                   FMAs, rounded once to bf16) and, optionally, its RMSNorm in f16 / bf16 for the
//                   sublayer's first GEMM.  The coefficients stay in a small per-row record for
//                   tf_hc_post.
//   tf_hc_post      y_c = post_c * a + sum_k comb[k, c] * x_k for the sublayer output a.
// fp32 reference: the model oracle's hc_coefficients / hc_collapse / hc_post
// (reference arithmetic: kernels/core.cu:859-936, fused variant kernels/roce_oneshot_hc.cuh:52-63;
// Rust side src/mhc.rs:946 prepare, :1186 finish).
#include <cooperative_groups.h>

#include "common.cuh"

namespace {
constexpr int kMaxH = 4;
constexpr int kMaxMix = kMaxH * (2 + kMaxH);     // 24

struct HcCoef {                                    // per row, 32 floats
  float pre[kMaxH], post[kMaxH], comb[kMaxH * kMaxH], pad[8];
};

// One CTA per row, any width and alignment.  HEAD: the collapse in front of the vocabulary head (H mixes, no post / comb,
// bf16 values in both normalised rows) and the plain mean of the copies.
template <bool HEAD>
__global__ void __launch_bounds__(256) hc_prepare_kernel(const __nv_bfloat16* __restrict__ x,
                                                         const float* __restrict__ fn,
                                                         const float* __restrict__ base,
                                                         const float* __restrict__ scale, HcCoef* __restrict__ coef,
                                                         __nv_bfloat16* __restrict__ v_out,
                                                         __nv_bfloat16* __restrict__ mean,
                                                         const __nv_bfloat16* __restrict__ norm_w,
                                                         __half* __restrict__ h16, __nv_bfloat16* __restrict__ hb,
                                                         int H, int d, int iters, float eps, float rms_eps) {
  tf_pdl_sync();
  __shared__ float red[kMaxMix + 1][8];
  __shared__ float mix[kMaxMix + 1];
  __shared__ float s_pre[kMaxH];
  __shared__ float s_vv[8];
  const int r = blockIdx.x, nmix = HEAD ? H : H * (2 + H), n = H * d;
  const __nv_bfloat16* xr = x + (long)r * n;
  float acc[kMaxMix + 1];
#pragma unroll
  for (int q = 0; q <= kMaxMix; ++q) acc[q] = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) {
    const float a = __bfloat162float(xr[i]);
    acc[kMaxMix] += a * a;
#pragma unroll
    for (int q = 0; q < kMaxMix; ++q)
      if (q < nmix) acc[q] = fmaf(a, fn[(long)q * n + i], acc[q]);
  }
#pragma unroll
  for (int q = 0; q <= kMaxMix; ++q) {
    float t = acc[q];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = t;
  }
  __syncthreads();
  if (threadIdx.x <= kMaxMix) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
    mix[threadIdx.x] = t;
  }
  __syncthreads();
  if (HEAD) {
    if (threadIdx.x < H)
      s_pre[threadIdx.x] = 1.f / (1.f + expf(-(mix[threadIdx.x] * rsqrtf(mix[kMaxMix] / n + rms_eps) * scale[0] +
                                               base[threadIdx.x]))) + eps;
  } else if (threadIdx.x == 0) {
    const float inv = rsqrtf(mix[kMaxMix] / n + rms_eps);
    HcCoef c;
    for (int h = 0; h < H; ++h) {
      c.pre[h] = 1.f / (1.f + expf(-(mix[h] * inv * scale[0] + base[h]))) + eps;
      c.post[h] = 2.f / (1.f + expf(-(mix[H + h] * inv * scale[1] + base[H + h])));
      s_pre[h] = c.pre[h];
    }
    float m[kMaxH][kMaxH];
    for (int i = 0; i < H; ++i) {
      float mx = -1e30f, sum = 0.f;
      for (int j = 0; j < H; ++j) {
        m[i][j] = mix[2 * H + i * H + j] * inv * scale[2] + base[2 * H + i * H + j];
        mx = fmaxf(mx, m[i][j]);
      }
      for (int j = 0; j < H; ++j) {
        m[i][j] = expf(m[i][j] - mx);
        sum += m[i][j];
      }
      for (int j = 0; j < H; ++j) m[i][j] = m[i][j] / sum + eps;
    }
    auto cols = [&]() {
      for (int j = 0; j < H; ++j) {
        float s = 0.f;
        for (int i = 0; i < H; ++i) s += m[i][j];
        for (int i = 0; i < H; ++i) m[i][j] /= (s + eps);
      }
    };
    auto rows = [&]() {
      for (int i = 0; i < H; ++i) {
        float s = 0.f;
        for (int j = 0; j < H; ++j) s += m[i][j];
        for (int j = 0; j < H; ++j) m[i][j] /= (s + eps);
      }
    };
    cols();
    for (int it = 1; it < iters; ++it) {
      rows();
      cols();
    }
    for (int i = 0; i < H; ++i)
      for (int j = 0; j < H; ++j) c.comb[i * kMaxH + j] = m[i][j];
    coef[r] = c;
  }
  __syncthreads();
  // collapse (+ optional RMSNorm of the collapsed row)
  float vv = 0.f;
  for (int i = threadIdx.x; i < d; i += 256) {
    float v = 0.f;
    float m = 0.f;
    for (int h = 0; h < H; ++h) {
      const float a = __bfloat162float(xr[h * d + i]);
      v = fmaf(s_pre[h], a, v);
      m += a;
    }
    const __nv_bfloat16 vb = __float2bfloat16_rn(v);
    v_out[(long)r * d + i] = vb;
    if (HEAD && mean) mean[(long)r * d + i] = __float2bfloat16_rn(m / H);
    const float vr = __bfloat162float(vb);
    vv += vr * vr;
  }
  if (norm_w == nullptr) return;
#pragma unroll
  for (int o = 16; o; o >>= 1) vv += __shfl_xor_sync(0xffffffffu, vv, o);
  if ((threadIdx.x & 31) == 0) s_vv[threadIdx.x >> 5] = vv;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) tot += s_vv[w];
  const float inv = rsqrtf(tot / d + rms_eps);
  for (int i = threadIdx.x; i < d; i += 256) {
    float y = __bfloat162float(v_out[(long)r * d + i]) * inv * __bfloat162float(norm_w[i]);
    if (HEAD) y = bf16_round(y);
    if (h16) h16[(long)r * d + i] = __float2half(y);
    if (hb) hb[(long)r * d + i] = __float2bfloat16_rn(y);
  }
}

// ---------------------------------------------------------------------------------------------
// The same boundary by a cluster of eight CTAs for R rows.  CTA c of the cluster owns columns
// [c w, c w + w) of EVERY residual copy: its part of the mixes, and afterwards its columns of the
// collapsed and normalised rows, come from the one slice of x that it stages in shared memory, so x
// is read from HBM once.  Partial mixes and sums of squares meet through distributed shared memory
// (added in CTA order).  Warp q computes mixes 3q .. 3q + 2 of all R rows: a weight pair is loaded
// once for R rows, two columns per packed fp32 FMA.
//   R = 1   few rows (decode): bound by the latency of streaming fn (1.97 MB at 4 x 5120) from L2; eight
//           CTAs a row shorten the stream eightfold.  One CTA per row took 202 us for 24 rows; a decode
//           step with 14 of these and 6 head collapses (then a chain of library calls): 10.1 -> 6.8 ms
//   R = 16  many rows (prefill): fn crosses L2 once per 16 rows (one row per CTA moves 2 MB per row:
//           1.14 ms for 4,001 rows; four of these, four tf_hc_post and one head of a prefill: 58.2 ->
//           50.2 ms together with the scale re-ordering of csrc/gemm_mx.cu, 55.5 before)
// HEAD: the collapse in front of the vocabulary head (H mixes, no post / comb) and the plain mean
// of the copies.
// ---------------------------------------------------------------------------------------------
constexpr int kHcCtas = 8;

__device__ __forceinline__ unsigned long long pack_f2(float a, float b) {
  return ((unsigned long long)__float_as_uint(b) << 32) | __float_as_uint(a);
}
__device__ __forceinline__ void fma_f2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 bf2_to_f2(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

struct HcArgs {
  const __nv_bfloat16* x;
  const float *fn, *base, *scale;
  HcCoef* coef;
  __nv_bfloat16* v;
  __nv_bfloat16* mean;
  const __nv_bfloat16* norm_w;
  __half* h16;
  __nv_bfloat16* hb;
  int rows, H, d, w, iters;
  float eps, rms_eps;
};

template <int R, bool HEAD>
__global__ void __cluster_dims__(kHcCtas, 1, 1) __launch_bounds__(256) hc_cluster_kernel(const HcArgs p) {
  tf_pdl_sync();
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int kCols = kMaxMix + 1;
  extern __shared__ __align__(16) uint8_t hc_smem[];
  __shared__ float part[R][kCols];            // this CTA's partial mixes (last: sum of squares)
  __shared__ float mix[R][kCols];
  __shared__ float red[R][8];
  __shared__ float s_pre[R][kMaxH];
  __shared__ float vv[R];
  const int H = p.H, d = p.d, w = p.w, n = H * d, nmix = HEAD ? H : H * (2 + H);
  __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(hc_smem);          // [R][H][w]
  const int c = (int)cluster.block_rank();
  const int row0 = (int)(blockIdx.x / kHcCtas) * R;
  const int c0 = c * w, wc = max(0, min(w, d - c0));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  // ---- stage this CTA's columns of the rows (16-byte pieces), sums of squares on the way
  const int w8 = wc / 8;
  if (R == 1) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < H * w8; i += 256) {
      const int h = i / w8, k = (i - h * w8) * 8;
      const uint4 raw = *reinterpret_cast<const uint4*>(p.x + (long)row0 * n + (long)h * d + c0 + k);
      *reinterpret_cast<uint4*>(xs + h * w + k) = raw;
      const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = bf2_to_f2(u[j]);
        ss += f.x * f.x + f.y * f.y;
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) red[0][warp] = ss;
  } else {
    for (int r = warp; r < R; r += 8) {
      float ss = 0.f;
      const bool live = row0 + r < p.rows;
      for (int i = lane; i < H * w8; i += 32) {
        const int h = i / w8, k = (i - h * w8) * 8;
        uint4 raw = make_uint4(0u, 0u, 0u, 0u);
        if (live) raw = *reinterpret_cast<const uint4*>(p.x + (long)(row0 + r) * n + (long)h * d + c0 + k);
        *reinterpret_cast<uint4*>(xs + (r * H + h) * w + k) = raw;
        const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = bf2_to_f2(u[j]);
          ss += f.x * f.x + f.y * f.y;
        }
      }
      ss = warp_sum(ss);
      if (lane == 0) part[r][kMaxMix] = ss;
    }
  }
  __syncthreads();
  if (R == 1 && threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += red[0][q];
    part[0][kMaxMix] = t;
  }

  // ---- mixes 3 warp .. 3 warp + 2 over this CTA's columns
  {
    unsigned long long acc[3][R];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[m][r] = 0ull;
    const int q0 = warp * 3;
    if (q0 < nmix) {
      for (int h = 0; h < H; ++h) {
        const float* f0 = p.fn + (long)h * d + c0;
        const __nv_bfloat16* xh = xs + h * w;
#pragma unroll(R == 1 ? 5 : 1)
        for (int i = lane * 2; i < wc; i += 64) {
          unsigned long long f[3];
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int q = min(q0 + m, nmix - 1);
            const float2 t = __ldg(reinterpret_cast<const float2*>(f0 + (long)q * n + i));
            f[m] = pack_f2(t.x, t.y);
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float2 a = bf2_to_f2(*reinterpret_cast<const uint32_t*>(xh + (long)r * H * w + i));
            const unsigned long long a2 = pack_f2(a.x, a.y);
#pragma unroll
            for (int m = 0; m < 3; ++m) fma_f2(acc[m][r], f[m], a2);
          }
        }
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float t = warp_sum(__uint_as_float((uint32_t)acc[m][r]) + __uint_as_float((uint32_t)(acc[m][r] >> 32)));
          if (lane == 0 && q0 + m < nmix) part[r][q0 + m] = t;
        }
    }
  }
  cluster.sync();
  for (int i = threadIdx.x; i < R * kCols; i += 256) {
    const int q = i % kCols;
    if (q >= nmix && q != kMaxMix) continue;
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < kHcCtas; ++k) t += cluster.map_shared_rank(&part[0][0], k)[i];
    (&mix[0][0])[i] = t;
  }
  __syncthreads();

  // ---- coefficients: one warp per row; lane i * 4 + j of the first sixteen holds comb[i][j] (the
  // other sixteen repeat them, so that every shuffle is by whole warps)
  for (int r = warp; r < R; r += 8) {
    const float inv = rsqrtf(mix[r][kMaxMix] / n + p.rms_eps);
    float pre = 0.f, post = 0.f;
    if (lane < H) {
      pre = 1.f / (1.f + expf(-(mix[r][lane] * inv * p.scale[0] + p.base[lane]))) + p.eps;
      if (!HEAD) post = 2.f / (1.f + expf(-(mix[r][H + lane] * inv * p.scale[1] + p.base[H + lane])));
      s_pre[r][lane] = pre;
    }
    if (!HEAD) {
      const int i = (lane >> 2) & 3, j = lane & 3;
      const bool on = i < H && j < H;
      const int q = on ? 2 * H + i * H + j : 0;
      const float m0 = on ? mix[r][q] * inv * p.scale[2] + p.base[q] : -1e30f;
      float mx = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      float m = on ? expf(m0 - mx) : 0.f;
      auto row_sum = [&](float v) {
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        return v + __shfl_xor_sync(0xffffffffu, v, 2);
      };
      auto col_sum = [&](float v) {
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        return v + __shfl_xor_sync(0xffffffffu, v, 8);
      };
      const float s0 = row_sum(m);
      m = on ? m / s0 + p.eps : 0.f;
      const float s1 = col_sum(m);
      m = on ? m / (s1 + p.eps) : 0.f;
      for (int it = 1; it < p.iters; ++it) {
        const float sr = row_sum(m);
        m = on ? m / (sr + p.eps) : 0.f;
        const float sc = col_sum(m);
        m = on ? m / (sc + p.eps) : 0.f;
      }
      if (c == 0 && row0 + r < p.rows) {
        HcCoef* k = p.coef + row0 + r;
        if (lane < H) {
          k->pre[lane] = pre;
          k->post[lane] = post;
        }
        if (lane < 16 && on) k->comb[i * kMaxH + j] = m;
      }
    }
  }
  __syncthreads();

  // ---- collapse: this CTA's columns; the bf16 result replaces copy 0 in shared memory
  const bool norm = p.norm_w != nullptr;
  for (int r = R == 1 ? 0 : warp; r < R; r += 8) {
    const int gr = row0 + r;
    float pre[kMaxH];
#pragma unroll
    for (int h = 0; h < kMaxH; ++h) pre[h] = h < H ? s_pre[r][h] : 0.f;
    float ss = 0.f;
    __nv_bfloat16* xr = xs + (long)r * H * w;
    for (int i = (R == 1 ? (int)threadIdx.x : lane) * 2; i < wc; i += R == 1 ? 512 : 64) {
      float a = 0.f, b = 0.f, ma = 0.f, mb = 0.f;
#pragma unroll
      for (int h = 0; h < kMaxH; ++h)
        if (h < H) {
          const float2 f = bf2_to_f2(*reinterpret_cast<const uint32_t*>(xr + h * w + i));
          a = fmaf(pre[h], f.x, a);
          b = fmaf(pre[h], f.y, b);
          ma += f.x;
          mb += f.y;
        }
      const __nv_bfloat162 o = __floats2bfloat162_rn(a, b);
      *reinterpret_cast<__nv_bfloat162*>(xr + i) = o;
      if (gr < p.rows) {
        *reinterpret_cast<__nv_bfloat162*>(p.v + (long)gr * d + c0 + i) = o;
        if (HEAD && p.mean)
          *reinterpret_cast<__nv_bfloat162*>(p.mean + (long)gr * d + c0 + i) = __floats2bfloat162_rn(ma / H, mb / H);
      }
      const float2 fr = __bfloat1622float2(o);
      ss += fr.x * fr.x + fr.y * fr.y;
    }
    ss = warp_sum(ss);
    if (lane == 0) {
      if (R == 1) red[0][warp] = ss;
      else vv[r] = ss;
    }
  }
  if (R == 1) {
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) t += red[0][q];
      vv[0] = t;
    }
  }
  cluster.sync();                             // (also: nobody leaves before its partials have been read)
  if (norm) {
    for (int r = R == 1 ? 0 : warp; r < R; r += 8) {
      const int gr = row0 + r;
      float tot = 0.f;
#pragma unroll
      for (int k = 0; k < kHcCtas; ++k) tot += cluster.map_shared_rank(&vv[0], k)[r];
      if (gr >= p.rows) continue;
      const float inv = rsqrtf(tot / d + p.rms_eps);
      const __nv_bfloat16* xr = xs + (long)r * H * w;
      for (int i = (R == 1 ? (int)threadIdx.x : lane) * 2; i < wc; i += R == 1 ? 512 : 64) {
        const float2 f = bf2_to_f2(*reinterpret_cast<const uint32_t*>(xr + i));
        const float2 g = bf2_to_f2(*reinterpret_cast<const uint32_t*>(p.norm_w + c0 + i));
        float a = f.x * inv * g.x, b = f.y * inv * g.y;
        if (HEAD) {                           // the final norm hands out bf16 values (f16 copies of them)
          a = bf16_round(a);
          b = bf16_round(b);
        }
        if (p.h16) *reinterpret_cast<__half2*>(p.h16 + (long)gr * d + c0 + i) = __floats2half2_rn(a, b);
        if (p.hb) *reinterpret_cast<__nv_bfloat162*>(p.hb + (long)gr * d + c0 + i) = __floats2bfloat162_rn(a, b);
      }
    }
    cluster.sync();                           // the sums of squares have been read
  }
}

// grid (rows, H)
__global__ void __launch_bounds__(256) hc_post_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ a,
                                                      const HcCoef* __restrict__ coef,
                                                      __nv_bfloat16* __restrict__ y, int H, int d) {
  tf_pdl_sync();
  const int r = blockIdx.x, c = blockIdx.y;
  const HcCoef k = coef[r];
  const __nv_bfloat16* xr = x + (long)r * H * d;
  for (int i = threadIdx.x; i < d; i += 256) {
    float v = k.post[c] * a[(long)r * d + i];
    for (int q = 0; q < H; ++q) v = fmaf(k.comb[q * kMaxH + c], __bfloat162float(xr[q * d + i]), v);
    y[((long)r * H + c) * d + i] = __float2bfloat16_rn(v);
  }
}
// Eight columns per thread, all H outputs from one read of the H copies (the kernel above reads every
// copy once per output, two bytes a load): 4,001 rows of 4 x 5120 are 410 MB.
__global__ void __launch_bounds__(128) hc_post_vec_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const float* __restrict__ a,
                                                          const HcCoef* __restrict__ coef,
                                                          __nv_bfloat16* __restrict__ y, int H, int d) {
  tf_pdl_sync();
  const long r = blockIdx.y;
  const int i = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (i >= d) return;
  const HcCoef& k = coef[r];
  const float4 a0 = *reinterpret_cast<const float4*>(a + r * d + i), a1 = *reinterpret_cast<const float4*>(a + r * d + i + 4);
  const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
  uint4 raw[kMaxH];
#pragma unroll
  for (int h = 0; h < kMaxH; ++h)
    if (h < H) raw[h] = *reinterpret_cast<const uint4*>(x + (r * H + h) * d + i);
#pragma unroll
  for (int c = 0; c < kMaxH; ++c) {
    if (c >= H) break;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = k.post[c] * av[j];
#pragma unroll
    for (int q = 0; q < kMaxH; ++q)
      if (q < H) {
        const float kq = k.comb[q * kMaxH + c];
        const uint32_t u[4] = {raw[q].x, raw[q].y, raw[q].z, raw[q].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = bf2_to_f2(u[j]);
          v[2 * j] = fmaf(kq, f.x, v[2 * j]);
          v[2 * j + 1] = fmaf(kq, f.y, v[2 * j + 1]);
        }
      }
    __nv_bfloat162 o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    *reinterpret_cast<uint4*>(y + (r * H + c) * d + i) = *reinterpret_cast<uint4*>(o);
  }
}

inline bool aligned16(const void* a) { return !(reinterpret_cast<uintptr_t>(a) & 15); }

constexpr int kHcGeneral = -100;
// 0 or a CUDA error: launched; kHcGeneral: these rows need the general kernel (width or an address off the vector
// grain, or too wide)
template <bool HEAD>
int launch_hc_cluster(HcArgs p, cudaStream_t st) {
  if (p.d % 8 || !aligned16(p.x) || !aligned16(p.fn) || !aligned16(p.v) || !aligned16(p.mean) || !aligned16(p.norm_w) ||
      !aligned16(p.h16) || !aligned16(p.hb))
    return kHcGeneral;
  p.w = ((p.d + kHcCtas - 1) / kHcCtas + 7) / 8 * 8;
  // one row per cluster while that is one wave of two CTAs an SM (37 rows of eight CTAs); beyond it
  // the sixteen-row form reads fn once for sixteen rows (rows too wide for its slice stay at one)
  constexpr int kMaxSlice = 160 * 1024;
  const size_t slice = (size_t)p.H * p.w * 2;
  const int R = p.rows <= 37 || 16 * slice > kMaxSlice ? 1 : 16;
  const size_t smem = R * slice;
  if (smem > kMaxSlice) return kHcGeneral;
  auto kernel = R == 1 ? hc_cluster_kernel<1, HEAD> : hc_cluster_kernel<16, HEAD>;
  // the limit of any width, once: set to the bytes of each launch, a narrower engine of another thread could lower it
  // between this thread's set and its launch
  static unsigned long long limit_set[2] = {0, 0};
  const cudaError_t e = tf_smem_limit((const void*)kernel, kMaxSlice, &limit_set[R == 1]);
  if (e != cudaSuccess) return (int)e;
  tf_launch(kernel, dim3((p.rows + R - 1) / R * kHcCtas), dim3(256), smem, st, p);
  return (int)cudaGetLastError();
}
}  // namespace

TF_API int tf_hc_coef_bytes() { return (int)sizeof(HcCoef); }

// x [rows, H, d] bf16; fn [H*(2+H), H*d] f32; base [H*(2+H)], scale [3] f32; coef [rows] records;
// v [rows, d] bf16 collapsed input; norm_w (optional) [d] bf16 -> h16 / hb normalised copies
TF_API int tf_hc_prepare(const void* x, const float* fn, const float* base, const float* scale, void* coef, void* v,
                         const void* norm_w, void* h16, void* hb, int rows, int H, int d, int iters, float eps,
                         float rms_eps, cudaStream_t st) {
  if (H < 1 || H > kMaxH) return -1;
  if (rows <= 0) return 0;
  HcArgs p = {(const __nv_bfloat16*)x, fn, base, scale, (HcCoef*)coef, (__nv_bfloat16*)v, nullptr,
              (const __nv_bfloat16*)norm_w, (__half*)h16, (__nv_bfloat16*)hb, rows, H, d, 0, iters, eps, rms_eps};
  const int c = launch_hc_cluster<false>(p, st);
  if (c != kHcGeneral) return c;
  tf_launch(hc_prepare_kernel<false>, dim3(rows), dim3(256), 0, st, (const __nv_bfloat16*)x, fn, base, scale, (HcCoef*)coef, (__nv_bfloat16*)v,
                                          nullptr, (const __nv_bfloat16*)norm_w, (__half*)h16, (__nv_bfloat16*)hb, H, d, iters,
                                          eps, rms_eps);
  return (int)cudaGetLastError();
}

// Collapse in front of the vocabulary head: pre_h = sigmoid(m_h * scale[0] + base[h]) + eps with the H
// mixes of x [rows, H, d] against fn [H, H*d], all scaled by rsqrt(mean(x^2) + rms_eps); v = bf16(sum_h
// pre_h x_h), h16 / hb (optional) = RMSNorm of v with norm_w (bf16 values), mean (optional) = bf16 mean of the
// copies.
TF_API int tf_hc_head(const void* x, const float* fn, const float* base, const float* scale, void* v, void* mean,
                      const void* norm_w, void* h16, void* hb, int rows, int H, int d, float eps, float rms_eps,
                      cudaStream_t st) {
  if (H < 1 || H > kMaxH || !x || !fn || !base || !scale || !v) return -1;
  if (rows <= 0) return 0;
  HcArgs p = {(const __nv_bfloat16*)x, fn, base, scale, nullptr, (__nv_bfloat16*)v, (__nv_bfloat16*)mean,
              (const __nv_bfloat16*)norm_w, (__half*)h16, (__nv_bfloat16*)hb, rows, H, d, 0, 0, eps, rms_eps};
  const int c = launch_hc_cluster<true>(p, st);
  if (c != kHcGeneral) return c;
  tf_launch(hc_prepare_kernel<true>, dim3(rows), dim3(256), 0, st, p.x, fn, base, scale, nullptr, p.v, p.mean, p.norm_w, p.h16,
            p.hb, H, d, 0, eps, rms_eps);
  return (int)cudaGetLastError();
}

// y [rows, H, d] bf16 = post * a + comb^T x with a [rows, d] f32 (the reduced sublayer output)
TF_API int tf_hc_post(const void* x, const float* a, const void* coef, void* y, int rows, int H, int d,
                      cudaStream_t st) {
  if (H < 1 || H > kMaxH) return -1;
  if (rows <= 0) return 0;
  if (d % 8 == 0 && rows <= 65535 && aligned16(x) && aligned16(a) && aligned16(y))
    tf_launch(hc_post_vec_kernel, dim3((d + 1023) / 1024, rows), dim3(128), 0, st, (const __nv_bfloat16*)x, a,
              (const HcCoef*)coef, (__nv_bfloat16*)y, H, d);
  else
    tf_launch(hc_post_kernel, dim3(dim3(rows, H)), dim3(256), 0, st, (const __nv_bfloat16*)x, a, (const HcCoef*)coef, (__nv_bfloat16*)y, H, d);
  return (int)cudaGetLastError();
}
