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
// (added in CTA order).
//   R = 1   warp q computes mixes 3q .. 3q + 2, two columns per packed fp32 FMA.  Few rows (decode): bound by the latency of streaming fn (1.97 MB at 4 x 5120) from L2; eight
//           CTAs a row shorten the stream eightfold.  One CTA per row took 202 us for 24 rows; a decode
//           step with 14 of these and 6 head collapses (then a chain of library calls): 10.1 -> 6.8 ms
//   R = 16  many rows (prefill): fn crosses L2 once per 16 rows.  The mixes are a product of 16 rows by 24 mixes on the
//           tensor cores (mma.sync, bf16): x is bf16, and an fp32 weight is the sum of three bf16 numbers (8 of
//           its 24 bits each), so every product is exact as in an fp32 FMA and sums are fp32.  A warp takes every eighth
//           step of 16 columns.  The Sinkhorn steps of a row (20 dependent pairs of sums and divisions) are done by
//           one CTA of the cluster, two rows at once by one warp, while the others collapse.
//           4,001 rows of 4 x 5,120: 440 us with packed fp32 FMAs and pieces loaded one by one, 240 so (mixes 24,000 of a CTA's
//           58,000 cycles before the split by truncation and the walk without divisions); x alone takes 25 us.
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
__device__ __forceinline__ void mma_bf16_16816(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// the upper halves of a pair as a bf16 pair (its first eight significant bits); v becomes what is left of it, exactly
__device__ __forceinline__ uint32_t take_bf2(float2& v) {
  const uint32_t x = __float_as_uint(v.x), y = __float_as_uint(v.y);
  v.x -= __uint_as_float(x & 0xffff0000u);
  v.y -= __uint_as_float(y & 0xffff0000u);
  return __byte_perm(x, y, 0x7632);
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
  // (many rows: rows 16 bytes off a multiple of 128, so that the eight rows of a fragment load lie in different banks)
  const int pitch = H * w + (R > 1 ? 8 : 0);
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
    // asynchronous copies: a warp's rows are all requested before any is waited for (loaded and stored one piece after another,
    // the twenty pieces of a lane were twenty trips to HBM, half of the launch)
    for (int r = warp; r < R; r += 8) {
      const bool live = row0 + r < p.rows;
      for (int i = lane; i < H * w8; i += 32) {
        const int h = i / w8, k = (i - h * w8) * 8;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(xs + r * pitch + h * w + k);
        const __nv_bfloat16* src = p.x + (long)(live ? row0 + r : row0) * n + (long)h * d + c0 + k;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  if (R == 1 && threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += red[0][q];
    part[0][kMaxMix] = t;
  }

  if (R == 1) {
    // ---- mixes 3 warp .. 3 warp + 2 over this CTA's columns
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
  } else {
    // ---- mixes of the sixteen rows: A = rows, B = the three parts of fn; inside a step lane t of a quad takes columns
    // 4t .. 4t + 3 of both (any order of the columns does, as long as it is the same one)
    __shared__ float wpart[R > 1 ? 8 : 1][R][kCols];
    float acc[3][4];
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
    const int g = lane >> 2, t4 = (lane & 3) * 4;
    const int sh = (wc + 15) / 16, total = H * sh, tiles = (nmix + 7) / 8;
    const int span = max(sh, 1) * 16;         // columns of a copy in whole steps (a CTA may have none)
    struct Place {                            // of a step: copy and first column (walked, not divided out)
      int h, i;
    };
    auto advance = [&](Place& q) {
      q.i += 8 * 16;
      while (q.i >= span) {
        q.i -= span;
        ++q.h;
      }
    };
    Place ahead = {0, warp * 16}, at = ahead;
    while (ahead.i >= span) {
      ahead.i -= span;
      ++ahead.h;
    }
    at = ahead;
    const float* fn_row = p.fn + (long)g * n + c0 + t4;
    auto load_fn = [&](float4 (&f)[3]) {
      const float* src = fn_row + (long)ahead.h * d + ahead.i;
      const bool on = ahead.h < H && ahead.i + t4 < wc;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        f[m] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (on && m < tiles && m * 8 + g < nmix) f[m] = __ldg(reinterpret_cast<const float4*>(src + (long)(m * 8) * n));
      }
      advance(ahead);
    };
    constexpr int kAhead = 3;                 // steps of fn requested ahead
    float4 ring[kAhead][3];
    float ss0 = 0.f, ss1 = 0.f;               // sums of squares of rows g and g + 8 (every element passes through one lane)
    const __nv_bfloat16* x_row = xs + g * pitch + t4;
    auto step_of = [&](const float4 (&f)[3]) {
      uint2 lo = make_uint2(0u, 0u), hi = lo;
      if (at.i + t4 < wc) {
        lo = *reinterpret_cast<const uint2*>(x_row + at.h * w + at.i);
        hi = *reinterpret_cast<const uint2*>(x_row + 8 * pitch + at.h * w + at.i);
      }
      advance(at);
      const uint32_t a[4] = {lo.x, hi.x, lo.y, hi.y};
      const float2 q0 = bf2_to_f2(lo.x), q1 = bf2_to_f2(lo.y), q2 = bf2_to_f2(hi.x), q3 = bf2_to_f2(hi.y);
      ss0 += (q0.x * q0.x + q0.y * q0.y) + (q1.x * q1.x + q1.y * q1.y);
      ss1 += (q2.x * q2.x + q2.y * q2.y) + (q3.x * q3.x + q3.y * q3.y);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        if (m >= tiles) break;
        float2 u = make_float2(f[m].x, f[m].y), v = make_float2(f[m].z, f[m].w);
        uint32_t b[3][2];
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) {
          b[piece][0] = take_bf2(u);
          b[piece][1] = take_bf2(v);
        }
        // the step's sum from zero, smallest parts first, then one rounded fp32 addition: the tensor core truncates what it adds
        // to its accumulator (all steps into one: pre at 20,480 columns 5.4e-7 from fp64; so 1.1e-7, fp32 FMAs 1.3e-7)
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int piece = 2; piece >= 0; --piece) mma_bf16_16816(d, a, b[piece]);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][e] += d[e];
      }
    };
#pragma unroll
    for (int k = 0; k < kAhead; ++k) load_fn(ring[k]);
    for (int step = warp; step < total; step += 8 * kAhead) {
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const float4 f[3] = {ring[k][0], ring[k][1], ring[k][2]};
        load_fn(ring[k]);
        if (step + 8 * k < total) step_of(f);
      }
    }
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) wpart[warp][g + (e >> 1) * 8][m * 8 + (lane & 3) * 2 + (e & 1)] = acc[m][e];
    ss0 += __shfl_xor_sync(0xffffffffu, ss0, 1);
    ss1 += __shfl_xor_sync(0xffffffffu, ss1, 1);
    ss0 += __shfl_xor_sync(0xffffffffu, ss0, 2);
    ss1 += __shfl_xor_sync(0xffffffffu, ss1, 2);
    if ((lane & 3) == 0) {
      wpart[warp][g][kMaxMix] = ss0;
      wpart[warp][g + 8][kMaxMix] = ss1;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < R * kCols; i += 256) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = (&wpart[q][0][0])[i];
      (&part[0][0])[i] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
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

  // ---- coefficients.  pre of every row in every CTA; post and comb of row r in CTA r % 8 (one row: in CTA 0).
  for (int r = warp; r < R; r += 8) {
    const float inv = rsqrtf(mix[r][kMaxMix] / n + p.rms_eps);
    if (lane < H) s_pre[r][lane] = 1.f / (1.f + expf(-(mix[r][lane] * inv * p.scale[0] + p.base[lane]))) + p.eps;
  }
  __syncthreads();
  // The warp at the coefficients of many rows has nothing that the others wait for: it arrives at their barrier first.
  const bool apart = R > 1 && !HEAD && warp == 7;
  auto arrive = [&]() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); };
  if (apart) arrive();
  if (!HEAD && (R == 1 ? c == 0 && warp == 0 : warp == 7)) {
    // lane i * 4 + j of a half warp holds comb[i][j]; the second half: the second row (one row: the same again, so that
    // every shuffle is by whole warps)
    const int r = R == 1 ? 0 : c + kHcCtas * (lane >> 4), hl = lane & 15;
    const float inv = rsqrtf(mix[r][kMaxMix] / n + p.rms_eps);
    float post = 0.f;
    if (hl < H) post = 2.f / (1.f + expf(-(mix[r][H + hl] * inv * p.scale[1] + p.base[H + hl])));
    const int i = hl >> 2, j = hl & 3;
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
    if (row0 + r < p.rows && (R > 1 || lane < 16)) {
      HcCoef* k = p.coef + row0 + r;
      if (hl < H) {
        k->pre[hl] = s_pre[r][hl];
        k->post[hl] = post;
      }
      if (on) k->comb[i * kMaxH + j] = m;
    }
  }

  // ---- collapse: this CTA's columns; the bf16 result replaces copy 0 in shared memory
  const bool norm = p.norm_w != nullptr;
  const int busy = R > 1 && !HEAD ? 7 : 8;        // (the last warp is at the coefficients)
  for (int r = R == 1 ? 0 : warp < busy ? warp : R; r < R; r += busy) {
    const int gr = row0 + r;
    float pre[kMaxH];
#pragma unroll
    for (int h = 0; h < kMaxH; ++h) pre[h] = h < H ? s_pre[r][h] : 0.f;
    float ss = 0.f;
    __nv_bfloat16* xr = xs + (long)r * pitch;
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
  if (!apart) arrive();                       // (also: nobody leaves before its partials have been read)
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (norm) {
    for (int r = R == 1 ? 0 : warp < busy ? warp : R; r < R; r += busy) {
      const int gr = row0 + r;
      float tot = 0.f;
#pragma unroll
      for (int k = 0; k < kHcCtas; ++k) tot += cluster.map_shared_rank(&vv[0], k)[r];
      if (gr >= p.rows) continue;
      const float inv = rsqrtf(tot / d + p.rms_eps);
      const __nv_bfloat16* xr = xs + (long)r * pitch;
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
  const size_t smem = R * slice + (R > 1 ? R * 16 : 0);
  if (R * slice > kMaxSlice) return kHcGeneral;
  auto kernel = R == 1 ? hc_cluster_kernel<1, HEAD> : hc_cluster_kernel<16, HEAD>;
  // the limit of any width, once: set to the bytes of each launch, a narrower engine of another thread could lower it
  // between this thread's set and its launch
  static unsigned long long limit_set[2] = {0, 0};
  const cudaError_t e = tf_smem_limit((const void*)kernel, kMaxSlice + 16 * 16, &limit_set[R == 1]);
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
