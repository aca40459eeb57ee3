// Glue kernels of the vision tower (ViT): everything between its tensor-core GEMMs.
//
//   tf_vis_bias            y = x + bias (per column)
//   tf_vis_norm            RMSNorm rows, optionally after adding a delta (+ bias) into the residual
//   tf_vis_rope_split      qkv [n, 3*width] + bias -> per-head q, k, v with 2-D rotary embedding: of each head's
//                          32 rotation pairs the first 16 turn with the patch row, the last 16
//                          with the patch column, frequency 10000^(-(c mod 16)/16)
//   tf_vis_swiglu          silu(gate) rounded to bf16, times up
//   tf_vis_unfold          3x3 neighbourhoods (channel, dy, dx order; zero beyond the bottom/right edge)
//   tf_vis_gelu            exact (erf) GELU of x + bias
//   tf_vis_span            start | feature rows each followed by a newline embedding | end
// (reference: kernels/vision.cu:7-177, 12 kernels; encoder dataflow src/vision.rs:481 encode).
#include "common.cuh"

namespace {
typedef __nv_bfloat16 B;

// All of these move rows between GEMMs and are bound by memory: eight bf16 per thread and access (V = 8), and the
// bias of a projection is added (and rounded, as a separate pass would) by the kernel that reads its rows next.
// One element per thread and a pass per bias: 3.3 ms of an eight-layer encoding of 8,580 patches.  V = 1 is the
// form for widths that eight does not divide and for operands off the 16-byte grain (a weight that is a
// view into a larger tensor): an access of eight would fault there.
template <int V>
struct Vec {
  float f[V];
};
template <int V>
__device__ __forceinline__ Vec<V> ld(const B* p) {
  Vec<V> v;
  if constexpr (V == 8) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      v.f[2 * j] = f.x;
      v.f[2 * j + 1] = f.y;
    }
  } else {
    v.f[0] = __bfloat162float(*p);
  }
  return v;
}
template <int V>
__device__ __forceinline__ void st(B* p, const Vec<V>& v) {
  if constexpr (V == 8) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v.f[2 * j], v.f[2 * j + 1]);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(h);
  } else {
    *p = __float2bfloat16_rn(v.f[0]);
  }
}
// x + bias, rounded to bf16; without a bias x as it is
template <int V>
__device__ __forceinline__ Vec<V> ld_bias(const B* p, const B* bias) {
  Vec<V> v = ld<V>(p);
  if (bias) {
    const Vec<V> b = ld<V>(bias);
#pragma unroll
    for (int j = 0; j < V; ++j) v.f[j] = bf16_round(v.f[j] + b.f[j]);
  }
  return v;
}

template <int V>
__global__ void __launch_bounds__(256) vis_bias_kernel(const B* x, const B* bias, B* y, long count, int width) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (i < count) st<V>(y + i, ld_bias<V>(x + i, bias + i % width));
}

// x += delta (+ the bias of the projection that made delta); y = rmsnorm(x) * w
template <int V>
__global__ void __launch_bounds__(128) vis_norm_kernel(B* x, const B* delta, const B* bias, const B* w, B* y, int width,
                                                       float eps) {
  tf_pdl_sync();
  __shared__ float red[4];
  const long row = blockIdx.x * (long)width;
  float s = 0.f;
  for (int c = threadIdx.x * V; c < width; c += 128 * V) {
    Vec<V> v = ld<V>(x + row + c);
    if (delta) {
      const Vec<V> d = ld_bias<V>(delta + row + c, bias ? bias + c : nullptr);
#pragma unroll
      for (int j = 0; j < V; ++j) v.f[j] = bf16_round(v.f[j] + d.f[j]);
      st<V>(x + row + c, v);
    }
#pragma unroll
    for (int j = 0; j < V; ++j) s += v.f[j] * v.f[j];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  const float inv = rsqrtf((red[0] + red[1] + red[2] + red[3]) / width + eps);
  for (int c = threadIdx.x * V; c < width; c += 128 * V) {      // (a thread reads back what it wrote)
    Vec<V> v = ld<V>(x + row + c);
    const Vec<V> g = ld<V>(w + c);
#pragma unroll
    for (int j = 0; j < V; ++j) v.f[j] = v.f[j] * inv * g.f[j];
    st<V>(y + row + c, v);
  }
}

// q, k, v: [heads][n_pad][64]; rows n .. n_pad - 1 become zeros.  A thread turns pairs g .. g + V - 1 of one head.
template <int V>
__global__ void __launch_bounds__(256) vis_rope_split_kernel(const B* qkv, const B* bias, B* q, B* k, B* v, int n,
                                                             int n_pad, int grid_w, int heads) {
  tf_pdl_sync();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kPer = 32 / V;                      // threads per head and row
  if (i >= (long)n_pad * heads * kPer) return;
  const int width = heads * 64, g = (int)(i % kPer) * V, head = (int)(i / kPer % heads), row = (int)(i / kPer / heads);
  const long dst = ((long)head * n_pad + row) * 64 + g;
  if (row >= n) {
    const Vec<V> z = {};
#pragma unroll
    for (int h = 0; h < 64; h += 32) {
      st<V>(q + dst + h, z);
      st<V>(k + dst + h, z);
      st<V>(v + dst + h, z);
    }
    return;
  }
  float sn[V], cs[V];
  const float pos = (float)(g < 16 ? row / grid_w : row % grid_w);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const float freq = 1.f / powf(10000.f, (float)((g + j) % 16) / 16.f);
    sincosf(pos * freq, &sn[j], &cs[j]);
  }
  const int col = head * 64 + g;
  const B* src = qkv + (long)row * 3 * width + col;
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const Vec<V> a = ld_bias<V>(src + part * width, bias + part * width + col);
    const Vec<V> b = ld_bias<V>(src + part * width + 32, bias + part * width + col + 32);
    Vec<V> o1, o2;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      o1.f[j] = a.f[j] * cs[j] - b.f[j] * sn[j];
      o2.f[j] = b.f[j] * cs[j] + a.f[j] * sn[j];
    }
    B* out = part ? k : q;
    st<V>(out + dst, o1);
    st<V>(out + dst + 32, o2);
  }
  st<V>(v + dst, ld_bias<V>(src + 2 * width, bias + 2 * width + col));
  st<V>(v + dst + 32, ld_bias<V>(src + 2 * width + 32, bias + 2 * width + col + 32));
}

template <int V>
__global__ void __launch_bounds__(256) vis_swiglu_kernel(const B* gu, B* y, long count, int inter) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (i >= count) return;
  const long row = i / inter;
  const int c = (int)(i - row * inter);
  Vec<V> g = ld<V>(gu + row * 2 * inter + c);
  const Vec<V> u = ld<V>(gu + row * 2 * inter + inter + c);
#pragma unroll
  for (int j = 0; j < V; ++j) g.f[j] = bf16_round(g.f[j] / (1.f + expf(-g.f[j]))) * u.f[j];
  st<V>(y + i, g);
}

__global__ void vis_unfold_kernel(const B* x, B* y, int h, int w, int width, long count) {
  tf_pdl_sync();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int cols = width * 9, out_w = (w + 2) / 3;
  const int row = (int)(i / cols), col = (int)(i % cols);
  const int sy = (row / out_w) * 3 + (col % 9) / 3, sx = (row % out_w) * 3 + col % 3;
  y[i] = (sy < h && sx < w) ? x[((long)sy * w + sx) * width + col / 9] : __float2bfloat16_rn(0.f);
}

template <int V>
__global__ void __launch_bounds__(256) vis_gelu_kernel(const B* x, const B* bias, B* y, long count, int width) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (i >= count) return;
  Vec<V> v = ld_bias<V>(x + i, bias + i % width);
#pragma unroll
  for (int j = 0; j < V; ++j) v.f[j] = (v.f[j] * 0.5f) * (1.f + erff(v.f[j] * 0.70710678118654752440f));
  st<V>(y + i, v);
}

template <int V>
__global__ void __launch_bounds__(256) vis_span_kernel(const B* f, const B* bias, const B* start, const B* newline,
                                                       const B* end, B* out, int width, int tokens, int d) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (i >= (long)tokens * d) return;
  const int row = (int)(i / d), col = (int)(i % d);
  Vec<V> v;
  if (row == 0) v = ld<V>(start + col);
  else if (row + 1 == tokens) v = ld<V>(end + col);
  else {
    const int r = row - 1, x = r % (width + 1), y = r / (width + 1);
    v = x == width ? ld<V>(newline + col) : ld_bias<V>(f + ((long)y * width + x) * d + col, bias + col);
  }
  st<V>(out + i, v);
}

inline unsigned blocks(long n) { return (unsigned)((n + 255) / 256); }
// elements per access: eight when every row is a multiple of eight and every pointer on the 16-byte grain, else one
template <typename... P>
int grain(long width, P... ptr) {
  return width % 8 == 0 && !((0 | ... | reinterpret_cast<uintptr_t>(ptr)) & 15) ? 8 : 1;
}
}  // namespace

TF_API int tf_vis_bias(const void* x, const void* bias, void* y, long count, int width, cudaStream_t st) {
  const int V = grain(width | count, x, bias, y);
  tf_launch(V == 8 ? vis_bias_kernel<8> : vis_bias_kernel<1>, dim3(blocks(count / V)), dim3(256), 0, st, (const B*)x,
            (const B*)bias, (B*)y, count, width);
  return (int)cudaGetLastError();
}
// x [rows, width] += delta (optional; with its projection's bias, optional); y = rmsnorm(x) * w
TF_API int tf_vis_norm(void* x, const void* delta, const void* bias, const void* w, void* y, int rows, int width, float eps,
                       cudaStream_t st) {
  tf_launch(grain(width, x, delta, bias, w, y) == 8 ? vis_norm_kernel<8> : vis_norm_kernel<1>, dim3(rows), dim3(128), 0, st,
            (B*)x, (const B*)delta, (const B*)bias, (const B*)w, (B*)y, width, eps);
  return (int)cudaGetLastError();
}
// qkv [n, 3 * heads * 64] and its bias -> q, k, v [heads][n_pad][64], rows n .. zero
TF_API int tf_vis_rope_split(const void* qkv, const void* bias, void* q, void* k, void* v, int n, int n_pad, int grid_w,
                             int heads, cudaStream_t st) {
  if (n > n_pad || !bias) return -1;
  const int V = grain(64, qkv, bias, q, k, v);
  tf_launch(V == 8 ? vis_rope_split_kernel<8> : vis_rope_split_kernel<1>, dim3(blocks((long)n_pad * heads * (32 / V))),
            dim3(256), 0, st, (const B*)qkv, (const B*)bias, (B*)q, (B*)k, (B*)v, n, n_pad, grid_w, heads);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_swiglu(const void* gu, void* y, long rows, int inter, cudaStream_t st) {
  const int V = grain(inter, gu, y);
  tf_launch(V == 8 ? vis_swiglu_kernel<8> : vis_swiglu_kernel<1>, dim3(blocks(rows * inter / V)), dim3(256), 0, st,
            (const B*)gu, (B*)y, rows * inter, inter);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_unfold(const void* x, void* y, int h, int w, int width, cudaStream_t st) {
  const long count = (long)((h + 2) / 3) * ((w + 2) / 3) * width * 9;
  tf_launch(vis_unfold_kernel, dim3(blocks(count)), dim3(256), 0, st, (const B*)x, (B*)y, h, w, width, count);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_gelu(const void* x, const void* bias, void* y, long count, int width, cudaStream_t st) {
  const int V = grain(width | count, x, bias, y);
  tf_launch(V == 8 ? vis_gelu_kernel<8> : vis_gelu_kernel<1>, dim3(blocks(count / V)), dim3(256), 0, st, (const B*)x,
            (const B*)bias, (B*)y, count, width);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_span(const void* f, const void* bias, const void* start, const void* newline, const void* end, void* out,
                       int width, int tokens, int d, cudaStream_t st) {
  const int V = grain(d, f, bias, start, newline, end, out);
  tf_launch(V == 8 ? vis_span_kernel<8> : vis_span_kernel<1>, dim3(blocks((long)tokens * d / V)), dim3(256), 0, st,
            (const B*)f, (const B*)bias, (const B*)start, (const B*)newline, (const B*)end, (B*)out, width, tokens, d);
  return (int)cudaGetLastError();
}
