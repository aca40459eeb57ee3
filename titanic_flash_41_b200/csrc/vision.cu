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

// All of these move rows between GEMMs and are bound by memory: eight bf16 per thread and access (widths
// are multiples of 8, rows 16-byte aligned), and the bias of a projection is added (and rounded, as a
// separate pass would) by the kernel that reads its rows next.  One element per thread and a pass per
// bias: 3.3 ms of an eight-layer encoding of 8,580 patches.
struct V8 {
  float f[8];
};
__device__ __forceinline__ V8 ld8(const B* p) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  V8 v;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __bfloat1622float2(h[j]);
    v.f[2 * j] = f.x;
    v.f[2 * j + 1] = f.y;
  }
  return v;
}
__device__ __forceinline__ void st8(B* p, const V8& v) {
  __nv_bfloat162 h[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v.f[2 * j], v.f[2 * j + 1]);
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(h);
}
// x + bias, rounded to bf16; without a bias x as it is
__device__ __forceinline__ V8 ld8_bias(const B* p, const B* bias) {
  V8 v = ld8(p);
  if (bias) {
    const V8 b = ld8(bias);
#pragma unroll
    for (int j = 0; j < 8; ++j) v.f[j] = bf16_round(v.f[j] + b.f[j]);
  }
  return v;
}

__global__ void __launch_bounds__(256) vis_bias_kernel(const B* x, const B* bias, B* y, long count, int width) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i < count) st8(y + i, ld8_bias(x + i, bias + i % width));
}

// x += delta (+ the bias of the projection that made delta); y = rmsnorm(x) * w
__global__ void __launch_bounds__(128) vis_norm_kernel(B* x, const B* delta, const B* bias, const B* w, B* y, int width,
                                                       float eps) {
  tf_pdl_sync();
  __shared__ float red[4];
  const long row = blockIdx.x * (long)width;
  float s = 0.f;
  for (int c = threadIdx.x * 8; c < width; c += 1024) {
    V8 v = ld8(x + row + c);
    if (delta) {
      const V8 d = ld8_bias(delta + row + c, bias ? bias + c : nullptr);
#pragma unroll
      for (int j = 0; j < 8; ++j) v.f[j] = bf16_round(v.f[j] + d.f[j]);
      st8(x + row + c, v);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v.f[j] * v.f[j];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  const float inv = rsqrtf((red[0] + red[1] + red[2] + red[3]) / width + eps);
  for (int c = threadIdx.x * 8; c < width; c += 1024) {      // (a thread reads back what it wrote)
    V8 v = ld8(x + row + c);
    const V8 g = ld8(w + c);
#pragma unroll
    for (int j = 0; j < 8; ++j) v.f[j] = v.f[j] * inv * g.f[j];
    st8(y + row + c, v);
  }
}

// q, k, v: [heads][n_pad][64]; rows n .. n_pad - 1 become zeros.  A thread turns pairs 8 g .. 8 g + 7 of one head.
__global__ void __launch_bounds__(256) vis_rope_split_kernel(const B* qkv, const B* bias, B* q, B* k, B* v, int n,
                                                             int n_pad, int grid_w, int heads) {
  tf_pdl_sync();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n_pad * heads * 4) return;
  const int width = heads * 64, g = (int)(i & 3) * 8, head = (int)(i >> 2) % heads, row = (int)((i >> 2) / heads);
  const long dst = ((long)head * n_pad + row) * 64 + g;
  if (row >= n) {
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int h = 0; h < 64; h += 32) {
      *reinterpret_cast<uint4*>(q + dst + h) = z;
      *reinterpret_cast<uint4*>(k + dst + h) = z;
      *reinterpret_cast<uint4*>(v + dst + h) = z;
    }
    return;
  }
  float sn[8], cs[8];
  const float pos = (float)(g < 16 ? row / grid_w : row % grid_w);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float freq = 1.f / powf(10000.f, (float)((g + j) % 16) / 16.f);
    sincosf(pos * freq, &sn[j], &cs[j]);
  }
  const int col = head * 64 + g;
  const B* src = qkv + (long)row * 3 * width + col;
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const V8 a = ld8_bias(src + part * width, bias + part * width + col);
    const V8 b = ld8_bias(src + part * width + 32, bias + part * width + col + 32);
    V8 o1, o2;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o1.f[j] = a.f[j] * cs[j] - b.f[j] * sn[j];
      o2.f[j] = b.f[j] * cs[j] + a.f[j] * sn[j];
    }
    B* out = part ? k : q;
    st8(out + dst, o1);
    st8(out + dst + 32, o2);
  }
  st8(v + dst, ld8_bias(src + 2 * width, bias + 2 * width + col));
  st8(v + dst + 32, ld8_bias(src + 2 * width + 32, bias + 2 * width + col + 32));
}

__global__ void __launch_bounds__(256) vis_swiglu_kernel(const B* gu, B* y, long count, int inter) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= count) return;
  const long row = i / inter;
  const int c = (int)(i - row * inter);
  V8 g = ld8(gu + row * 2 * inter + c);
  const V8 u = ld8(gu + row * 2 * inter + inter + c);
#pragma unroll
  for (int j = 0; j < 8; ++j) g.f[j] = bf16_round(g.f[j] / (1.f + expf(-g.f[j]))) * u.f[j];
  st8(y + i, g);
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

__global__ void __launch_bounds__(256) vis_gelu_kernel(const B* x, const B* bias, B* y, long count, int width) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= count) return;
  V8 v = ld8_bias(x + i, bias + i % width);
#pragma unroll
  for (int j = 0; j < 8; ++j) v.f[j] = (v.f[j] * 0.5f) * (1.f + erff(v.f[j] * 0.70710678118654752440f));
  st8(y + i, v);
}

__global__ void __launch_bounds__(256) vis_span_kernel(const B* f, const B* bias, const B* start, const B* newline,
                                                       const B* end, B* out, int width, int tokens, int d) {
  tf_pdl_sync();
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= (long)tokens * d) return;
  const int row = (int)(i / d), col = (int)(i % d);
  V8 v;
  if (row == 0) v = ld8(start + col);
  else if (row + 1 == tokens) v = ld8(end + col);
  else {
    const int r = row - 1, x = r % (width + 1), y = r / (width + 1);
    v = x == width ? ld8(newline + col) : ld8_bias(f + ((long)y * width + x) * d + col, bias + col);
  }
  st8(out + i, v);
}

inline unsigned blocks(long n) { return (unsigned)((n + 255) / 256); }
}  // namespace

TF_API int tf_vis_bias(const void* x, const void* bias, void* y, long count, int width, cudaStream_t st) {
  if (width % 8) return -1;
  tf_launch(vis_bias_kernel, dim3(blocks(count / 8)), dim3(256), 0, st, (const B*)x, (const B*)bias, (B*)y, count, width);
  return (int)cudaGetLastError();
}
// x [rows, width] += delta (optional; with its projection's bias, optional); y = rmsnorm(x) * w
TF_API int tf_vis_norm(void* x, const void* delta, const void* bias, const void* w, void* y, int rows, int width, float eps,
                       cudaStream_t st) {
  if (width % 8) return -1;
  tf_launch(vis_norm_kernel, dim3(rows), dim3(128), 0, st, (B*)x, (const B*)delta, (const B*)bias, (const B*)w, (B*)y,
            width, eps);
  return (int)cudaGetLastError();
}
// qkv [n, 3 * heads * 64] and its bias -> q, k, v [heads][n_pad][64], rows n .. zero
TF_API int tf_vis_rope_split(const void* qkv, const void* bias, void* q, void* k, void* v, int n, int n_pad, int grid_w,
                             int heads, cudaStream_t st) {
  if (n > n_pad || !bias) return -1;
  tf_launch(vis_rope_split_kernel, dim3(blocks((long)n_pad * heads * 4)), dim3(256), 0, st, (const B*)qkv, (const B*)bias,
            (B*)q, (B*)k, (B*)v, n, n_pad, grid_w, heads);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_swiglu(const void* gu, void* y, long rows, int inter, cudaStream_t st) {
  if (inter % 8) return -1;
  tf_launch(vis_swiglu_kernel, dim3(blocks(rows * inter / 8)), dim3(256), 0, st, (const B*)gu, (B*)y, rows * inter, inter);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_unfold(const void* x, void* y, int h, int w, int width, cudaStream_t st) {
  const long count = (long)((h + 2) / 3) * ((w + 2) / 3) * width * 9;
  tf_launch(vis_unfold_kernel, dim3(blocks(count)), dim3(256), 0, st, (const B*)x, (B*)y, h, w, width, count);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_gelu(const void* x, const void* bias, void* y, long count, int width, cudaStream_t st) {
  if (width % 8) return -1;
  tf_launch(vis_gelu_kernel, dim3(blocks(count / 8)), dim3(256), 0, st, (const B*)x, (const B*)bias, (B*)y, count, width);
  return (int)cudaGetLastError();
}
TF_API int tf_vis_span(const void* f, const void* bias, const void* start, const void* newline, const void* end, void* out,
                       int width, int tokens, int d, cudaStream_t st) {
  if (d % 8) return -1;
  tf_launch(vis_span_kernel, dim3(blocks((long)tokens * d / 8)), dim3(256), 0, st, (const B*)f, (const B*)bias,
            (const B*)start, (const B*)newline, (const B*)end, (B*)out, width, tokens, d);
  return (int)cudaGetLastError();
}
