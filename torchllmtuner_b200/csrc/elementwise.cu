// Memory-bound training kernels for sm_100a: RMSNorm (with residual add) fwd/bwd, per-head QK-norm + RoPE
// fwd/bwd, SwiGLU fwd/bwd, row-wise cross-entropy with in-place gradient, fused AdamW on flat shards,
// deterministic squared-norm. bf16 storage, fp32 math, 16-byte vector accesses.
// (reference call sites: llmtuner/models/qwen/ops.py:80-131,503; llmtuner/components/loss.py:35-70;
//  llmtuner/components/optimizer/optimizer.py:62-106; llmtuner/accelerator/collectives.py:290-558)
#include <initializer_list>
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace llmt {

constexpr int kRowThreads = 256;

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < nw) ? red[l] : 0.f;
  t = warp_sum(t);
  return t;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < nw) ? red[l] : -INFINITY;
  t = warp_max(t);
  return t;
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(b[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* f) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]);
  u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]);
  u.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ------------------------------------------------------------------------------------------ RMSNorm
// A row is owned by TR threads (a warp up to the whole block), each holding NV groups of 8 columns:
// col = (v * TR + t) * 8, so that narrow rows (a 512-wide model: 64 vectors) leave no thread idle. Bound by memory; NV and TR by
// width in fwd_by_row_width and bwd_by_row_width (TR = 32 needs no barrier).
// The forward gives a group a block of its own (or a warp of an eight-row block): named barriers with a computed id reserve
// all sixteen of a block and then only four blocks fit an SM (57 us against 42 us at 8192 x 4096). The backward, which has two
// blocks per SM anyway, puts 256 / TR groups into a block to keep the number of weight-gradient partials down.
// 8192 x 4096 bf16 with the residual: forward 42 us, backward 50 us + 3.5 us for the column sums (before: 95 + 14 us, one row
// after another without the prefetch); the 268 MB that each reads and writes take 42 us at copy speed.
// The order of a row's additions is that of 256 threads with one vector each up to 2048 columns (two or four beyond), whatever group
// computes it: a group whose threads hold PARTS vectors of such a row keeps their sums apart, and the partial sums of the warps meet in
// a tree. Bits then do not depend on the group, and a rounding that differs here travels through a whole network of bf16 layers.
template <int TR, int NV>
__host__ __device__ constexpr int row_parts() { return TR * NV <= kRowThreads ? NV : 1; }
template <int TR, int PARTS, bool ONE_GROUP>
__device__ __forceinline__ float row_sum(const float (&v)[PARTS], float* red, int& buf) {
  constexpr int NW = TR / 32, N = NW * PARTS;
  const int t = threadIdx.x % TR;
  float s = v[0];
  if constexpr (PARTS == 2) {                          // two warp sums for six shuffles: each half of the warp finishes one of them
    const bool hi = threadIdx.x & 16;
    s = (hi ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[1], 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  } else {
    static_assert(PARTS == 1, "one or two vectors whose sums are kept apart");
    s = warp_sum(s);
  }
  if constexpr (TR == 32) return PARTS == 2 ? s + __shfl_xor_sync(0xffffffffu, s, 16) : s;
  // one barrier per row: the partial sums alternate between two buffers, and no warp can be two rows ahead
  float* r = red + buf * (PARTS * (TR > kRowThreads ? TR : kRowThreads) / 32) + threadIdx.x / TR * N;
  if ((t & (32 / PARTS - 1)) == 0) r[(PARTS == 2 ? (t >> 4 & 1) * NW : 0) + (t >> 5)] = s;
  if constexpr (ONE_GROUP) __syncthreads();
  else named_bar_sync(1 + threadIdx.x / TR, TR);
  float a[N];
#pragma unroll
  for (int i = 0; i < N; ++i) a[i] = r[i];
  buf ^= 1;
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) a[i] += a[i + o];
  return a[0];
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(b[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}

// y = (x [+ res]) * rsqrt(mean((x+res)^2) + eps) * w ; optionally writes s = x + res (the new residual stream).
template <int NV, int TR>
__global__ void __launch_bounds__(TR > 32 ? TR : kRowThreads) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                                  const __nv_bfloat16* __restrict__ res,
                                                                  const __nv_bfloat16* __restrict__ w,
                                                                  __nv_bfloat16* __restrict__ y,
                                                                  __nv_bfloat16* __restrict__ sum_out,
                                                                  float* __restrict__ rstd, int T, int D, float eps) {
  constexpr int RPB = TR > 32 ? 1 : kRowThreads / TR, PARTS = row_parts<TR, NV>();
  __shared__ float red[2 * PARTS * (kRowThreads / 32)];
  const int t = threadIdx.x % TR;
  int buf = 0;
  for (int row = blockIdx.x * RPB + threadIdx.x / TR; row < T; row += gridDim.x * RPB) {
    float v[NV][8];
    float ss[PARTS] = {0.f};
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * TR + t) * 8;
      if (col < D) {
        load8(x + (int64_t)row * D + col, v[i]);
        if (res != nullptr) {
          float r[8];
          load8(res + (int64_t)row * D + col, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(__float2bfloat16_rn(v[i][j] + r[j]));
          if (sum_out != nullptr) store8(sum_out + (int64_t)row * D + col, v[i]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss[PARTS > 1 ? i : 0] += v[i][j] * v[i][j];
      }
    }
    const float r = rsqrtf(row_sum<TR, PARTS, true>(ss, red, buf) / (float)D + eps);
    if (t == 0 && rstd != nullptr) rstd[row] = r;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * TR + t) * 8;
      if (col < D) {
        float wv[8], o[8];
        load8(w + col, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = v[i][j] * r * wv[j];
        store8(y + (int64_t)row * D + col, o);
      }
    }
  }
}

// dx = r * (g - x * r^2 * mean(g * x)) [+ dres], g = dy * w ; dw partial per block = sum_rows dy * x * r.
// Bound by memory (x, dy, dres read, dx written). The weight gradient stays in registers over all rows of the block, so
// there are only 512 threads per SM; the operands of the next row are fetched before the reduction of this one, which keeps
// loads in flight across the barrier.
template <int TR>
struct RowBlock { static constexpr int kThreads = TR > kRowThreads ? TR : kRowThreads, kRows = kThreads / TR; };

template <int NV, int TR>
__global__ void __launch_bounds__(RowBlock<TR>::kThreads, 512 / RowBlock<TR>::kThreads) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                                     const __nv_bfloat16* __restrict__ x,
                                                                     const __nv_bfloat16* __restrict__ w,
                                                                     const float* __restrict__ rstd,
                                                                     const __nv_bfloat16* __restrict__ dres,
                                                                     __nv_bfloat16* __restrict__ dx,
                                                                     float* __restrict__ dw_partial, int T, int D) {
  constexpr int NT = RowBlock<TR>::kThreads, RPB = RowBlock<TR>::kRows, PARTS = row_parts<TR, NV>();
  __shared__ float red[2 * PARTS * (NT / 32)];
  __shared__ float parts[RPB > 1 ? RPB * NV * TR * 8 : 1];
  const int t = threadIdx.x % TR, grp = threadIdx.x / TR;
  int buf = 0;
  float dw[NV][8];
  uint4 wr[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (i * TR + t) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[i][j] = 0.f;
    wr[i] = col < D ? *reinterpret_cast<const uint4*>(w + col) : make_uint4(0, 0, 0, 0);
  }
  const int step = gridDim.x * RPB;
  uint4 xr[NV], dr[NV], er[NV];
  float r = 0.f;
  auto fetch = [&](int row, uint4* fx, uint4* fd, uint4* fe, float& fr) {
    fr = rstd[row];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * TR + t) * 8;
      const int64_t at = (int64_t)row * D + col;
      const uint4 zero = make_uint4(0, 0, 0, 0);
      fx[i] = fd[i] = fe[i] = zero;
      if (col < D) {
        fx[i] = *reinterpret_cast<const uint4*>(x + at);
        fd[i] = *reinterpret_cast<const uint4*>(dy + at);
        if (dres != nullptr) fe[i] = *reinterpret_cast<const uint4*>(dres + at);
      }
    }
  };
  int row = blockIdx.x * RPB + grp;
  if (row < T) fetch(row, xr, dr, er, r);
  for (; row < T; row += step) {
    float c[PARTS] = {0.f};
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float xv[8], d[8], wv[8];
      unpack8(xr[i], xv); unpack8(dr[i], d); unpack8(wr[i], wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        c[PARTS > 1 ? i : 0] += d[j] * wv[j] * xv[j];
        dw[i][j] += d[j] * xv[j] * r;
      }
    }
    uint4 nx[NV], nd[NV], ne[NV];
    float nr = 0.f;
    if (row + step < T) fetch(row + step, nx, nd, ne, nr);
    const float k = r * r * r * row_sum<TR, PARTS, (RPB == 1)>(c, red, buf) / (float)D;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * TR + t) * 8;
      if (col < D) {
        float xv[8], d[8], wv[8], e[8], o[8];
        unpack8(xr[i], xv); unpack8(dr[i], d); unpack8(wr[i], wv); unpack8(er[i], e);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = r * (d[j] * wv[j]) - xv[j] * k;
        if (dres != nullptr) {
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += e[j];
        }
        store8(dx + (int64_t)row * D + col, o);
      }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) { xr[i] = nx[i]; dr[i] = nd[i]; er[i] = ne[i]; }
    r = nr;
  }
  if constexpr (RPB > 1) {                         // the row groups of the block, added in a fixed order
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) parts[grp * (NV * TR * 8) + (i * TR + t) * 8 + j] = dw[i][j];
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += NT) {
      float s = 0.f;
#pragma unroll
      for (int g = 0; g < RPB; ++g) s += parts[g * (NV * TR * 8) + c];
      dw_partial[(int64_t)blockIdx.x * D + c] = s;
    }
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * TR + t) * 8;
      if (col < D) {
        float4* p = reinterpret_cast<float4*>(dw_partial + (int64_t)blockIdx.x * D + col);
        p[0] = make_float4(dw[i][0], dw[i][1], dw[i][2], dw[i][3]);
        p[1] = make_float4(dw[i][4], dw[i][5], dw[i][6], dw[i][7]);
      }
    }
  }
}

// out[c] (+)= sum_p partial[p][c]. A block owns 32 columns; its 32 warps take every 32nd partial row (one 128-byte line
// each) and the 32 sums of a column are added in a fixed order. One thread per column (the earlier form) was a chain of up
// to 592 dependent loads in as few as one block: 10-15 us per call, now 3 us.
__global__ void __launch_bounds__(1024) colsum_kernel(const float* __restrict__ partial, float* __restrict__ out_f32,
                                                      __nv_bfloat16* __restrict__ out_bf16, int P, int D, int accumulate) {
  __shared__ float part[32][33];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < D) {
#pragma unroll 4
    for (int p = wid; p < P; p += 32) s += partial[(int64_t)p * D + c];
  }
  part[wid][lane] = s;
  __syncthreads();
  s = warp_sum(part[lane][wid]);                   // warp w adds the 32 sums of column w
  const int oc = blockIdx.x * 32 + wid;
  if (lane == 0 && oc < D) {
    if (out_f32 != nullptr) out_f32[oc] = accumulate ? out_f32[oc] + s : s;
    if (out_bf16 != nullptr) out_bf16[oc] = __float2bfloat16_rn(accumulate ? __bfloat162float(out_bf16[oc]) + s : s);
  }
}

// ------------------------------------------------------------------------------------------ QK-norm + RoPE
// A group of G = 8 * P lanes per (token, head); HD = 64 * P, so a warp holds 32 / G items (HD 128: two items per warp).
// Lane g of the group owns columns [4g, 4g + 4) of the first half and their rotation partners [HD/2 + 4g, ...): every
// access is an 8-byte vector (bf16 x 4) or a 16-byte vector (cos / sin fp32 x 4). Token rows are `tok_stride` elements
// apart, heads are packed (HD apart), all strides multiples of 4 elements.
// Forward: n = x * rsqrt(mean x^2 + eps) * w (skipped when w == nullptr), then half rotation with cos/sin [T, HD/2]:
//   y1 = n1 cos - n2 sin ; y2 = n2 cos + n1 sin.
__device__ __forceinline__ void ld_bf16x4(const __nv_bfloat16* p, float* f) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void st_bf16x4(__nv_bfloat16* p, const float* f) {
  uint2 v;
  v.x = pack_bf16x2(f[0], f[1]);
  v.y = pack_bf16x2(f[2], f[3]);
  *reinterpret_cast<uint2*>(p) = v;
}
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int P>
__global__ void __launch_bounds__(256) qk_norm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ x, int64_t tok_stride,
                                                               const __nv_bfloat16* __restrict__ w,
                                                               const float* __restrict__ cosb,
                                                               const float* __restrict__ sinb,
                                                               __nv_bfloat16* __restrict__ y, int64_t y_tok_stride,
                                                               float* __restrict__ rstd, int T, int H, float eps) {
  constexpr int HD = 64 * P, HALF = HD / 2, G = 8 * P, IPW = 32 / G;
  const int lane = threadIdx.x & 31, g = lane % G;
  const int64_t total = (int64_t)T * H;
  int64_t item = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * IPW + lane / G;
  const bool live = item < total;
  if (!live) item = total - 1;                       // keep the whole warp in the shuffles
  const int t = (int)(item / H), h = (int)(item % H);
  const __nv_bfloat16* px = x + (int64_t)t * tok_stride + (int64_t)h * HD + 4 * g;
  float a[4], b[4];
  ld_bf16x4(px, a);
  ld_bf16x4(px + HALF, b);
  float r = 1.f;
  float wa[4] = {1.f, 1.f, 1.f, 1.f}, wb[4] = {1.f, 1.f, 1.f, 1.f};
  if (w != nullptr) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) ss += a[j] * a[j] + b[j] * b[j];
    ss = group_sum<G>(ss);
    r = rsqrtf(ss / (float)HD + eps);
    if (g == 0 && live && rstd != nullptr) rstd[item] = r;
    ld_bf16x4(w + 4 * g, wa);
    ld_bf16x4(w + HALF + 4 * g, wb);
  }
  const float4 cs = *reinterpret_cast<const float4*>(cosb + (int64_t)t * HALF + 4 * g);
  const float4 sn = *reinterpret_cast<const float4*>(sinb + (int64_t)t * HALF + 4 * g);
  const float c4[4] = {cs.x, cs.y, cs.z, cs.w}, s4[4] = {sn.x, sn.y, sn.z, sn.w};
  float o1[4], o2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float n1 = a[j] * r * wa[j], n2 = b[j] * r * wb[j];
    o1[j] = n1 * c4[j] - n2 * s4[j];
    o2[j] = n2 * c4[j] + n1 * s4[j];
  }
  if (live) {
    __nv_bfloat16* py = y + (int64_t)t * y_tok_stride + (int64_t)h * HD + 4 * g;
    st_bf16x4(py, o1);
    st_bf16x4(py + HALF, o2);
  }
}

// Backward: un-rotate dy (dn1 = d1 cos + d2 sin ; dn2 = d2 cos - d1 sin), then RMSNorm backward per head.
// The weight gradient is accumulated per lane over its items, then per block in shared memory and written to
// dw_partial[blockIdx.x][HD].
template <int P>
__global__ void __launch_bounds__(256) qk_norm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ dy, int64_t dy_tok_stride,
                                                               const __nv_bfloat16* __restrict__ x, int64_t tok_stride,
                                                               const __nv_bfloat16* __restrict__ w,
                                                               const float* __restrict__ cosb,
                                                               const float* __restrict__ sinb,
                                                               const float* __restrict__ rstd,
                                                               __nv_bfloat16* __restrict__ dx, int64_t dx_tok_stride,
                                                               float* __restrict__ dw_partial, int T, int H) {
  constexpr int HD = 64 * P, HALF = HD / 2, G = 8 * P, IPW = 32 / G;
  // weight-gradient partials of the block's 256 / G thread groups, summed in a fixed order at the end (an atomic add into
  // one row would make the last bit depend on the order in which the groups arrive)
  constexpr int kGroups = 256 / G;
  __shared__ float sparts[kGroups * HD];
  const int lane = threadIdx.x & 31, g = lane % G;
  const int wpb = blockDim.x >> 5;
  const int64_t total = (int64_t)T * H;
  float dwa[4] = {0.f, 0.f, 0.f, 0.f}, dwb[4] = {0.f, 0.f, 0.f, 0.f};
  float wa[4] = {1.f, 1.f, 1.f, 1.f}, wb[4] = {1.f, 1.f, 1.f, 1.f};
  if (w != nullptr) {
    ld_bf16x4(w + 4 * g, wa);
    ld_bf16x4(w + HALF + 4 * g, wb);
  }
  // every warp runs the same number of rounds so that the group shuffles stay converged
  const int64_t warp_items = (int64_t)gridDim.x * wpb * IPW;
  const int64_t rounds = (total + warp_items - 1) / warp_items;
  for (int64_t rd = 0; rd < rounds; ++rd) {
    int64_t item = rd * warp_items + ((int64_t)blockIdx.x * wpb + (threadIdx.x >> 5)) * IPW + lane / G;
    const bool live = item < total;
    if (!live) item = total - 1;
    const int t = (int)(item / H), h = (int)(item % H);
    const int64_t off = (int64_t)h * HD + 4 * g;
    float d1[4], d2[4], xa[4] = {0.f, 0.f, 0.f, 0.f}, xb[4] = {0.f, 0.f, 0.f, 0.f};
    ld_bf16x4(dy + (int64_t)t * dy_tok_stride + off, d1);
    ld_bf16x4(dy + (int64_t)t * dy_tok_stride + off + HALF, d2);
    const float4 cs = *reinterpret_cast<const float4*>(cosb + (int64_t)t * HALF + 4 * g);
    const float4 sn = *reinterpret_cast<const float4*>(sinb + (int64_t)t * HALF + 4 * g);
    const float c4[4] = {cs.x, cs.y, cs.z, cs.w}, s4[4] = {sn.x, sn.y, sn.z, sn.w};
    const float r = (w != nullptr) ? rstd[item] : 1.f;
    if (w != nullptr) {
      ld_bf16x4(x + (int64_t)t * tok_stride + off, xa);
      ld_bf16x4(x + (int64_t)t * tok_stride + off + HALF, xb);
    }
    float ga[4], gb[4], c_acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float dn1 = d1[j] * c4[j] + d2[j] * s4[j];
      float dn2 = d2[j] * c4[j] - d1[j] * s4[j];
      if (w != nullptr) {
        if (live) {
          dwa[j] += dn1 * xa[j] * r;
          dwb[j] += dn2 * xb[j] * r;
        }
        dn1 *= wa[j];
        dn2 *= wb[j];
        c_acc += dn1 * xa[j] + dn2 * xb[j];
      }
      ga[j] = dn1;
      gb[j] = dn2;
    }
    float k = 0.f;
    if (w != nullptr) {
      c_acc = group_sum<G>(c_acc);
      k = r * r * r * c_acc / (float)HD;
    }
    float o1[4], o2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o1[j] = (w != nullptr) ? r * ga[j] - xa[j] * k : ga[j];
      o2[j] = (w != nullptr) ? r * gb[j] - xb[j] * k : gb[j];
    }
    if (live) {
      st_bf16x4(dx + (int64_t)t * dx_tok_stride + off, o1);
      st_bf16x4(dx + (int64_t)t * dx_tok_stride + off + HALF, o2);
    }
  }
  if (w != nullptr && dw_partial != nullptr) {
    float* mine = sparts + (threadIdx.x / G) * HD;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      mine[4 * g + j] = dwa[j];
      mine[HALF + 4 * g + j] = dwb[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < HD; i += blockDim.x) {
      float acc = 0.f;
#pragma unroll 4
      for (int c = 0; c < kGroups; ++c) acc += sparts[c * HD + i];
      dw_partial[(int64_t)blockIdx.x * HD + i] = acc;
    }
  }
}

// ------------------------------------------------------------------------------------------ attention backward by rows
// The two elementwise steps of the attention backward that rebuilds probabilities per block of query rows (head sizes with
// a forward kernel only): S [rows, C] fp32 from a batched product -> P = exp(S * scale - lse[row]) in bf16 with the causal
// limit applied, and dS = (dP - delta[row]) * P in bf16. One read of the fp32 block and one bf16 write each, where the
// same algebra as tensor expressions takes eight passes. Row r of the block is query (r % n) of the chunk; it sees columns
// [0, (r % n) + diag + 1).
__global__ void attn_rows_probs_kernel(const float* __restrict__ s, const float* __restrict__ lse, __nv_bfloat16* __restrict__ p,
                                       int64_t rows, int C, int n, int diag, float scale_log2, int causal) {
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const float l = lse[row];
    const float l2 = isinf(l) ? 0.f : l * 1.4426950408889634f;    // a row that sees no key: every column is beyond its limit
    const int i = (int)(row % n);
    const int lim = causal ? min(C, i + diag + 1) : C;
    const float* sr = s + row * (int64_t)C;
    __nv_bfloat16* pr = p + row * (int64_t)C;
    for (int c = threadIdx.x; c < C; c += blockDim.x)
      pr[c] = __float2bfloat16_rn(c < lim ? exp2f(sr[c] * scale_log2 - l2) : 0.f);
  }
}
__global__ void attn_rows_ds_kernel(const float* __restrict__ dp, const __nv_bfloat16* __restrict__ p, const float* __restrict__ delta,
                                    __nv_bfloat16* __restrict__ ds, int64_t rows, int C) {
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const float dl = delta[row];
    const float* dr = dp + row * (int64_t)C;
    const __nv_bfloat16* pr = p + row * (int64_t)C;
    __nv_bfloat16* or_ = ds + row * (int64_t)C;
    for (int c = threadIdx.x; c < C; c += blockDim.x) or_[c] = __float2bfloat16_rn((dr[c] - dl) * __bfloat162float(pr[c]));
  }
}

// ------------------------------------------------------------------------------------------ SwiGLU
// Rows of `gate` and `up` may be strided (views into one [T, 2F] buffer); out/dgate/dup likewise.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ up,
                                  __nv_bfloat16* __restrict__ out, int64_t T, int F, int64_t ld_in, int64_t ld_out,
                                  const int* __restrict__ row_limit) {
  // row_limit (optional, device memory): rows at or beyond *row_limit of a statically sized buffer hold nothing
  if (row_limit != nullptr && *row_limit < T) T = *row_limit;
  const int64_t nvec = T * (F / 8);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / (F / 8);
    const int col = (int)(i % (F / 8)) * 8;
    float g[8], u[8], o[8];
    load8(gate + row * ld_in + col, g);
    load8(up + row * ld_in + col, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    store8(out + row * ld_out + col, o);
  }
}
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ gate,
                                  const __nv_bfloat16* __restrict__ up, __nv_bfloat16* __restrict__ dgate,
                                  __nv_bfloat16* __restrict__ dup, int64_t T, int F, int64_t ld_in, int64_t ld_dout,
                                  int64_t ld_dg, const int* __restrict__ row_limit) {
  if (row_limit != nullptr && *row_limit < T) T = *row_limit;
  const int64_t nvec = T * (F / 8);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / (F / 8);
    const int col = (int)(i % (F / 8)) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    load8(gate + row * ld_in + col, g);
    load8(up + row * ld_in + col, u);
    load8(dout + row * ld_dout + col, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * s;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * (s + silu * (1.f - s));
    }
    store8(dgate + row * ld_dg + col, dg);
    store8(dup + row * ld_dg + col, du);
  }
}

// ------------------------------------------------------------------------------------------ cross-entropy
// One CTA per row of bf16 logits [rows, V] (row stride ld). Pass 1: online max / sum-exp. Pass 2: overwrite the
// logits with d(loss_sum)/d(logit) * grad_scale = (softmax - onehot) * grad_scale. Rows whose label is
// ignore_index get zero gradient and no loss. Row losses go to `row_loss` (fp32); the caller sums them
// (deterministic), lse goes to `row_lse` when given.
// Bound by memory. The second pass must not go to DRAM again: the first `cached` vectors of the row stay in shared memory and
// few enough rows are in flight that the rest of them is still in L2 (the launch picks threads and cache). Two vectors per
// thread and step keep it at 32 registers and the SM full; four took 64 registers and half the threads. 2048 x 151936:
// 250 us, 5.0 TB/s (before, with the whole row read again from DRAM: 305 us).
template <int NT>
__global__ void __launch_bounds__(NT, 2048 / NT) ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ labels,
                                                        float* __restrict__ row_loss, float* __restrict__ row_lse,
                                                        int V, int64_t ld, const float* __restrict__ grad_scale_ptr,
                                                        float grad_scale, int ignore_index, int write_grad, int cached) {
  extern __shared__ uint4 row_cache[];
  __shared__ float red[32];
  constexpr int U = 2;
  const int64_t row = blockIdx.x;
  __nv_bfloat16* p = logits + row * ld;
  uint4* pv = reinterpret_cast<uint4*>(p);
  const int64_t label = labels[row];
  const bool valid = (label != ignore_index) && label >= 0 && label < V;
  float m = -INFINITY, s = 0.f;
  const int nvec = V / 8;
  // x - max first, then the exponential: folding the scale into one multiply-add would overflow on logits masked with the
  // lowest finite value. A thread whose logits so far are all -inf has a maximum of -inf: it subtracts 0 instead.
  auto take = [&](const uint4* u, auto n) {          // n vectors of 8 logits into the running (max, sum)
    constexpr int W = decltype(n)::value;
    float f[W][8];
    float m4[4] = {m, m, m, m};
#pragma unroll
    for (int k = 0; k < W; ++k) {
      unpack8(u[k], f[k]);
#pragma unroll
      for (int j = 0; j < 8; ++j) m4[j & 3] = fmaxf(m4[j & 3], f[k][j]);
    }
    const float nm = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])), c = nm == -INFINITY ? 0.f : nm;
    float a4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < W; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) a4[j & 3] += __expf(f[k][j] - c);
    s = s * __expf(m - c) + ((a4[0] + a4[1]) + (a4[2] + a4[3]));
    m = nm;
  };
  int i = threadIdx.x;
  for (; i + (U - 1) * NT < nvec; i += U * NT) {
    uint4 u[U];
#pragma unroll
    for (int k = 0; k < U; ++k) u[k] = pv[i + k * NT];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * NT < cached) row_cache[i + k * NT] = u[k];
    take(u, std::integral_constant<int, U>{});
  }
  for (; i < nvec; i += NT) {
    const uint4 u = pv[i];
    if (i < cached) row_cache[i] = u;
    take(&u, std::integral_constant<int, 1>{});
  }
  for (int e = nvec * 8 + threadIdx.x; e < V; e += NT) {
    const float f = __bfloat162float(p[e]);
    const float nm = fmaxf(m, f), c = nm == -INFINITY ? 0.f : nm;
    s = s * __expf(m - c) + __expf(f - c);
    m = nm;
  }
  const float gm = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum(s, red);
  const float lse = gm + logf(gs);
  if (threadIdx.x == 0) {
    if (row_lse != nullptr) row_lse[row] = lse;
    row_loss[row] = valid ? (lse - __bfloat162float(p[label])) : 0.f;
  }
  if (!write_grad) return;
  __syncthreads();  // the label logit was read above before anyone overwrites it
  const float gsc = valid ? grad_scale * (grad_scale_ptr != nullptr ? *grad_scale_ptr : 1.f) : 0.f;
  const int lab_vec = valid ? (int)(label >> 3) : -1, lab_j = (int)(label & 7);
  auto grad = [&](const uint4& u, int at) {
    float f[8];
    unpack8(u, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __expf(f[j] - lse);
    if (at == lab_vec) {                             // before the factor: p - 1 is exact where p is close to 1
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j == lab_j) f[j] -= 1.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] *= gsc;
    store8(p + (int64_t)at * 8, f);
  };
  i = threadIdx.x;
  for (; i + (U - 1) * NT < nvec; i += U * NT) {     // every thread reads back the vectors it cached itself
    uint4 u[U];
#pragma unroll
    for (int k = 0; k < U; ++k) u[k] = i + k * NT < cached ? row_cache[i + k * NT] : pv[i + k * NT];
#pragma unroll
    for (int k = 0; k < U; ++k) grad(u[k], i + k * NT);
  }
  for (; i < nvec; i += NT) grad(i < cached ? row_cache[i] : pv[i], i);
  for (int e = nvec * 8 + threadIdx.x; e < V; e += NT) {
    float g = __expf(__bfloat162float(p[e]) - lse);
    if (e == label) g -= 1.f;
    p[e] = __float2bfloat16_rn(g * gsc);
  }
}

// out = bf16(x * *scale), scale on the device: a gradient that was computed ahead of its upstream factor leaves in one pass
// (read once, written once). 151936 x 4096 fp32 -> bf16: 646 us (5.8 TB/s); as broadcast multiplication and cast it took 2340 us.
template <typename T>
__global__ void __launch_bounds__(256) scale_to_bf16_kernel(const T* __restrict__ x, const float* __restrict__ scale,
                                                            __nv_bfloat16* __restrict__ out, int64_t n) {
  const float g = *scale;
  const int64_t nt = (int64_t)gridDim.x * blockDim.x, nvec = n / 8;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += nt) {
    float f[8];
    if constexpr (sizeof(T) == 2) unpack8(reinterpret_cast<const uint4*>(x)[i], f);
    else {
      const float4 a = __ldcs(reinterpret_cast<const float4*>(x) + 2 * i), b = __ldcs(reinterpret_cast<const float4*>(x) + 2 * i + 1);
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] *= g;
    store8(out + i * 8, f);
  }
  for (int64_t i = nvec * 8 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nt) out[i] = __float2bfloat16_rn((float)x[i] * g);
}

// ------------------------------------------------------------------------------------------ AdamW on a flat shard
// p32: fp32 master, m/v: fp32 moments, g: bf16 or fp32 gradient, p16: bf16 working copy (optional).
// clip_coef (device, optional) multiplies the gradient: it is min(1, max_norm / (norm + 1e-6)) computed on the device.
template <typename GT>
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p32, __nv_bfloat16* __restrict__ p16, const GT* __restrict__ g,
                                                    float* __restrict__ m, float* __restrict__ v, int64_t n, float lr, float b1,
                                                    float b2, float eps, float wd, float bc1, float bc2,
                                                    const float* __restrict__ clip_coef, float grad_scale, int decoupled) {
  const float gs = grad_scale * (clip_coef != nullptr ? *clip_coef : 1.f);
  if (!isfinite(gs)) return;  // non-finite gradient norm: leave parameters and moments untouched
  const float inv_bc1 = 1.f / bc1, inv_bc2 = 1.f / bc2, decay = decoupled ? (1.f - lr * wd) : 1.f;
  auto update = [&](float& p, float& mi, float& vi, float gr) {
    gr *= gs;
    if (!decoupled) gr += wd * p;
    mi = b1 * mi + (1.f - b1) * gr;
    vi = b2 * vi + (1.f - b2) * gr * gr;
    p = p * decay - lr * (mi * inv_bc1) / (sqrtf(vi * inv_bc2) + eps);
  };
  // 4 elements per thread per iteration, 16-byte accesses when every base pointer allows it
  const bool vec = ((reinterpret_cast<uintptr_t>(p32) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(g) & (sizeof(GT) * 4 - 1)) == 0 &&
                   (p16 == nullptr || (reinterpret_cast<uintptr_t>(p16) & 7) == 0);
  const int64_t n4 = vec ? n / 4 : 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    float4 p = reinterpret_cast<float4*>(p32)[i];
    float4 mm = reinterpret_cast<float4*>(m)[i];
    float4 vv = reinterpret_cast<float4*>(v)[i];
    float gr[4];
    if constexpr (sizeof(GT) == 2) {
      const uint2 u = reinterpret_cast<const uint2*>(g)[i];
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
      gr[0] = a.x; gr[1] = a.y; gr[2] = b.x; gr[3] = b.y;
    } else {
      const float4 u = reinterpret_cast<const float4*>(g)[i];
      gr[0] = u.x; gr[1] = u.y; gr[2] = u.z; gr[3] = u.w;
    }
    update(p.x, mm.x, vv.x, gr[0]);
    update(p.y, mm.y, vv.y, gr[1]);
    update(p.z, mm.z, vv.z, gr[2]);
    update(p.w, mm.w, vv.w, gr[3]);
    reinterpret_cast<float4*>(p32)[i] = p;
    reinterpret_cast<float4*>(m)[i] = mm;
    reinterpret_cast<float4*>(v)[i] = vv;
    if (p16 != nullptr) {
      uint2 o;
      o.x = pack_bf16x2(p.x, p.y);
      o.y = pack_bf16x2(p.z, p.w);
      reinterpret_cast<uint2*>(p16)[i] = o;
    }
  }
  for (int64_t i = n4 * 4 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float gr;
    if constexpr (sizeof(GT) == 2) gr = __bfloat162float(g[i]);
    else gr = g[i];
    float p = p32[i], mi = m[i], vi = v[i];
    update(p, mi, vi, gr);
    p32[i] = p; m[i] = mi; v[i] = vi;
    if (p16 != nullptr) p16[i] = __float2bfloat16_rn(p);
  }
}

// ------------------------------------------------------------------------------------------ squared norm
// Deterministic two-stage sum of squares: stage 1 writes one partial per block into `scratch`, stage 2 (one
// block) adds them in index order into out[0] (accumulating when `accumulate`).
template <typename T>
__global__ void __launch_bounds__(256) sqnorm_partial_kernel(const T* __restrict__ x, int64_t n, float* __restrict__ scratch) {
  __shared__ float red[32];
  float s = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float f;
    if constexpr (sizeof(T) == 2) f = __bfloat162float(x[i]);
    else f = x[i];
    s += f * f;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) scratch[blockIdx.x] = s;
}
// Streaming 16-byte load that stays where it is written: a batch of them is in flight before the first result is used (left to
// itself the compiler folds each load into the chain of additions and keeps two in flight).
__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// The same sums, bit for bit, from 16-byte loads (x on a 16-byte boundary): a warp stands for one block of the kernel above and a
// lane for eight of its neighbouring threads, whose private sums it keeps apart; the shuffles then pair the sums exactly as
// that block's reduction does (a warp of the block is four lanes here). Bound by memory; 256 bytes in flight per
// thread make up for the eight warps per SM. 193 M bf16 values: 67 us against 114 us (60 us at copy speed; with a launch bound that let ptxas keep only two loads in flight: 159 us). Results keep
// their bits because a clip coefficient off by one part in 1e7 already moves bf16 parameters that lie between two values.
template <typename T>
__global__ void __launch_bounds__(256, 1) sqnorm_partial_vec_kernel(const T* __restrict__ x, int64_t n, int nblocks, float* __restrict__ scratch) {
  constexpr int kWords = sizeof(T) == 2 ? 1 : 2, U = sizeof(T) == 2 ? 16 : 8;
  const int lane = threadIdx.x & 31, vb = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (vb >= nblocks) return;
  const int64_t nt = (int64_t)nblocks * 256;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  auto add = [&](const uint4* u) {
    float f[8];
    if constexpr (kWords == 1) unpack8(u[0], f);
    else {
      f[0] = __uint_as_float(u[0].x); f[1] = __uint_as_float(u[0].y); f[2] = __uint_as_float(u[0].z); f[3] = __uint_as_float(u[0].w);
      f[4] = __uint_as_float(u[1].x); f[5] = __uint_as_float(u[1].y); f[6] = __uint_as_float(u[1].z); f[7] = __uint_as_float(u[1].w);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] += f[e] * f[e];
  };
  int64_t i = (int64_t)vb * 256 + lane * 8;
  auto batch = [&](auto nc) -> bool {                  // N vectors, all in flight before the first is added; false: fewer are left
    constexpr int N = decltype(nc)::value;
    if (i + (N - 1) * nt + 8 > n) return false;
    uint4 u[N][kWords];
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int w = 0; w < kWords; ++w) u[k][w] = ld_stream(reinterpret_cast<const uint4*>(x + i + k * nt) + w);
#pragma unroll
    for (int k = 0; k < N; ++k) add(u[k]);
    i += N * nt;
    return true;
  };
  while (batch(std::integral_constant<int, U>{})) {}
  // the rest in halving batches: one vector after another, up to U - 1 of them were as long a chain as the whole of a mid-sized tensor
  // (4.6 M bf16 values 11.7 us, against 8.6 with the scalar loads below)
  if constexpr (U > 8) batch(std::integral_constant<int, 8>{});
  batch(std::integral_constant<int, 4>{});
  batch(std::integral_constant<int, 2>{});
  batch(std::integral_constant<int, 1>{});
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (i + e < n) {
      const float f = (float)x[i + e];
      s[e] += f * f;
    }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
    s[e] += __shfl_xor_sync(0xffffffffu, s[e], 1);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (e < o) s[e] += s[e + o];
  float t = s[0];
#pragma unroll
  for (int o = 16; o >= 4; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) scratch[vb] = t;
}
__global__ void __launch_bounds__(256) sqnorm_final_kernel(const float* __restrict__ scratch, int nparts,
                                                           float* __restrict__ out, int accumulate) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += scratch[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + s : s;
}
// clip_coef[0] = min(1, max_norm / (sqrt(total_sq[0]) + 1e-6)); norm_out[0] = sqrt(total_sq[0]); finite[0] = isfinite
__global__ void clip_coef_kernel(const float* __restrict__ total_sq, float max_norm, float* __restrict__ clip_coef,
                                 float* __restrict__ norm_out, int* __restrict__ finite) {
  const float n = sqrtf(total_sq[0]);
  norm_out[0] = n;
  clip_coef[0] = isfinite(n) ? fminf(1.f, max_norm / (n + 1e-6f)) : NAN;
  if (finite != nullptr) finite[0] = isfinite(n) ? 1 : 0;
}

int sm_count();   // gemm.cu: SMs of the current device

static inline int grid_for(int64_t n, int threads, int per_sm = 8) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sm_count() * per_sm;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace llmt

using namespace llmt;

#define LLMT_CHECK_LAUNCH() return (cudaGetLastError() == cudaSuccess) ? 0 : -3

// Is one of the addresses off a 16-byte boundary? The launchers refuse those (-10): the kernels load and store 16 bytes at a time.
static inline bool off16(std::initializer_list<const void*> ps) {
  uintptr_t a = 0;
  for (const void* p : ps) a |= reinterpret_cast<uintptr_t>(p);
  return (a & 15) != 0;
}

// The forward by width: the smallest thread group that covers a row with one vector per thread, up to 256 threads (two or four
// vectors beyond). A row's time is the chain load - reduce - store, which a second vector lengthens, and the two-vector groups of 64 and
// 128 threads take 40 registers, so that only 12 of 16 blocks of the grid are resident. us without / with the residual, two vectors on
// half the threads -> one vector: 2048 x 704 3.4 / 4.0 -> 3.0 / 3.7, 2048 x 1344 5.1 / 7.5 -> 4.2 / 5.7, 13434 x 1024 13.6 / 20.7 ->
// 11.8 / 20.2, 13434 x 2048 25.6 / 45.8 -> 22.2 / 38.2. Rows of 257 to 512 are the exception once there is more than a wave of
// blocks of eight rows: 13434 x 512 5.9 / 10.1 us with a warp per row against 6.2 / 10.9, but 2048 x 512 3.0 / 3.6 against 2.6 / 3.6.
template <typename F>
static inline void fwd_by_row_width(int T, int D, F&& f) {
  using std::integral_constant;
  if (D <= 256) f(integral_constant<int, 1>{}, integral_constant<int, 32>{});
  else if (D <= 512 && T > 64 * sm_count()) f(integral_constant<int, 2>{}, integral_constant<int, 32>{});
  else if (D <= 512) f(integral_constant<int, 1>{}, integral_constant<int, 64>{});
  else if (D <= 1024) f(integral_constant<int, 1>{}, integral_constant<int, 128>{});
  else if (D <= 2048) f(integral_constant<int, 1>{}, integral_constant<int, 256>{});
  else if (D <= 4096) f(integral_constant<int, 2>{}, integral_constant<int, 256>{});
  else f(integral_constant<int, 4>{}, integral_constant<int, 256>{});
}
// The backward by width: the smallest thread group that covers a row with two vectors per thread (it prefetches the next row, so its
// chain is hidden, and fewer groups mean fewer partial sums); above 4096 two vectors on 512 threads, as four would spill.
template <typename F>
static inline void bwd_by_row_width(int D, F&& f) {
  using std::integral_constant;
  if (D <= 512) f(integral_constant<int, 2>{}, integral_constant<int, 32>{});
  else if (D <= 1024) f(integral_constant<int, 2>{}, integral_constant<int, 64>{});
  else if (D <= 2048) f(integral_constant<int, 2>{}, integral_constant<int, 128>{});
  else if (D <= 4096) f(integral_constant<int, 2>{}, integral_constant<int, 256>{});
  else f(integral_constant<int, 2>{}, integral_constant<int, 512>{});
}

extern "C" int llmt_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* sum_out, float* rstd, int T,
                                int D, float eps, cudaStream_t st) {
  if (T <= 0) return 0;
  if (D % 8 || D > 8 * kRowThreads * 4 || off16({x, res, w, y, sum_out})) return -10;
  auto X = (const __nv_bfloat16*)x; auto R = (const __nv_bfloat16*)res; auto W = (const __nv_bfloat16*)w;
  auto Y = (__nv_bfloat16*)y; auto S = (__nv_bfloat16*)sum_out;
  fwd_by_row_width(T, D, [&](auto nv, auto tr) {
    constexpr int TR = decltype(tr)::value, NT = TR > 32 ? TR : kRowThreads, RPB = NT / TR;
    const int blocks = (T + RPB - 1) / RPB, cap = sm_count() * (2048 / NT);
    rmsnorm_fwd_kernel<decltype(nv)::value, TR><<<blocks < cap ? blocks : cap, NT, 0, st>>>(X, R, W, Y, S, rstd, T, D, eps);
  });
  LLMT_CHECK_LAUNCH();
}

// dw_partial: fp32 scratch of llmt_rmsnorm_bwd_partials(T) * D floats.
// Two row blocks per SM, at most 296 (the allocation-free entry point in noalloc.cu sizes its scratch for that bound).
extern "C" int llmt_rmsnorm_bwd_partials(int T) {
  const int cap = sm_count() * 2 < 296 ? sm_count() * 2 : 296;
  return T < cap ? (T < 1 ? 1 : T) : cap;
}
extern "C" int llmt_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                                float* dw_partial, float* dw_f32, void* dw_bf16, int accumulate, int T, int D,
                                cudaStream_t st) {
  if (T <= 0) return 0;
  if (D % 8 || D > 8 * kRowThreads * 4 || off16({dy, x, w, dres, dx, dw_partial})) return -10;
  auto DY = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w;
  auto DR = (const __nv_bfloat16*)dres; auto DX = (__nv_bfloat16*)dx;
  int grid = 0;
  bwd_by_row_width(D, [&](auto nv, auto tr) {
    constexpr int NV = decltype(nv)::value, TR = decltype(tr)::value, NT = RowBlock<TR>::kThreads, RPB = RowBlock<TR>::kRows;
    const int blocks = (T + RPB - 1) / RPB, most = llmt_rmsnorm_bwd_partials(T), cap = NT > 256 ? (most + 1) / 2 : most;
    grid = blocks < cap ? blocks : cap;
    rmsnorm_bwd_kernel<NV, TR><<<grid, NT, 0, st>>>(DY, X, W, rstd, DR, DX, dw_partial, T, D);
  });
  colsum_kernel<<<(D + 31) / 32, 1024, 0, st>>>(dw_partial, dw_f32, (__nv_bfloat16*)dw_bf16, grid, D, accumulate);
  LLMT_CHECK_LAUNCH();
}

// out[c] = sum over P rows of partial [P][D], into fp32 or bf16.
extern "C" int llmt_colsum(const float* partial, float* out_f32, void* out_bf16, int P, int D, cudaStream_t st) {
  if (D <= 0) return 0;
  colsum_kernel<<<(D + 31) / 32, 1024, 0, st>>>(partial, out_f32, (__nv_bfloat16*)out_bf16, P, D, 0);
  LLMT_CHECK_LAUNCH();
}

extern "C" int llmt_qk_norm_rope_fwd(const void* x, int64_t tok_stride, const void* w, const float* cosb, const float* sinb,
                                     void* y, int64_t y_tok_stride, float* rstd, int T, int H, int HD, float eps,
                                     cudaStream_t st) {
  if (T <= 0 || H <= 0) return 0;
  if ((tok_stride & 3) || (y_tok_stride & 3) || (reinterpret_cast<uintptr_t>(x) & 7) || (reinterpret_cast<uintptr_t>(y) & 7)) return -10;
  const int64_t items = (int64_t)T * H;
  const int ipw = HD == 64 ? 4 : (HD == 128 ? 2 : 1);          // items per warp
  const int grid = (int)((items + 8 * ipw - 1) / (8 * ipw));
  auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w; auto Y = (__nv_bfloat16*)y;
  if (HD == 64) qk_norm_rope_fwd_kernel<1><<<grid, 256, 0, st>>>(X, tok_stride, W, cosb, sinb, Y, y_tok_stride, rstd, T, H, eps);
  else if (HD == 128) qk_norm_rope_fwd_kernel<2><<<grid, 256, 0, st>>>(X, tok_stride, W, cosb, sinb, Y, y_tok_stride, rstd, T, H, eps);
  else if (HD == 256) qk_norm_rope_fwd_kernel<4><<<grid, 256, 0, st>>>(X, tok_stride, W, cosb, sinb, Y, y_tok_stride, rstd, T, H, eps);
  else return -10;
  LLMT_CHECK_LAUNCH();
}

extern "C" int llmt_qk_norm_rope_bwd_partials(int T, int H) {
  const int64_t items = (int64_t)T * H;
  const int64_t b = (items + 7) / 8;
  const int64_t cap = (int64_t)sm_count() * 4;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}
extern "C" int llmt_qk_norm_rope_bwd(const void* dy, int64_t dy_tok_stride, const void* x, int64_t tok_stride, const void* w,
                                     const float* cosb, const float* sinb, const float* rstd, void* dx,
                                     int64_t dx_tok_stride, float* dw_partial, float* dw_f32, void* dw_bf16,
                                     int accumulate, int T, int H, int HD, cudaStream_t st) {
  if (T <= 0 || H <= 0) return 0;
  if ((tok_stride & 3) || (dy_tok_stride & 3) || (dx_tok_stride & 3) || (reinterpret_cast<uintptr_t>(x) & 7) ||
      (reinterpret_cast<uintptr_t>(dy) & 7) || (reinterpret_cast<uintptr_t>(dx) & 7))
    return -10;
  const int grid = llmt_qk_norm_rope_bwd_partials(T, H);
  auto DY = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w;
  auto DX = (__nv_bfloat16*)dx;
  if (HD == 64) qk_norm_rope_bwd_kernel<1><<<grid, 256, 0, st>>>(DY, dy_tok_stride, X, tok_stride, W, cosb, sinb, rstd, DX, dx_tok_stride, dw_partial, T, H);
  else if (HD == 128) qk_norm_rope_bwd_kernel<2><<<grid, 256, 0, st>>>(DY, dy_tok_stride, X, tok_stride, W, cosb, sinb, rstd, DX, dx_tok_stride, dw_partial, T, H);
  else if (HD == 256) qk_norm_rope_bwd_kernel<4><<<grid, 256, 0, st>>>(DY, dy_tok_stride, X, tok_stride, W, cosb, sinb, rstd, DX, dx_tok_stride, dw_partial, T, H);
  else return -10;
  if (w != nullptr && dw_partial != nullptr)
    colsum_kernel<<<(HD + 31) / 32, 1024, 0, st>>>(dw_partial, dw_f32, (__nv_bfloat16*)dw_bf16, grid, HD, accumulate);
  LLMT_CHECK_LAUNCH();
}

extern "C" int llmt_attn_rows_probs(const float* s, const float* lse, void* p, int64_t rows, int C, int n, int diag, float scale,
                                    int causal, cudaStream_t st) {
  if (rows <= 0 || C <= 0) return 0;
  if (n <= 0) return -10;
  const int64_t cap = (int64_t)sm_count() * 8;
  attn_rows_probs_kernel<<<(int)(rows < cap ? rows : cap), 256, 0, st>>>(s, lse, (__nv_bfloat16*)p, rows, C, n, diag,
                                                                          scale * 1.4426950408889634f, causal);
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_attn_rows_ds(const float* dp, const void* p, const float* delta, void* ds, int64_t rows, int C, cudaStream_t st) {
  if (rows <= 0 || C <= 0) return 0;
  const int64_t cap = (int64_t)sm_count() * 8;
  attn_rows_ds_kernel<<<(int)(rows < cap ? rows : cap), 256, 0, st>>>(dp, (const __nv_bfloat16*)p, delta, (__nv_bfloat16*)ds, rows, C);
  LLMT_CHECK_LAUNCH();
}

extern "C" int llmt_swiglu_fwd(const void* gate, const void* up, void* out, int64_t T, int F, int64_t ld_in, int64_t ld_out,
                               const int* row_limit, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8 || ld_in % 8 || ld_out % 8) return -10;
  swiglu_fwd_kernel<<<grid_for(T * (F / 8), 256), 256, 0, st>>>((const __nv_bfloat16*)gate, (const __nv_bfloat16*)up,
                                                                 (__nv_bfloat16*)out, T, F, ld_in, ld_out, row_limit);
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_swiglu_bwd(const void* dout, const void* gate, const void* up, void* dgate, void* dup, int64_t T, int F,
                               int64_t ld_in, int64_t ld_dout, int64_t ld_dg, const int* row_limit, cudaStream_t st) {
  if (T <= 0) return 0;
  if (F % 8 || ld_in % 8 || ld_dout % 8 || ld_dg % 8) return -10;
  swiglu_bwd_kernel<<<grid_for(T * (F / 8), 256), 256, 0, st>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)gate,
                                                                 (const __nv_bfloat16*)up, (__nv_bfloat16*)dgate,
                                                                 (__nv_bfloat16*)dup, T, F, ld_in, ld_dout, ld_dg, row_limit);
  LLMT_CHECK_LAUNCH();
}

extern "C" int llmt_ce_fwd_bwd(void* logits, const int64_t* labels, float* row_loss, float* row_lse, int rows, int V,
                               int64_t ld, const float* grad_scale_ptr, float grad_scale, int ignore_index, int write_grad,
                               cudaStream_t st) {
  if (rows <= 0) return 0;
  if (ld % 8 || (V >= 8 && off16({logits}))) return -10;
  auto L = (__nv_bfloat16*)logits;
  const int nvec = V / 8;
  auto go = [&](auto nt, int most) {                       // `most`: vectors of a row that may be cached
    constexpr int NT = decltype(nt)::value;
    const int cached = !write_grad ? 0 : (nvec < most ? nvec : most);
    if (most * 16 > 48 * 1024)
      cudaFuncSetAttribute(ce_fwd_bwd_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most * 16);
    ce_fwd_bwd_kernel<NT><<<rows, NT, (size_t)cached * 16, st>>>(L, labels, row_loss, row_lse, V, ld, grad_scale_ptr, grad_scale, ignore_index,
                                                                 write_grad, cached);
  };
  // With more rows than SMs, rows in flight times their size decides: up to 150 KB a row, four blocks of 512 threads per SM stay
  // inside L2 (592 rows); beyond that two blocks of 1024 with 64 KB of each row in shared memory do. Without gradients nothing is
  // read twice: 512 threads there too, and 256 for more than four rows per SM of up to 51200 columns. Measured us, 256 / 512 / 1024 threads at 1000 x 4096: 6.8 / 8.6 / 13, 4000 x 32000: 98 / 96 / 114,
  // 2000 x 50000: 95 / 80 / 89, 2000 x 151936: 300 / 274 / 247; no gradients 4000 x 20536: 33 / 41 / 59, 1000 x 76800: 31.5 / 30.7 / 33.6,
  // 4000 x 76808: 101 / 103 / 121.
  // Up to one row per SM it is the chain of one row: 110 x 4096 2.8 / 2.9 / 3.1, 40 x 11728 4.4 / 3.8 / 4.2, 40 x 20536 6.3 / 5.5 / 4.9,
  // 110 x 76800 25 / 17 / 13.
  const bool few = rows <= sm_count();
  using std::integral_constant;
  if (V <= (few ? 4096 : 8192) || (!write_grad && rows > 4 * sm_count() && V <= 51200)) go(integral_constant<int, 256>{}, 1024);
  else if (V <= (few ? 16384 : 76800) || !(few || write_grad)) go(integral_constant<int, 512>{}, 2560);
  else go(integral_constant<int, 1024>{}, 4096);
  LLMT_CHECK_LAUNCH();
}

// x and out on 16-byte boundaries.
extern "C" int llmt_scale_to_bf16(const void* x, int is_bf16, const float* scale, void* out, int64_t n, cudaStream_t st) {
  if (n <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) return -10;
  const int grid = grid_for((n + 7) / 8, 256);
  if (is_bf16) scale_to_bf16_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)x, scale, (__nv_bfloat16*)out, n);
  else scale_to_bf16_kernel<float><<<grid, 256, 0, st>>>((const float*)x, scale, (__nv_bfloat16*)out, n);
  LLMT_CHECK_LAUNCH();
}

extern "C" int llmt_adamw(float* p32, void* p16, const void* g, int g_is_bf16, float* m, float* v, int64_t n, float lr,
                          float b1, float b2, float eps, float wd, int step, const float* clip_coef, float grad_scale,
                          int decoupled, cudaStream_t st) {
  if (n <= 0) return 0;
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  const int grid = grid_for((n + 3) / 4, 256, 16);
  if (g_is_bf16)
    adamw_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(p32, (__nv_bfloat16*)p16, (const __nv_bfloat16*)g, m, v, n, lr, b1, b2,
                                                       eps, wd, bc1, bc2, clip_coef, grad_scale, decoupled);
  else
    adamw_kernel<float><<<grid, 256, 0, st>>>(p32, (__nv_bfloat16*)p16, (const float*)g, m, v, n, lr, b1, b2, eps, wd, bc1,
                                               bc2, clip_coef, grad_scale, decoupled);
  LLMT_CHECK_LAUNCH();
}

// scratch must hold llmt_sqnorm_scratch_floats() floats.
extern "C" int llmt_sqnorm_scratch_floats() { return sm_count() * 8; }
extern "C" int llmt_sqnorm(const void* x, int is_bf16, int64_t n, float* scratch, float* out, int accumulate,
                           cudaStream_t st) {
  if (n <= 0) {
    if (!accumulate) cudaMemsetAsync(out, 0, sizeof(float), st);
    return 0;
  }
  const int grid = grid_for(n, 256);
  if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    if (is_bf16) sqnorm_partial_vec_kernel<__nv_bfloat16><<<(grid + 7) / 8, 256, 0, st>>>((const __nv_bfloat16*)x, n, grid, scratch);
    else sqnorm_partial_vec_kernel<float><<<(grid + 7) / 8, 256, 0, st>>>((const float*)x, n, grid, scratch);
  } else if (is_bf16) sqnorm_partial_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)x, n, scratch);
  else sqnorm_partial_kernel<float><<<grid, 256, 0, st>>>((const float*)x, n, scratch);
  sqnorm_final_kernel<<<1, 256, 0, st>>>(scratch, grid, out, accumulate);
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_clip_coef(const float* total_sq, float max_norm, float* clip_coef, float* norm_out, int* finite,
                              cudaStream_t st) {
  clip_coef_kernel<<<1, 1, 0, st>>>(total_sq, max_norm, clip_coef, norm_out, finite);
  LLMT_CHECK_LAUNCH();
}
