// Kernels around the gated delta rule for sm_100a (reference call sites: llmtuner/models/qwen/qwen3_5_moe/gated_delta.py:13-189,
// llmtuner/models/kimi/kimi_k3/causal_convolution.py): the short causal convolution with SiLU, the split of its output into
// normalised queries / keys and values, and the gated RMSNorm of the mixer's output. Each is one pass over its data with
// fp32 arithmetic and one rounding; as tensor expressions they were chains of 8 to 20 elementwise kernels, each rounding to bf16.
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace llmt {

__device__ __forceinline__ void up8(const uint4& u, float* f) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(b[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 down8(const float* f) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }

// ------------------------------------------------------------------------------------------ causal convolution + SiLU
// z[t, c] = sum_j x[t - j, c] * w[c, K - 1 - j] over j = 0 and the taps j <= pos[t] (the index of row t in its document); y = silu(z).
// A thread owns 8 channels and walks the `tok` rows of its block with the last K rows in registers, so every row is read once (plus
// K - 1 rows per block). Bound by the latency of one row's loads per thread: at 96 and 144 registers 28 % and 17 % of the warps are
// resident, DRAM is at 30 % and 22 %, issue slots at 37 % and 43 %; the backward also writes and sums fp32 partials of the weight gradient
// ([blocks, C, K], 17 MB at 2048 x 8192). 2048 x 8192, K = 4: 26 us forward, 82 us backward (67 and 100 MB; as tensor expressions
// about 1.1 ms together).
// 16 rows per block; rows of more than 16 x kConvBlocks tokens get longer blocks, which bounds the grid (gridDim.y ends at 65535) and the
// partial sums of the weight gradient.
constexpr int kConvTok = 16, kConvBlocks = 4096;
template <int K>
__global__ void __launch_bounds__(128) conv_silu_fwd_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, const __nv_bfloat16* __restrict__ w,
                                                            const int64_t* __restrict__ pos, __nv_bfloat16* __restrict__ y, int T, int C, int tok) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (c >= C) return;
  float wt[8][K];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < K; ++j) wt[i][j] = __bfloat162float(w[(int64_t)(c + i) * K + K - 1 - j]);   // wt[.][j]: tap j rows back
  const int t0 = blockIdx.y * tok, t1 = min(T, t0 + tok);
  uint4 win[K];                                        // win[j]: row t - j
#pragma unroll
  for (int j = 1; j < K; ++j) win[j - 1] = t0 - j >= 0 ? *reinterpret_cast<const uint4*>(x + (int64_t)(t0 - j) * ldx + c) : make_uint4(0, 0, 0, 0);
#pragma unroll 4
  for (int t = t0; t < t1; ++t) {
#pragma unroll
    for (int j = K - 1; j > 0; --j) win[j] = win[j - 1];
    win[0] = *reinterpret_cast<const uint4*>(x + (int64_t)t * ldx + c);
    const int64_t p = pos[t];
    float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (j > 0 && p < j) continue;
      float f[8];
      up8(win[j], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) z[i] += f[i] * wt[i][j];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] *= sigmoid_f(z[i]);
    *reinterpret_cast<uint4*>(y + (int64_t)t * C + c) = down8(z);
  }
}

// dz = dy * silu'(z) with z rebuilt from x; dx[t] = sum_j dz[t + j] * w[K - 1 - j] over rows t + j with pos >= j; the weight
// gradient of the block's rows goes to dw_part[blockIdx.y][C][K]. Rows are walked downwards: dz of rows t .. t + K - 1 is at hand.
template <int K>
__global__ void __launch_bounds__(128) conv_silu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, int64_t lddy, const __nv_bfloat16* __restrict__ x,
                                                            int64_t ldx, const __nv_bfloat16* __restrict__ w, const int64_t* __restrict__ pos,
                                                            __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part, int T, int C, int tok) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (c >= C) return;
  float wt[8][K], dw[8][K];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < K; ++j) { wt[i][j] = __bfloat162float(w[(int64_t)(c + i) * K + K - 1 - j]); dw[i][j] = 0.f; }
  const int t0 = blockIdx.y * tok, t1 = min(T, t0 + tok), last = min(T, t1 + K - 1) - 1;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 win[K];                                        // win[j]: row t - j
#pragma unroll
  for (int j = 0; j < K; ++j) win[j] = last - j >= 0 ? *reinterpret_cast<const uint4*>(x + (int64_t)(last - j) * ldx + c) : zero;
  float dz[K][8];                                      // dz[j]: row t + j
  int64_t ps[K];                                       // ps[j]: pos of row t + j
#pragma unroll
  for (int j = 0; j < K; ++j) {
    ps[j] = -1;
#pragma unroll
    for (int i = 0; i < 8; ++i) dz[j][i] = 0.f;
  }
  for (int t = last; t >= t0; --t) {
#pragma unroll
    for (int j = K - 1; j > 0; --j) {
      ps[j] = ps[j - 1];
#pragma unroll
      for (int i = 0; i < 8; ++i) dz[j][i] = dz[j - 1][i];
    }
    ps[0] = pos[t];
    const uint4 next = t - K >= 0 ? *reinterpret_cast<const uint4*>(x + (int64_t)(t - K) * ldx + c) : zero;
    float d[8], z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    up8(*reinterpret_cast<const uint4*>(dy + (int64_t)t * lddy + c), d);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (j > 0 && ps[0] < j) continue;
      float f[8];
      up8(win[j], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) z[i] += f[i] * wt[i][j];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = sigmoid_f(z[i]);
      dz[0][i] = d[i] * (s + z[i] * s * (1.f - s));
    }
    if (t < t1) {
      float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (j > 0 && ps[j] < j) continue;              // also rows beyond the last one (pos -1)
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += dz[j][i] * wt[i][j];
      }
      *reinterpret_cast<uint4*>(dx + (int64_t)t * C + c) = down8(o);
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (j > 0 && ps[0] < j) continue;
        float f[8];
        up8(win[j], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) dw[i][j] += dz[0][i] * f[i];
      }
    }
#pragma unroll
    for (int j = 0; j + 1 < K; ++j) win[j] = win[j + 1];
    win[K - 1] = next;
  }
  float* o = dw_part + ((int64_t)blockIdx.y * C + c) * K;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < K; ++j) o[i * K + K - 1 - j] = dw[i][j];
}

// ------------------------------------------------------------------------------------------ q, k, v of the delta rule
// mixed [T, 2 Hk d + Hv dv] bf16 -> q, k [T, Hv, d] fp32 (each key head L2-normalised, q scaled by qscale, repeated for the value
// heads of its group), v [T, Hv, dv] fp32. A group of d / 8 lanes per (token, head); d, dv in {64, 128, 256}.
template <int G>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void st8f(float* p, const float* f) {
  reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void ld8f(const float* p, float* f) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <int G>      // head width 8 * G for keys and values
__global__ void __launch_bounds__(256) delta_qkv_fwd_kernel(const __nv_bfloat16* __restrict__ mixed, float* __restrict__ q, float* __restrict__ k,
                                                            float* __restrict__ v, int64_t T, int Hk, int Hv, float qscale, float eps) {
  constexpr int D = 8 * G, IPW = 32 / G;
  const int lane = threadIdx.x & 31, g = lane % G, slots = 2 * Hk + Hv, rep = Hv / Hk;
  const int64_t total = T * slots;
  int64_t item = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * IPW + lane / G;
  const bool live = item < total;
  if (!live) item = total - 1;                         // keep the warp whole for the shuffles
  const int64_t t = item / slots;
  const int s = (int)(item % slots);
  float f[8];
  up8(*reinterpret_cast<const uint4*>(mixed + t * (int64_t)slots * D + (int64_t)s * D + g * 8), f);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  ss = lanes_sum<G>(ss);
  if (!live) return;
  if (s >= 2 * Hk) {
    st8f(v + (t * Hv + s - 2 * Hk) * D + g * 8, f);
    return;
  }
  const float r = rsqrtf(ss + eps) * (s < Hk ? qscale : 1.f);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] *= r;
  float* o = (s < Hk ? q : k) + (t * Hv + (int64_t)(s % Hk) * rep) * D + g * 8;
  for (int i = 0; i < rep; ++i) st8f(o + (int64_t)i * D, f);
}
// n = x * r, r = (|x|^2 + eps)^-1/2 : dx = scale * (r * dn - x * r^3 * <x, dn>), dn summed over the value heads of the group.
template <int G>
__global__ void __launch_bounds__(256) delta_qkv_bwd_kernel(const float* __restrict__ dq, const float* __restrict__ dk, const float* __restrict__ dv,
                                                            const __nv_bfloat16* __restrict__ mixed, __nv_bfloat16* __restrict__ dmixed, int64_t T,
                                                            int Hk, int Hv, float qscale, float eps) {
  constexpr int D = 8 * G, IPW = 32 / G;
  const int lane = threadIdx.x & 31, g = lane % G, slots = 2 * Hk + Hv, rep = Hv / Hk;
  const int64_t total = T * slots;
  int64_t item = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * IPW + lane / G;
  const bool live = item < total;
  if (!live) item = total - 1;
  const int64_t t = item / slots;
  const int s = (int)(item % slots);
  const int64_t at = t * (int64_t)slots * D + (int64_t)s * D + g * 8;
  float d[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (s >= 2 * Hk) {
    ld8f(dv + (t * Hv + s - 2 * Hk) * D + g * 8, d);
  } else {
    const float* p = (s < Hk ? dq : dk) + (t * Hv + (int64_t)(s % Hk) * rep) * D + g * 8;
    for (int i = 0; i < rep; ++i) {
      float u[8];
      ld8f(p + (int64_t)i * D, u);
#pragma unroll
      for (int j = 0; j < 8; ++j) d[j] += u[j];
    }
  }
  float f[8], ss = 0.f, xd = 0.f;
  up8(*reinterpret_cast<const uint4*>(mixed + at), f);
#pragma unroll
  for (int i = 0; i < 8; ++i) { ss += f[i] * f[i]; xd += f[i] * d[i]; }
  ss = lanes_sum<G>(ss);
  xd = lanes_sum<G>(xd);
  if (!live) return;
  if (s < 2 * Hk) {
    const float r = rsqrtf(ss + eps), sc = s < Hk ? qscale : 1.f, c = r * r * r * xd;
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = sc * (r * d[i] - f[i] * c);
  }
  *reinterpret_cast<uint4*>(dmixed + at) = down8(d);
}

// ------------------------------------------------------------------------------------------ gated RMSNorm
// y = x * rsqrt(mean x^2 + eps) * w * silu(gate) over rows of D = 8 * G channels.
template <int G>
__global__ void __launch_bounds__(256) gated_norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gate,
                                                             const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y, int64_t R, float eps) {
  constexpr int D = 8 * G, IPW = 32 / G;
  const int lane = threadIdx.x & 31, g = lane % G;
  int64_t row = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * IPW + lane / G;
  const bool live = row < R;
  if (!live) row = R - 1;
  float f[8], a[8], wv[8], ss = 0.f;
  up8(*reinterpret_cast<const uint4*>(x + row * D + g * 8), f);
  up8(*reinterpret_cast<const uint4*>(gate + row * D + g * 8), a);
  up8(*reinterpret_cast<const uint4*>(w + g * 8), wv);
#pragma unroll
  for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  const float r = rsqrtf(lanes_sum<G>(ss) / (float)D + eps);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = f[i] * r * wv[i] * (a[i] * sigmoid_f(a[i]));
  if (live) *reinterpret_cast<uint4*>(y + row * D + g * 8) = down8(f);
}
template <int G>
__global__ void __launch_bounds__(256) gated_norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                             const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ w,
                                                             __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dgate,
                                                             float* __restrict__ dw_part, int64_t R, float eps) {
  constexpr int D = 8 * G, IPW = 32 / G, kGroups = 256 / G;
  __shared__ float parts[kGroups][D];
  const int lane = threadIdx.x & 31, g = lane % G;
  float wv[8], dw[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  up8(*reinterpret_cast<const uint4*>(w + g * 8), wv);
  const int64_t step = (int64_t)gridDim.x * 8 * IPW, rounds = (R + step - 1) / step;      // the same number of rounds for every warp
  for (int64_t rd = 0; rd < rounds; ++rd) {
    int64_t row = rd * step + ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * IPW + lane / G;
    const bool live = row < R;
    if (!live) row = R - 1;
    float f[8], a[8], d[8], ss = 0.f, c = 0.f;
    up8(*reinterpret_cast<const uint4*>(x + row * D + g * 8), f);
    up8(*reinterpret_cast<const uint4*>(gate + row * D + g * 8), a);
    up8(*reinterpret_cast<const uint4*>(dy + row * D + g * 8), d);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    const float r = rsqrtf(lanes_sum<G>(ss) / (float)D + eps);
    float dg[8], gn[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = sigmoid_f(a[i]), silu = a[i] * s, xn = f[i] * r;
      dg[i] = d[i] * xn * wv[i] * (s + silu * (1.f - s));
      if (live) dw[i] += d[i] * xn * silu;
      gn[i] = d[i] * wv[i] * silu;
      c += gn[i] * f[i];
    }
    const float k = r * r * r * lanes_sum<G>(c) / (float)D;
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = r * gn[i] - f[i] * k;
    if (live) {
      *reinterpret_cast<uint4*>(dx + row * D + g * 8) = down8(f);
      *reinterpret_cast<uint4*>(dgate + row * D + g * 8) = down8(dg);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) parts[threadIdx.x / G][g * 8 + i] = dw[i];
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += 256) {          // the groups of the block in a fixed order
    float s = 0.f;
#pragma unroll 4
    for (int i = 0; i < kGroups; ++i) s += parts[i][c];
    dw_part[(int64_t)blockIdx.x * D + c] = s;
  }
}

int sm_count();   // gemm.cu

}  // namespace llmt

using namespace llmt;
#define LLMT_CHECK_LAUNCH() return (cudaGetLastError() == cudaSuccess) ? 0 : -3

static inline int conv_tok(int T) {            // rows per block, a multiple of kConvTok
  const int64_t per = ((int64_t)T + kConvBlocks - 1) / kConvBlocks;
  return per <= kConvTok ? kConvTok : (int)((per + kConvTok - 1) / kConvTok * kConvTok);
}
extern "C" int llmt_conv_silu_blocks(int T) {
  const int tok = conv_tok(T);
  return (int)(((int64_t)T + tok - 1) / tok);
}
template <typename F>
static inline int by_taps(int K, F&& f) {
  switch (K) {
    case 2: f(std::integral_constant<int, 2>{}); return 0;
    case 3: f(std::integral_constant<int, 3>{}); return 0;
    case 4: f(std::integral_constant<int, 4>{}); return 0;
  }
  return -10;
}
extern "C" int llmt_conv_silu_fwd(const void* x, int64_t ldx, const void* w, const int64_t* pos, void* y, int T, int C, int K, cudaStream_t st) {
  if (T <= 0 || C <= 0) return 0;
  if (C % 8 || ldx % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15)) return -10;
  const dim3 grid((C / 8 + 127) / 128, llmt_conv_silu_blocks(T));
  if (by_taps(K, [&](auto k) {
        conv_silu_fwd_kernel<decltype(k)::value><<<grid, 128, 0, st>>>((const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, pos, (__nv_bfloat16*)y, T, C, conv_tok(T));
      }))
    return -10;
  LLMT_CHECK_LAUNCH();
}
// dw_part: fp32 [llmt_conv_silu_blocks(T)][C][K]; dw: bf16 [C][K].
extern "C" int llmt_conv_silu_bwd(const void* dy, int64_t lddy, const void* x, int64_t ldx, const void* w, const int64_t* pos, void* dx, float* dw_part,
                                  void* dw, int T, int C, int K, cudaStream_t st) {
  if (T <= 0 || C <= 0) return 0;
  if (C % 8 || ldx % 8 || lddy % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) & 15)) return -10;
  const dim3 grid((C / 8 + 127) / 128, llmt_conv_silu_blocks(T));
  if (by_taps(K, [&](auto k) {
        conv_silu_bwd_kernel<decltype(k)::value><<<grid, 128, 0, st>>>((const __nv_bfloat16*)dy, lddy, (const __nv_bfloat16*)x, ldx,
                                                                       (const __nv_bfloat16*)w, pos, (__nv_bfloat16*)dx, dw_part, T, C, conv_tok(T));
      }))
    return -10;
  llmt_colsum(dw_part, nullptr, dw, grid.y, C * K, st);
  LLMT_CHECK_LAUNCH();
}
template <typename F>
static inline int by_width(int D, F&& f) {
  switch (D) {
    case 64: f(std::integral_constant<int, 8>{}); return 0;
    case 128: f(std::integral_constant<int, 16>{}); return 0;
    case 256: f(std::integral_constant<int, 32>{}); return 0;
  }
  return -10;
}
extern "C" int llmt_delta_qkv_fwd(const void* mixed, float* q, float* k, float* v, int T, int Hk, int Hv, int D, float qscale, float eps, cudaStream_t st) {
  if (T <= 0) return 0;
  if (Hk < 1 || Hv % Hk || (reinterpret_cast<uintptr_t>(mixed) & 15)) return -10;
  const int64_t items = (int64_t)T * (2 * Hk + Hv), per = 8 * 256 / D;          // items per block: 8 warps of 256 / D
  if (by_width(D, [&](auto g) {
        delta_qkv_fwd_kernel<decltype(g)::value><<<(unsigned)((items + per - 1) / per), 256, 0, st>>>((const __nv_bfloat16*)mixed, q, k, v, T, Hk, Hv, qscale, eps);
      }))
    return -10;
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_delta_qkv_bwd(const float* dq, const float* dk, const float* dv, const void* mixed, void* dmixed, int T, int Hk, int Hv, int D,
                                  float qscale, float eps, cudaStream_t st) {
  if (T <= 0) return 0;
  if (Hk < 1 || Hv % Hk || ((reinterpret_cast<uintptr_t>(mixed) | reinterpret_cast<uintptr_t>(dmixed) | reinterpret_cast<uintptr_t>(dq) |
                             reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 15))
    return -10;
  const int64_t items = (int64_t)T * (2 * Hk + Hv), per = 8 * 256 / D;
  if (by_width(D, [&](auto g) {
        delta_qkv_bwd_kernel<decltype(g)::value><<<(unsigned)((items + per - 1) / per), 256, 0, st>>>(dq, dk, dv, (const __nv_bfloat16*)mixed,
                                                                                                        (__nv_bfloat16*)dmixed, T, Hk, Hv, qscale, eps);
      }))
    return -10;
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_gated_norm_fwd(const void* x, const void* gate, const void* w, void* y, int64_t R, int D, float eps, cudaStream_t st) {
  if (R <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15) return -10;
  const int64_t per = 8 * 256 / D;
  if (by_width(D, [&](auto g) {
        gated_norm_fwd_kernel<decltype(g)::value><<<(unsigned)((R + per - 1) / per), 256, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)gate,
                                                                                                    (const __nv_bfloat16*)w, (__nv_bfloat16*)y, R, eps);
      }))
    return -10;
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_gated_norm_bwd_blocks(int64_t R, int D) {
  const int64_t per = 8 * 256 / D, b = (R + per - 1) / per, cap = (int64_t)sm_count() * 4;
  return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}
// dw_part: fp32 [llmt_gated_norm_bwd_blocks(R, D)][D]; dw: bf16 [D].
extern "C" int llmt_gated_norm_bwd(const void* dy, const void* x, const void* gate, const void* w, void* dx, void* dgate, float* dw_part, void* dw,
                                   int64_t R, int D, float eps, cudaStream_t st) {
  if (R <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(w) |
       reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(dgate)) & 15)
    return -10;
  const int blocks = llmt_gated_norm_bwd_blocks(R, D);
  if (by_width(D, [&](auto g) {
        gated_norm_bwd_kernel<decltype(g)::value><<<blocks, 256, 0, st>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)gate,
                                                                          (const __nv_bfloat16*)w, (__nv_bfloat16*)dx, (__nv_bfloat16*)dgate, dw_part, R, eps);
      }))
    return -10;
  llmt_colsum(dw_part, nullptr, dw, blocks, D, st);
  LLMT_CHECK_LAUNCH();
}
