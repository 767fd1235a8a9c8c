// Helpers shared by the attention kernels (attention.cu: forward and the two-kernel backward; attention_bwd.cu: the
// single-kernel backward): exp2, shared-memory descriptor offsets of the swizzled tiles, swizzled row stores and the
// [T, H, HD] tensor maps.
#pragma once
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace llmt {

constexpr int kAttnThreads = 192;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed two-lane fp32 arithmetic (one issue slot for two elements).
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  uint64_t ra, rb, rc, rd;
  float2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  uint64_t ra, rb, rd;
  float2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  uint64_t ra, rb, rd;
  float2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}
// Warp index that the compiler knows to be the same in all lanes. The warp that issues the products walks its loop as a whole
// and lets one lane issue: with uniform control flow, descriptors and barrier addresses are computed in uniform registers,
// where tcgen05.mma takes them. In a single-thread branch every operand is moved there instruction by instruction, and beside
// two softmax warps on the same scheduler that took twice as long as the 64 clocks of a product. 8192 tokens, 32 / 8 heads of
// 128: forward 642 us -> 513 us, one-kernel backward with its passes 1726 -> 1482; 4096 tokens, 16 / 4 heads of 256, backward
// kernel 461 -> 368; nothing else changed.
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// Store 32 consecutive bf16 (packed in 16 words) of row `row`, columns [col0, col0+32) into a swizzled K-major tile.
__device__ __forceinline__ void store_row32_swz(uint8_t* tile, int row, int col0, const uint32_t* w) {
  uint8_t* base = tile + (col0 >> 6) * 16384 + row * 128;
  const int chunk0 = (col0 & 63) >> 3;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 v = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
    *reinterpret_cast<uint4*>(base + (((chunk0 + c) ^ (row & 7)) << 4)) = v;
  }
}

template <int HD>
struct AttnSmem {
  static constexpr int kTile = 128 * HD * 2;   // Q / K / V / dO tile, 128 rows
  static constexpr int kP = 128 * 128 * 2;     // P / dS tile
};

// offset (in 16-byte units) of 16-column slice `ks` of a K-major tile with `rows` rows, stored as 64-column halves of [rows][128 B] / of
// 16-row slice `ks` of the same tile read as an MN-major operand (rows = reduction index)
__host__ __device__ constexpr uint32_t koff(int ks, int rows) { return (uint32_t)(((ks >> 2) * (rows * 128) + (ks & 3) * 32) >> 4); }
__host__ __device__ constexpr uint32_t mnoff(int ks) { return (uint32_t)((ks * 2048) >> 4); }

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; with `acc` the fp32 rows acc[t, h, :] are cleared too (the dQ accumulator of the
// one-kernel backward, which needs it before its first add). Bound by memory. A block owns 16 tokens x 8 heads: each group of
// 16 lanes walks the heads of one token with 16-byte accesses, and the sums leave as 64-byte runs per head. 8192 tokens x 32
// heads x 128: 45 us for 268 MB; as a 4-byte-per-lane kernel with one scattered store per warp, plus a memset, 80 us.
static __global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, int64_t o_stride,
                                                                const __nv_bfloat16* __restrict__ d_o, int64_t do_stride,
                                                                float* __restrict__ delta, float* __restrict__ acc, int T, int H, int HD) {
  constexpr int kTok = 16, kHeads = 8;
  __shared__ float sums[kHeads][kTok + 1];
  const int grp = threadIdx.x >> 4, gl = threadIdx.x & 15;
  const int t = blockIdx.x * kTok + grp, h0 = blockIdx.y * kHeads;
  float s[kHeads];
#pragma unroll
  for (int i = 0; i < kHeads; ++i) s[i] = 0.f;
  if (t < T) {
    for (int c = gl * 8; c < HD; c += 128) {
      uint4 a[kHeads], b[kHeads];
#pragma unroll
      for (int i = 0; i < kHeads; ++i) {
        const int h = min(h0 + i, H - 1);
        a[i] = *reinterpret_cast<const uint4*>(o + (int64_t)t * o_stride + (int64_t)h * HD + c);
        b[i] = *reinterpret_cast<const uint4*>(d_o + (int64_t)t * do_stride + (int64_t)h * HD + c);
      }
      if (acc != nullptr) {
#pragma unroll
        for (int i = 0; i < kHeads; ++i)
          if (h0 + i < H) {
            float4* z = reinterpret_cast<float4*>(acc + ((int64_t)t * H + h0 + i) * HD + c);
            z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
            z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
      }
#pragma unroll
      for (int i = 0; i < kHeads; ++i) {
        const __nv_bfloat162 *pa = reinterpret_cast<const __nv_bfloat162*>(&a[i]), *pb = reinterpret_cast<const __nv_bfloat162*>(&b[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 x = __bfloat1622float2(pa[j]), y = __bfloat1622float2(pb[j]);
          s[i] += x.x * y.x + x.y * y.y;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kHeads; ++i) {
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], w);
    if (gl == 0) sums[i][grp] = s[i];
  }
  __syncthreads();
  if (threadIdx.x < kTok * kHeads) {
    const int h = h0 + threadIdx.x / kTok, tt = blockIdx.x * kTok + threadIdx.x % kTok;
    if (h < H && tt < T) delta[(int64_t)h * T + tt] = sums[threadIdx.x / kTok][threadIdx.x % kTok];
  }
}
// O and dO must start on 16-byte boundaries and their token strides be multiples of 8 elements (as the TMA maps require).
static inline int launch_delta(const void* o, int64_t o_stride, const void* dout, int64_t do_stride, float* delta, float* acc, int T, int H, int HD,
                               cudaStream_t st) {
  if ((o_stride & 7) || (do_stride & 7) || ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(acc)) & 15))
    return -10;
  attn_delta_kernel<<<dim3((T + 15) / 16, (H + 7) / 8), 256, 0, st>>>((const __nv_bfloat16*)o, o_stride, (const __nv_bfloat16*)dout, do_stride, delta,
                                                                      acc, T, H, HD);
  return 0;
}

// ------------------------------------------------------------------------------------------- host
int make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                   const uint32_t* box);

// [T, H, HD] tensor with token stride `tok_stride` elements -> 3-D map {HD, H, T}, box {64, 1, rows}.
static inline int make_thd_map(CUtensorMap* m, const void* p, int T, int H, int HD, int64_t tok_stride, uint32_t rows = 128) {
  uint64_t dims[3] = {(uint64_t)HD, (uint64_t)H, (uint64_t)T};
  uint64_t str[2] = {(uint64_t)HD * 2, (uint64_t)tok_stride * 2};
  uint32_t box[3] = {64, 1, rows};
  return make_tmap_bf16(m, p, 3, dims, str, box);
}

template <typename K>
static inline int set_smem(K kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 0 : -2;
}


}  // namespace llmt
