// MoE routing and token movement kernels for sm_100a (reference call sites: llmtuner/models/common/moe/routing.py:31-345,
// llmtuner/models/qwen/routing.py:20-78, llmtuner/parallel/expert_parallel/token_dispatch.py:146-275,579-636):
//   router_topk      fp32 logits -> softmax / sigmoid scores -> (+bias for the selection only) -> top-k -> renormalise ->
//                    weights, indices and a per-expert histogram, one warp per token
//   router_topk_bwd  gradient of the combine weights back to the logits
//   moe_plan         destination row of every token copy in the expert-major layout, segment offsets and counts
//   permute_rows     token copies to their rows of the zero-padded expert-major layout
//   combine_rows     out[t] = sum_j w[t, j] * y[dest(t, j)] in fp32 (also the backward of permute with w = 1)
//   combine_bwd      dy rows and dw from d(out)
#include "common.cuh"
#include "kernels.h"

namespace llmt {

constexpr int kMaxEPerLane = 16;   // up to 512 experts; the router kernels are instantiated for 4, 8 and 16 experts per lane
                                   // (at 128 experts a loop over 16 spends three quarters of its instructions on nothing)
constexpr int kMaxTopK = 16;

// score_fn: 0 softmax, 1 sigmoid
template <int PER>
__global__ void __launch_bounds__(256) router_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                                                          float* __restrict__ weights, int64_t* __restrict__ indices,
                                                          float* __restrict__ counts, float* __restrict__ denom_out, int T, int E,
                                                          int k, int score_fn, int renorm, float route_scale) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  const int per = (E + 31) / 32;
  float sc[PER], sel[PER];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    sc[i] = (i < per && e < E) ? logits[(int64_t)t * E + e] : -INFINITY;
    mx = fmaxf(mx, sc[i]);
  }
  if (score_fn == 0) {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      sc[i] = (sc[i] == -INFINITY) ? 0.f : __expf(sc[i] - mx);
      sum += sc[i];
    }
    sum = warp_sum(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) sc[i] *= inv;
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) sc[i] = (sc[i] == -INFINITY) ? 0.f : 1.f / (1.f + __expf(-sc[i]));
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    sel[i] = (i < per && e < E) ? sc[i] + (bias != nullptr ? bias[e] : 0.f) : -INFINITY;
  }
  float wsel[kMaxTopK];
  int isel[kMaxTopK];
  float wsum = 0.f;
  for (int j = 0; j < k; ++j) {
    float best = -INFINITY;
    int bi = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (sel[i] > best) { best = sel[i]; bi = i; }
    int be = bi * 32 + lane;
    // warp argmax, ties to the lower expert id (matches a stable top-k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ob > best || (ob == best && oe < be)) { best = ob; be = oe; }
    }
    const int owner = be & 31, slot = be >> 5;
    float w = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i == slot && lane == owner) { w = sc[i]; sel[i] = -INFINITY; }
    w = __shfl_sync(0xffffffffu, w, owner);
    wsel[j] = w;
    isel[j] = be;
    wsum += w;
  }
  const float d = renorm ? (wsum + 1e-20f) : 1.f;
  if (lane == 0) {
    for (int j = 0; j < k; ++j) {
      weights[(int64_t)t * k + j] = wsel[j] / d * route_scale;
      indices[(int64_t)t * k + j] = isel[j];
      atomicAdd(&counts[isel[j]], 1.f);
    }
    if (denom_out != nullptr) denom_out[t] = d;
  }
}

// dlogits from dweights. softmax: s = softmax(l), w_j = scale * s_j / S (S = sum_sel s + 1e-20 when renorm, else 1).
template <int PER>
__global__ void __launch_bounds__(256) router_topk_bwd_kernel(const float* __restrict__ logits, const float* __restrict__ dweights,
                                                              const int64_t* __restrict__ indices, const float* __restrict__ denom,
                                                              float* __restrict__ dlogits, int T, int E, int k, int score_fn,
                                                              int renorm, float route_scale) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  const int per = (E + 31) / 32;
  float sc[PER], ds[PER];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    sc[i] = (i < per && e < E) ? logits[(int64_t)t * E + e] : -INFINITY;
    ds[i] = 0.f;
    mx = fmaxf(mx, sc[i]);
  }
  if (score_fn == 0) {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) { sc[i] = (sc[i] == -INFINITY) ? 0.f : __expf(sc[i] - mx); sum += sc[i]; }
    sum = warp_sum(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) sc[i] *= inv;
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) sc[i] = (sc[i] == -INFINITY) ? 0.f : 1.f / (1.f + __expf(-sc[i]));
  }
  const float S = renorm ? denom[t] : 1.f;
  // sum_j dW_j * w_j / scale, with w_j / scale = s_j / S
  float dot = 0.f;
  if (renorm) {
    for (int j = 0; j < k; ++j) {
      const int e = (int)indices[(int64_t)t * k + j];
      float sj = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i)
        if (i == (e >> 5) && lane == (e & 31)) sj = sc[i];
      sj = __shfl_sync(0xffffffffu, sj, e & 31);
      dot += dweights[(int64_t)t * k + j] * sj / S;
    }
  }
  for (int j = 0; j < k; ++j) {
    const int e = (int)indices[(int64_t)t * k + j];
    const float g = (dweights[(int64_t)t * k + j] - dot) * route_scale / S;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i == (e >> 5) && lane == (e & 31)) ds[i] = g;
  }
  if (score_fn == 0) {
    float inner = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) inner += ds[i] * sc[i];
    inner = warp_sum(inner);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = i * 32 + lane;
      if (i < per && e < E) dlogits[(int64_t)t * E + e] = sc[i] * (ds[i] - inner);
    }
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = i * 32 + lane;
      if (i < per && e < E) dlogits[(int64_t)t * E + e] = ds[i] * sc[i] * (1.f - sc[i]);
    }
  }
}

// ------------------------------------------------------------------------------------------ dispatch plan
// Stable counting sort of the token copies by expert, 1024 copies per block: (1) every block counts its experts, (2) one block
// turns the counts into the start of each (block, expert) run inside 128-row aligned segments, (3) every block ranks its
// copies (match within a warp, counts of the warps before it from shared memory). Three short launches and no host
// synchronisation; as tensor expressions (bincount, cumsum, stable argsort, scatter, gathers) the same plan took about 20
// launches, 150 us of device time at 32768 copies and a synchronisation of the host inside bincount.
constexpr int kPlanBlock = 1024;
constexpr int kPlanMaxExperts = 512;

// Expert id of copy c; an id outside [0, E) is reported once through the status word and counted as expert 0, so that no
// address is ever computed from it.
__device__ __forceinline__ int plan_expert(const int64_t* flat, int64_t c, int E, int* status) {
  const int64_t e = flat[c];
  if (e >= 0 && e < E) return (int)e;
  report_status(status, kStatusBadArgument, 3100, (int)c);
  return 0;
}

__global__ void __launch_bounds__(kPlanBlock) moe_plan_count_kernel(const int64_t* __restrict__ flat, int64_t n, int E, int* __restrict__ hist,
                                                                    int* status) {
  __shared__ int cnt[kPlanMaxExperts];
  for (int e = threadIdx.x; e < E; e += kPlanBlock) cnt[e] = 0;
  __syncthreads();
  const int64_t c = (int64_t)blockIdx.x * kPlanBlock + threadIdx.x;
  if (c < n) atomicAdd(&cnt[plan_expert(flat, c, E, status)], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kPlanBlock) hist[(int64_t)blockIdx.x * E + e] = cnt[e];
}

// One thread per expert: hist[b][e] becomes the row at which block b's copies of expert e start.
__global__ void __launch_bounds__(kPlanMaxExperts) moe_plan_scan_kernel(int* __restrict__ hist, int nblocks, int E, int align,
                                                                        int* __restrict__ seg, int64_t* __restrict__ counts) {
  __shared__ int wsum[kPlanMaxExperts / 32];
  const int e = threadIdx.x, lane = e & 31, w = e >> 5;
  int total = 0;
  if (e < E) {
#pragma unroll 8
    for (int b = 0; b < nblocks; ++b) total += hist[(int64_t)b * E + e];
  }
  const int padded = (total + align - 1) / align * align;
  int scan = padded;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, scan, o);
    if (lane >= o) scan += v;
  }
  if (lane == 31) wsum[w] = scan;
  __syncthreads();
  int base = scan - padded;
  for (int i = 0; i < w; ++i) base += wsum[i];
  if (e < E) {
    seg[e] = base;
    if (e == E - 1) seg[E] = base + padded;
    counts[e] = total;
    int at = base;
#pragma unroll 8
    for (int b = 0; b < nblocks; ++b) {
      const int h = hist[(int64_t)b * E + e];
      hist[(int64_t)b * E + e] = at;
      at += h;
    }
  }
}

__global__ void __launch_bounds__(kPlanBlock) moe_plan_place_kernel(const int64_t* __restrict__ flat, int64_t n, int E, const int* __restrict__ start,
                                                                    int64_t* __restrict__ dest) {
  constexpr int kWarps = kPlanBlock / 32;
  __shared__ uint16_t cnt[kWarps][kPlanMaxExperts];       // copies of expert e in warp w, then in the warps before it
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kWarps * kPlanMaxExperts; i += kPlanBlock) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t c = (int64_t)blockIdx.x * kPlanBlock + threadIdx.x;
  const bool live = c < n;
  int e = -1, rank = 0;
  if (live) {
    const int64_t id = flat[c];
    e = (id >= 0 && id < E) ? (int)id : 0;
  }
  const uint32_t same = __match_any_sync(0xffffffffu, e);
  rank = __popc(same & ((1u << lane) - 1u));
  if (live && rank == 0) cnt[w][e] = (uint16_t)__popc(same);
  __syncthreads();
  for (int x = threadIdx.x; x < E; x += kPlanBlock) {
    int run = 0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const int v = cnt[i][x];
      cnt[i][x] = (uint16_t)run;
      run += v;
    }
  }
  __syncthreads();
  if (live) dest[c] = (int64_t)start[(int64_t)blockIdx.x * E + e] + cnt[w][e] + rank;
}

// Rows of expert e between its last copy and the end of its segment are zeroed by kPadBlocks blocks each (the grouped weight
// gradient reduces over them); rows past the last segment are never read.
constexpr int kPadBlocks = 4;
__device__ __forceinline__ void zero_padding(__nv_bfloat16* rows, const int* seg, const int64_t* counts, int b, int D) {
  const int e = b / kPadBlocks;
  const int64_t lo = seg[e] + counts[e], hi = seg[e + 1];
  uint4* d = reinterpret_cast<uint4*>(rows + lo * D);
  const int64_t nv = (hi - lo) * (D / 8);
  for (int64_t i = (int64_t)(b % kPadBlocks) * blockDim.x + threadIdx.x; i < nv; i += kPadBlocks * blockDim.x) d[i] = make_uint4(0, 0, 0, 0);
}

// rows[dest[c]] = x[c / k] ; one warp per copy, 16-byte accesses (D % 8 == 0). With `seg` the last blocks of the grid zero the
// padding rows, so the caller need not clear the buffer first.
__global__ void __launch_bounds__(256) permute_rows_kernel(const __nv_bfloat16* __restrict__ x, const int64_t* __restrict__ dest,
                                                           __nv_bfloat16* __restrict__ rows, int64_t ncopies, int k, int D, int copy_blocks,
                                                           const int* __restrict__ seg, const int64_t* __restrict__ counts) {
  if ((int)blockIdx.x >= copy_blocks) {
    zero_padding(rows, seg, counts, blockIdx.x - copy_blocks, D);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t c = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= ncopies) return;
  const uint4* s = reinterpret_cast<const uint4*>(x + (c / k) * D);
  uint4* d = reinterpret_cast<uint4*>(rows + dest[c] * D);
#pragma unroll 4
  for (int i = lane; i < D / 8; i += 32) d[i] = s[i];
}

// out[t] = sum_j w[t, j] * y[dest[t * k + j]] (w == nullptr: plain sum), fp32 accumulate in the order of j. A warp owns 32
// vectors of one token (not a whole row: few tokens still fill the chip) and has the loads of eight copies in flight.
__global__ void __launch_bounds__(256) combine_rows_kernel(const __nv_bfloat16* __restrict__ y, const int64_t* __restrict__ dest,
                                                           const float* __restrict__ w, __nv_bfloat16* __restrict__ out, int T,
                                                           int k, int D, int slices) {
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t t = item / slices;
  const int i = (int)(item % slices) * 32 + lane;
  if (t >= T || i >= D / 8) return;
  float acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.f;
  for (int j0 = 0; j0 < k; j0 += 8) {
    uint4 v[8];
    float wj[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t c = t * k + min(j0 + j, k - 1);
      v[j] = reinterpret_cast<const uint4*>(y + dest[c] * D)[i];
      wj[j] = (w != nullptr) ? w[c] : 1.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j0 + j < k) {
        const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v[j]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = __bfloat1622float2(b[q]);
          acc[2 * q] += wj[j] * f.x;
          acc[2 * q + 1] += wj[j] * f.y;
        }
      }
    }
  }
  uint4 o;
  o.x = pack_bf16x2(acc[0], acc[1]); o.y = pack_bf16x2(acc[2], acc[3]);
  o.z = pack_bf16x2(acc[4], acc[5]); o.w = pack_bf16x2(acc[6], acc[7]);
  reinterpret_cast<uint4*>(out + t * D)[i] = o;
}

// dy[dest[c]] = w[c] * dout[c / k] ; dw[c] = <dout[c / k], y[dest[c]]> ; one warp per copy
__global__ void __launch_bounds__(256) combine_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ y,
                                                          const int64_t* __restrict__ dest, const float* __restrict__ w,
                                                          __nv_bfloat16* __restrict__ dy, float* __restrict__ dw, int64_t ncopies,
                                                          int k, int D, int copy_blocks, const int* __restrict__ seg,
                                                          const int64_t* __restrict__ counts) {
  if ((int)blockIdx.x >= copy_blocks) {
    zero_padding(dy, seg, counts, blockIdx.x - copy_blocks, D);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t c = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= ncopies) return;
  const uint4* g = reinterpret_cast<const uint4*>(dout + (c / k) * D);
  const uint4* yy = reinterpret_cast<const uint4*>(y + dest[c] * D);
  uint4* d = reinterpret_cast<uint4*>(dy + dest[c] * D);
  const float wc = w[c];
  float dot = 0.f;
#pragma unroll 4
  for (int i = lane; i < D / 8; i += 32) {
    const uint4 gv = g[i], yv = yy[i];
    const __nv_bfloat162 *gb = reinterpret_cast<const __nv_bfloat162*>(&gv), *yb = reinterpret_cast<const __nv_bfloat162*>(&yv);
    float o[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 gf = __bfloat1622float2(gb[q]), yf = __bfloat1622float2(yb[q]);
      dot += gf.x * yf.x + gf.y * yf.y;
      o[2 * q] = wc * gf.x;
      o[2 * q + 1] = wc * gf.y;
    }
    uint4 ov;
    ov.x = pack_bf16x2(o[0], o[1]); ov.y = pack_bf16x2(o[2], o[3]); ov.z = pack_bf16x2(o[4], o[5]); ov.w = pack_bf16x2(o[6], o[7]);
    d[i] = ov;
  }
  dot = warp_sum(dot);
  if (lane == 0 && dw != nullptr) dw[c] = dot;
}

}  // namespace llmt

using namespace llmt;
#define LLMT_CHECK_LAUNCH() return (cudaGetLastError() == cudaSuccess) ? 0 : -3

extern "C" int llmt_router_topk(const float* logits, const float* bias, float* weights, int64_t* indices, float* counts,
                                float* denom, int T, int E, int k, int score_fn, int renorm, float route_scale, cudaStream_t st) {
  if (T <= 0) return 0;
  if (E > 32 * kMaxEPerLane || k > kMaxTopK || k > E) return -10;
  auto go = [&](auto kern) { kern<<<(T + 7) / 8, 256, 0, st>>>(logits, bias, weights, indices, counts, denom, T, E, k, score_fn, renorm, route_scale); };
  if (E <= 128) go(router_topk_kernel<4>);
  else if (E <= 256) go(router_topk_kernel<8>);
  else go(router_topk_kernel<kMaxEPerLane>);
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_router_topk_bwd(const float* logits, const float* dweights, const int64_t* indices, const float* denom,
                                    float* dlogits, int T, int E, int k, int score_fn, int renorm, float route_scale, cudaStream_t st) {
  if (T <= 0) return 0;
  if (E > 32 * kMaxEPerLane || k > kMaxTopK) return -10;
  auto go = [&](auto kern) { kern<<<(T + 7) / 8, 256, 0, st>>>(logits, dweights, indices, denom, dlogits, T, E, k, score_fn, renorm, route_scale); };
  if (E <= 128) go(router_topk_bwd_kernel<4>);
  else if (E <= 256) go(router_topk_bwd_kernel<8>);
  else go(router_topk_bwd_kernel<kMaxEPerLane>);
  LLMT_CHECK_LAUNCH();
}
// hist: scratch of llmt_moe_plan_scratch_ints(n, E) ints. seg [E + 1], counts [E], dest [n].
extern "C" int64_t llmt_moe_plan_scratch_ints(int64_t n, int E) { return (n + kPlanBlock - 1) / kPlanBlock * E; }
extern "C" int llmt_moe_plan(const int64_t* flat, int64_t n, int E, int align, int* hist, int64_t* dest, int* seg, int64_t* counts,
                             int* status, cudaStream_t st) {
  if (E < 1 || E > kPlanMaxExperts || align < 1 || n < 0 || n + (int64_t)E * align >= (1ll << 31)) return -10;
  const int nb = (int)((n + kPlanBlock - 1) / kPlanBlock);
  if (nb > 0) moe_plan_count_kernel<<<nb, kPlanBlock, 0, st>>>(flat, n, E, hist, status);
  moe_plan_scan_kernel<<<1, kPlanMaxExperts, 0, st>>>(hist, nb, E, align, seg, counts);
  if (nb > 0) moe_plan_place_kernel<<<nb, kPlanBlock, 0, st>>>(flat, n, E, hist, dest);
  LLMT_CHECK_LAUNCH();
}
// Is one of the addresses off a 16-byte boundary? The launchers refuse those (-10): the kernels load and store 16 bytes at a time.
static inline bool off16(const void* a, const void* b, const void* c = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) != 0;
}
// With `seg` [E + 1] and `counts` [E] the padding rows of every segment are zeroed too.
extern "C" int llmt_permute_rows(const void* x, const int64_t* dest, void* rows, int64_t ncopies, int k, int D, const int* seg,
                                 const int64_t* counts, int E, cudaStream_t st) {
  if (ncopies <= 0) return 0;
  if (D % 8 || off16(x, rows)) return -10;
  const int nb = (int)((ncopies + 7) / 8);
  permute_rows_kernel<<<nb + (seg ? E * kPadBlocks : 0), 256, 0, st>>>((const __nv_bfloat16*)x, dest, (__nv_bfloat16*)rows, ncopies, k, D, nb, seg,
                                                                      counts);
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_combine_rows(const void* y, const int64_t* dest, const float* w, void* out, int T, int k, int D, cudaStream_t st) {
  if (T <= 0) return 0;
  if (D % 8 || k < 1 || off16(y, out)) return -10;
  const int slices = (D / 8 + 31) / 32;
  combine_rows_kernel<<<(unsigned)(((int64_t)T * slices + 7) / 8), 256, 0, st>>>((const __nv_bfloat16*)y, dest, w, (__nv_bfloat16*)out, T, k, D, slices);
  LLMT_CHECK_LAUNCH();
}
extern "C" int llmt_combine_bwd(const void* dout, const void* y, const int64_t* dest, const float* w, void* dy, float* dw,
                                int64_t ncopies, int k, int D, const int* seg, const int64_t* counts, int E, cudaStream_t st) {
  if (ncopies <= 0) return 0;
  if (D % 8 || off16(dout, y, dy)) return -10;
  const int nb = (int)((ncopies + 7) / 8);
  combine_bwd_kernel<<<nb + (seg ? E * kPadBlocks : 0), 256, 0, st>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)y, dest, w,
                                                                     (__nv_bfloat16*)dy, dw, ncopies, k, D, nb, seg, counts);
  LLMT_CHECK_LAUNCH();
}
