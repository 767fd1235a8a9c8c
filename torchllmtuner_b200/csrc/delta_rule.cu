// Gated delta rule (one decay per head) in chunk-parallel form, forward and backward, fp32 throughout
// (reference call sites: llmtuner/models/qwen/qwen3_5_moe/gated_delta.py:13-189). The algebra is that of
// models/families.py::chunked_delta_rule; with G the running sum of the log decays inside a 64-token chunk that starts from S:
//   A[t,i] = beta_t <k_t, k_i> e^(G_t - G_i)  (i < t)      P[t,i] = <q_t, k_i> e^(G_t - G_i)  (i <= t)
//   [W1 | W2] = (I + A)^-1 [beta v | beta e^G k]            U = W1 - W2 S
//   O = e^G (q S) + P U                                     S' = e^(G_C) S + sum_t e^(G_C - G_t) k_t u_t^T
// Four kernels: per (chunk, head) everything that does not depend on S; the walk over the chunks per (head, 32 value columns:
// the columns of S evolve independently); the same walk backwards for dU and the state gradients; and per (chunk, head) every
// input gradient from S, dS', U, dU. Rows past the end of the document have beta = k = q = v = 0 and decay 1.
//
// fp32 products on the FMA pipe: results must not lose precision against the fp32 tensor expressions they replace, which rules
// out 16-bit and TF32 operands. Bound by FMA issue: operands sit in shared memory, a thread holds 8 x 4 (or 8 x 2, 8 x 1, 16 x 1)
// results in registers, rows of the left operand are read as broadcasts. As tensor expressions (batched products, a triangular
// solve, a two-level scan over state maps, some 600 launches) forward + backward took 5.5 ms at 2048 tokens x 32 heads x 128;
// these kernels take 1.7 ms, and their error against 64 bits is 1.2e-7 instead of 3.3e-7 (outputs; gradients 0.4 to 1.0 of it).
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace llmt {

constexpr int kDC = 64;          // tokens per chunk
constexpr int kDThreads = 256;   // 8 warps: warp r owns rows 8r .. 8r + 7 of a 64-row result
constexpr int kDV = 32;          // value columns of a scan block
constexpr int kLP = kDC + 4;     // row pitch of 64-column tiles (floats)
constexpr int kLS = kDV + 4;     // row pitch of 32-column tiles

template <int R, int C>
__device__ __forceinline__ void zero(float (&acc)[R][C]) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[i][c] = 0.f;
}
// acc[i][c] += sum_k A[row0 + i][k] * B[k][lane + 32 c]            (A, B row-major in shared memory, K a multiple of 4)
template <int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_nn(float (&acc)[R][C], const float* A, const float* B, int row0, int lane) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float4 a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const float4*>(A + (row0 + i) * LDA + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float b[C];
#pragma unroll
      for (int c = 0; c < C; ++c) b[c] = B[(k + kk) * LDB + lane + 32 * c];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float av = kk == 0 ? a[i].x : kk == 1 ? a[i].y : kk == 2 ? a[i].z : a[i].w;
#pragma unroll
        for (int c = 0; c < C; ++c) acc[i][c] = fmaf(av, b[c], acc[i][c]);
      }
    }
  }
}
// acc[i][c] += sum_k A[row0 + i][k] * B[lane + 32 c][k]
template <int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_nt(float (&acc)[R][C], const float* A, const float* B, int row0, int lane) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float4 b[C];
#pragma unroll
    for (int c = 0; c < C; ++c) b[c] = *reinterpret_cast<const float4*>(B + (lane + 32 * c) * LDB + k);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(A + (row0 + i) * LDA + k);
#pragma unroll
      for (int c = 0; c < C; ++c)
        acc[i][c] = fmaf(a.w, b[c].w, fmaf(a.z, b[c].z, fmaf(a.y, b[c].y, fmaf(a.x, b[c].x, acc[i][c]))));
    }
  }
}
// acc[i][c] += sum_k A[k][row0 + i] * B[k][lane + 32 c]            (R a multiple of 4)
template <int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_tn(float (&acc)[R][C], const float* A, const float* B, int row0, int lane) {
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    float a[R], b[C];
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 v = *reinterpret_cast<const float4*>(A + k * LDA + row0 + i);
      a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) b[c] = B[k * LDB + lane + 32 * c];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[i][c] = fmaf(a[i], b[c], acc[i][c]);
  }
}
// The same products with the contraction summed in blocks of 16: a chain of 64 or 128 roundings at the size of the result
// becomes 4 to 8 of them.
constexpr int kBlk = 16;
template <int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_nn_b(float (&acc)[R][C], const float* A, const float* B, int row0, int lane) {
#pragma unroll 1
  for (int k = 0; k < K; k += kBlk) {
    float t[R][C];
    zero(t);
    mm_nn<R, C, kBlk, LDA, LDB>(t, A + k, B + k * LDB, row0, lane);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[i][c] += t[i][c];
  }
}
template <int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_nt_b(float (&acc)[R][C], const float* A, const float* B, int row0, int lane) {
#pragma unroll 1
  for (int k = 0; k < K; k += kBlk) {
    float t[R][C];
    zero(t);
    mm_nt<R, C, kBlk, LDA, LDB>(t, A + k, B + k, row0, lane);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[i][c] += t[i][c];
  }
}
template <int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_tn_b(float (&acc)[R][C], const float* A, const float* B, int row0, int lane) {
#pragma unroll 1
  for (int k = 0; k < K; k += kBlk) {
    float t[R][C];
    zero(t);
    mm_tn<R, C, kBlk, LDA, LDB>(t, A + k * LDA, B + k * LDB, row0, lane);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[i][c] += t[i][c];
  }
}
template <int R, int C, int LD>
__device__ __forceinline__ void put(float* dst, const float (&acc)[R][C], int row0, int lane) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) dst[(row0 + i) * LD + lane + 32 * c] = acc[i][c];
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// ROWS x COLS floats into shared memory with row pitch LD; rows at or beyond `live` are zero-filled (their address is not read).
template <int ROWS, int COLS, int LD>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int64_t ld, int live) {
  constexpr int V = COLS / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < ROWS * V; i += kDThreads) {
    const int r = i / V, c = (i % V) * 4;
    cp16(dst + r * LD + c, src + (int64_t)(r < live ? r : 0) * ld + c, r < live);
  }
}

// e^d for a difference of running log decays. The sums are kept in 64 bits: their size grows with the chunk (tens), and a
// rounding there would be a relative error of 1e-6 in every decay factor. 64 additions per chunk cost nothing.
__device__ __forceinline__ float exp_d(double d) {
  const float hi = (float)d, lo = (float)(d - (double)hi), e = expf(hi);
  return fmaf(e, lo, e);
}

struct DeltaArgs {
  const float *q, *k, *v, *beta, *g;         // [T, H, D] and [T, H]
  double *G;                                 // [N, H, 64] running log decay
  float *W1, *W2, *P, *inv;                  // [N, H, 64, D], [N, H, 64, 64]
  float *S, *U, *o;                          // [N, H, D, D] state at chunk starts, [T, H, D]
  const float* dout;
  float *dS, *dU;                            // [N, H, D, D] gradient of the state after the chunk, [T, H, D]
  float *dq, *dk, *dv, *dbeta, *dg;
  int T, H;
};

// ------------------------------------------------------------------------------------------ per chunk: A, P, inverse, W
template <int D>
struct PrepSmem {
  static constexpr int kL = D + 4, kTile = kDC * kL, kSq = kDC * kLP;
  static constexpr int kFloats = 3 * kTile + 3 * kSq + 3 * kDC;   // 2 * 64 of them for the 64-bit sums
};
template <int D>
__global__ void __launch_bounds__(kDThreads, 1) delta_prep_kernel(const DeltaArgs a) {
  constexpr int L = D + 4, C = D / 32;
  extern __shared__ __align__(16) float sm[];
  float *sK = sm, *sQ = sK + kDC * L, *sV = sQ + kDC * L, *sA = sV + kDC * L, *sI = sA + kDC * kLP, *sT = sI + kDC * kLP;
  double* sG = reinterpret_cast<double*>(sT + kDC * kLP);
  float* sB = reinterpret_cast<float*>(sG + kDC);
  const int n = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = warp * 8;
  const int t0 = n * kDC, live = min(kDC, a.T - t0);
  const int64_t at = ((int64_t)t0 * a.H + h) * D, ld = (int64_t)a.H * D, nh = (int64_t)n * a.H + h;
  load_tile<kDC, D, L>(sK, a.k + at, ld, live);
  load_tile<kDC, D, L>(sQ, a.q + at, ld, live);
  load_tile<kDC, D, L>(sV, a.v + at, ld, live);
  cp_commit();
  if (warp == 0) {                                         // running sum of the log decays, two tokens per lane
    const int t = 2 * lane;
    const double g0 = t < live ? a.g[(int64_t)(t0 + t) * a.H + h] : 0.0, g1 = t + 1 < live ? a.g[(int64_t)(t0 + t + 1) * a.H + h] : 0.0;
    double s = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    sG[t + 1] = s;
    sG[t] = s - g1;
  }
  if (threadIdx.x < kDC) sB[threadIdx.x] = (int)threadIdx.x < live ? a.beta[(int64_t)(t0 + threadIdx.x) * a.H + h] : 0.f;
  cp_wait<0>();
  __syncthreads();
  if (threadIdx.x < kDC) a.G[nh * kDC + threadIdx.x] = sG[threadIdx.x];
  {
    float kk[8][2], qk[8][2];
    zero(kk); zero(qk);
    mm_nt_b<8, 2, D, L, L>(kk, sK, sK, row0, lane);
    mm_nt_b<8, 2, D, L, L>(qk, sQ, sK, row0, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int t = row0 + i, s = lane + 32 * c;
        const float m = s <= t ? exp_d(fmin(sG[t] - sG[s], 0.0)) : 0.f;
        sA[t * kLP + s] = s < t ? sB[t] * kk[i][c] * m : 0.f;
        a.P[(nh * kDC + t) * kDC + s] = qk[i][c] * m;
      }
  }
  for (int i = threadIdx.x; i < kDC * kLP; i += kDThreads) sI[i] = 0.f;
  __syncthreads();
  // (I + A)^-1 by 16 x 16 blocks: the diagonal blocks by forward substitution, one column per thread ...
  if (threadIdx.x < kDC) {
    const int b = threadIdx.x / 16 * 16, j = threadIdx.x % 16;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      float s = r == j ? 1.f : 0.f;
#pragma unroll
      for (int i = 0; i < r; ++i) s -= sA[(b + r) * kLP + b + i] * x[i];
      x[r] = s;
      sI[(b + r) * kLP + b + j] = s;
    }
  }
  __syncthreads();
  // ... then the blocks d below the diagonal: X_ij = -X_ii (sum_{j <= k < i} A_ik X_kj)
  const int er = threadIdx.x / 16, ec = threadIdx.x % 16;
  for (int d = 1; d < 4; ++d) {
    for (int bi = d; bi < 4; ++bi) {
      const int bj = bi - d;
      float s = 0.f;
      for (int kcol = bj * 16; kcol < bi * 16; ++kcol) s += sA[(bi * 16 + er) * kLP + kcol] * sI[kcol * kLP + bj * 16 + ec];
      sT[(bi * 16 + er) * kLP + ec] = s;
    }
    __syncthreads();
    for (int bi = d; bi < 4; ++bi) {
      float s = 0.f;
#pragma unroll
      for (int r = 0; r < 16; ++r) s -= sI[(bi * 16 + er) * kLP + bi * 16 + r] * sT[(bi * 16 + r) * kLP + ec];
      sI[(bi * 16 + er) * kLP + (bi - d) * 16 + ec] = s;
    }
    __syncthreads();
  }
  // right-hand sides: beta v in place, beta e^G k over q
  for (int i = threadIdx.x; i < kDC * D; i += kDThreads) {
    const int r = i / D, c = i % D;
    sV[r * L + c] *= sB[r];
    sQ[r * L + c] = sB[r] * exp_d(sG[r]) * sK[r * L + c];
  }
  if (a.inv != nullptr)
    for (int i = threadIdx.x; i < kDC * kDC; i += kDThreads) a.inv[nh * kDC * kDC + i] = sI[i / kDC * kLP + i % kDC];
  __syncthreads();
  float w[8][C];
  zero(w);
  mm_nn_b<8, C, kDC, kLP, L>(w, sI, sV, row0, lane);
  put<8, C, D>(a.W1 + nh * kDC * D, w, row0, lane);
  zero(w);
  mm_nn_b<8, C, kDC, kLP, L>(w, sI, sQ, row0, lane);
  put<8, C, D>(a.W2 + nh * kDC * D, w, row0, lane);
}

// ------------------------------------------------------------------------------------------ walk over the chunks
// One block per (head, 32 value columns). Tiles are single-buffered: a tile's successor is fetched as soon as its last product
// has read it, so every fetch runs under the products of the other tiles.
template <int D>
struct ScanSmem {
  static constexpr int kL = D + 4;
  static constexpr int kFloats = 3 * kDC * kL + kDC * kLP + D * kLS + 3 * kDC * kLS + 2 * kDC;
};
template <int D>
__global__ void __launch_bounds__(kDThreads, 1) delta_scan_fwd_kernel(const DeltaArgs a) {
  constexpr int L = D + 4, SR = D / 8;
  extern __shared__ __align__(16) float sm[];
  float *sW = sm, *sQ = sW + kDC * L, *sK = sQ + kDC * L, *sP = sK + kDC * L, *sS = sP + kDC * kLP;
  float *sW1 = sS + D * kLS, *sU = sW1 + kDC * kLS, *sE = sU + kDC * kLS;
  double* sG = reinterpret_cast<double*>(sE + kDC * kLS);
  const int h = blockIdx.x, c0 = blockIdx.y * kDV, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = warp * 8;
  const int N = (a.T + kDC - 1) / kDC;
  const int64_t ld = (int64_t)a.H * D;
  auto fetch_w = [&](int n) {
    const int64_t nh = (int64_t)n * a.H + h;
    load_tile<kDC, D, L>(sW, a.W2 + nh * kDC * D, D, kDC);
    load_tile<kDC, kDV, kLS>(sW1, a.W1 + nh * kDC * D + c0, D, kDC);
    cp_commit();
  };
  auto fetch_q = [&](int n) {
    load_tile<kDC, D, L>(sQ, a.q + ((int64_t)n * kDC * a.H + h) * D, ld, min(kDC, a.T - n * kDC));
    load_tile<kDC, kDC, kLP>(sP, a.P + ((int64_t)n * a.H + h) * kDC * kDC, kDC, kDC);
    cp_commit();
  };
  auto fetch_k = [&](int n) {
    load_tile<kDC, D, L>(sK, a.k + ((int64_t)n * kDC * a.H + h) * D, ld, min(kDC, a.T - n * kDC));
    cp_commit();
  };
  for (int i = threadIdx.x; i < D * kLS; i += kDThreads) sS[i] = 0.f;
  fetch_w(0); fetch_q(0); fetch_k(0);
  for (int n = 0; n < N; ++n) {
    const int64_t nh = (int64_t)n * a.H + h;
    const int t0 = n * kDC, live = min(kDC, a.T - t0);
    if (threadIdx.x < kDC) sG[threadIdx.x] = a.G[nh * kDC + threadIdx.x];
    cp_wait<2>();                                          // W tiles (groups complete in order: w, q, k)
    __syncthreads();
    if (a.S != nullptr)
      for (int i = threadIdx.x; i < D * kDV; i += kDThreads) a.S[(nh * D + i / kDV) * D + c0 + i % kDV] = sS[i / kDV * kLS + i % kDV];
    float u[8][1];
    zero(u);
    mm_nn_b<8, 1, D, L, kLS>(u, sW, sS, row0, lane);
    const double gc = sG[kDC - 1];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = row0 + i;
      const float x = sW1[t * kLS + lane] - u[i][0];
      sU[t * kLS + lane] = x;
      sE[t * kLS + lane] = exp_d(gc - sG[t]) * x;
      if (t < live && a.U != nullptr) a.U[((int64_t)(t0 + t) * a.H + h) * D + c0 + lane] = x;
    }
    cp_wait<1>();
    __syncthreads();                                       // U complete, W tiles free, Q and P here
    if (n + 1 < N) fetch_w(n + 1); else cp_commit();
    float o[8][1], p[8][1];
    zero(o); zero(p);
    mm_nn_b<8, 1, D, L, kLS>(o, sQ, sS, row0, lane);
    mm_nn_b<8, 1, kDC, kLP, kLS>(p, sP, sU, row0, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = row0 + i;
      if (t < live) a.o[((int64_t)(t0 + t) * a.H + h) * D + c0 + lane] = exp_d(sG[t]) * o[i][0] + p[i][0];
    }
    cp_wait<1>();                                          // K (the newest group is W of the next chunk)
    __syncthreads();                                       // everyone is done with S, Q and P
    if (n + 1 < N) fetch_q(n + 1); else cp_commit();
    float s[SR][1];
    const float ec = exp_d(gc);
    zero(s);                                               // the chunk's sum first: one rounding at the size of the state
    mm_tn_b<SR, 1, kDC, L, kLS>(s, sK, sE, warp * SR, lane);
#pragma unroll
    for (int i = 0; i < SR; ++i) {
      float* p = sS + (warp * SR + i) * kLS + lane;
      *p = fmaf(ec, *p, s[i][0]);
    }
    __syncthreads();                                       // K is free
    if (n + 1 < N) fetch_k(n + 1); else cp_commit();
  }
  cp_wait<0>();
}

// Backwards: dU = P^T dO + e^(G_C - G) (k dS'),  dS = e^(G_C) dS' + q^T (e^G dO) - W2^T dU.
template <int D>
__global__ void __launch_bounds__(kDThreads, 1) delta_scan_bwd_kernel(const DeltaArgs a) {
  constexpr int L = D + 4, SR = D / 8;
  extern __shared__ __align__(16) float sm[];
  float *sW = sm, *sQ = sW + kDC * L, *sK = sQ + kDC * L, *sP = sK + kDC * L, *sS = sP + kDC * kLP;
  float *sO = sS + D * kLS, *sU = sO + kDC * kLS, *sE = sU + kDC * kLS;
  double* sG = reinterpret_cast<double*>(sE + kDC * kLS);
  const int h = blockIdx.x, c0 = blockIdx.y * kDV, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = warp * 8;
  const int N = (a.T + kDC - 1) / kDC;
  const int64_t ld = (int64_t)a.H * D;
  auto fetch_k = [&](int n) {                              // first group of a step: K, P, dO
    const int live = min(kDC, a.T - n * kDC);
    const int64_t at = ((int64_t)n * kDC * a.H + h) * D;
    load_tile<kDC, D, L>(sK, a.k + at, ld, live);
    load_tile<kDC, kDC, kLP>(sP, a.P + ((int64_t)n * a.H + h) * kDC * kDC, kDC, kDC);
    load_tile<kDC, kDV, kLS>(sO, a.dout + at + c0, ld, live);
    cp_commit();
  };
  auto fetch_qw = [&](int n) {                             // second group: Q, W2
    load_tile<kDC, D, L>(sQ, a.q + ((int64_t)n * kDC * a.H + h) * D, ld, min(kDC, a.T - n * kDC));
    load_tile<kDC, D, L>(sW, a.W2 + ((int64_t)n * a.H + h) * kDC * D, D, kDC);
    cp_commit();
  };
  for (int i = threadIdx.x; i < D * kLS; i += kDThreads) sS[i] = 0.f;
  fetch_k(N - 1); fetch_qw(N - 1);
  for (int n = N - 1; n >= 0; --n) {
    const int64_t nh = (int64_t)n * a.H + h;
    const int t0 = n * kDC, live = min(kDC, a.T - t0);
    if (threadIdx.x < kDC) sG[threadIdx.x] = a.G[nh * kDC + threadIdx.x];
    cp_wait<1>();
    __syncthreads();
    for (int i = threadIdx.x; i < D * kDV; i += kDThreads) a.dS[(nh * D + i / kDV) * D + c0 + i % kDV] = sS[i / kDV * kLS + i % kDV];
    float x[8][1], y[8][1];
    zero(x); zero(y);
    mm_tn_b<8, 1, kDC, kLP, kLS>(x, sP, sO, row0, lane);
    mm_nn_b<8, 1, D, L, kLS>(y, sK, sS, row0, lane);
    const double gc = sG[kDC - 1];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = row0 + i;
      const float d = x[i][0] + exp_d(gc - sG[t]) * y[i][0];
      sU[t * kLS + lane] = -d;
      sE[t * kLS + lane] = exp_d(sG[t]) * sO[t * kLS + lane];
      if (t < live) a.dU[((int64_t)(t0 + t) * a.H + h) * D + c0 + lane] = d;
    }
    cp_wait<0>();
    __syncthreads();                                       // dU complete; K, P and dO free; Q and W here
    if (n > 0) fetch_k(n - 1); else cp_commit();
    float s[SR][1];
    const float ec = exp_d(gc);
    zero(s);
    mm_tn_b<SR, 1, kDC, L, kLS>(s, sQ, sE, warp * SR, lane);
    float w[SR][1];
    zero(w);
    mm_tn_b<SR, 1, kDC, L, kLS>(w, sW, sU, warp * SR, lane);
#pragma unroll
    for (int i = 0; i < SR; ++i) {
      float* p = sS + (warp * SR + i) * kLS + lane;
      *p = fmaf(ec, *p, s[i][0] + w[i][0]);
    }
    __syncthreads();                                       // Q, W free
    if (n > 0) fetch_qw(n - 1); else cp_commit();
  }
  cp_wait<0>();
}

// ------------------------------------------------------------------------------------------ per chunk: input gradients
template <int D>
struct GradSmem {
  static constexpr int kL = D + 4;
  static constexpr int kBig = (D * kL > kDC * kL + kDC * kLP) ? D * kL : kDC * kL + kDC * kLP;   // a state, or dW2 and the inverse
  static constexpr int kFloats = 4 * kDC * kL + kBig + kDC * kLP + 5 * kDC + 8 * kDC + 32;
};
template <int D>
__global__ void __launch_bounds__(kDThreads, 1) delta_grad_kernel(const DeltaArgs a) {
  constexpr int L = D + 4, C = D / 32;
  extern __shared__ __align__(16) float sm[];
  float *sK = sm, *sQ = sK + kDC * L, *sX = sQ + kDC * L, *sY = sX + kDC * L, *sS = sY + kDC * L, *sP = sS + GradSmem<D>::kBig;
  double* sG = reinterpret_cast<double*>(sP + kDC * kLP);
  float *sB = reinterpret_cast<float*>(sG + kDC), *rG = sB + kDC, *rB = rG + kDC, *cG = rB + kDC, *red = cG + 8 * kDC;   // cG [8 warps][64]
  const int n = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = warp * 8;
  const int t0 = n * kDC, live = min(kDC, a.T - t0);
  const int64_t at = ((int64_t)t0 * a.H + h) * D, ld = (int64_t)a.H * D, nh = (int64_t)n * a.H + h;
  const float* S = a.S + nh * D * D;
  const float* dS = a.dS + nh * D * D;
  load_tile<kDC, D, L>(sK, a.k + at, ld, live);
  load_tile<kDC, D, L>(sQ, a.q + at, ld, live);
  load_tile<kDC, D, L>(sX, a.dout + at, ld, live);         // dO
  load_tile<kDC, D, L>(sY, a.dU + at, ld, live);           // dU = dW1
  load_tile<D, D, L>(sS, S, D, D);
  cp_commit();
  if (threadIdx.x < kDC) {
    sG[threadIdx.x] = a.G[nh * kDC + threadIdx.x];
    sB[threadIdx.x] = (int)threadIdx.x < live ? a.beta[(int64_t)(t0 + threadIdx.x) * a.H + h] : 0.f;
  }
  cp_wait<0>();
  __syncthreads();
  float eg[8], ee[8], bt[8], dGt[8], dBt[8];               // this warp's rows: e^G, e^(G_C - G), beta, row sums of dG and dbeta
  const double gc = sG[kDC - 1];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double g = sG[row0 + i];
    eg[i] = exp_d(g); ee[i] = exp_d(gc - g); bt[i] = sB[row0 + i];
    dGt[i] = 0.f; dBt[i] = 0.f;
  }
  float dq[8][C], dk[8][C], w[8][C];
  float dGc = 0.f;                                         // gradient of G at the end of the chunk (this thread's share)
  float col[2] = {0.f, 0.f};                               // column sums of dG over this warp's rows, columns lane and lane + 32
  // ---- products with the state: dq = e^G (dO S^T), dW2 = -dU S^T
  zero(dq);
  mm_nt<8, C, D, L, L>(dq, sX, sS, row0, lane);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      dq[i][c] *= eg[i];
      dGt[i] += dq[i][c] * sQ[(row0 + i) * L + lane + 32 * c];
    }
  zero(w);
  mm_nt<8, C, D, L, L>(w, sY, sS, row0, lane);             // -dW2, kept in registers until the state buffer is free
  __syncthreads();
  // ---- the state gradient takes the state's place; its product with the state is the gradient of the chunk's decay
  {
    constexpr int V = D / 4;
    float s = 0.f;
    for (int i = threadIdx.x; i < D * V; i += kDThreads) {
      const int r = i / V, c = (i % V) * 4;
      const float4 d = *reinterpret_cast<const float4*>(dS + (int64_t)r * D + c);
      float4* p = reinterpret_cast<float4*>(sS + r * L + c);
      const float4 x = *p;
      s += d.x * x.x + d.y * x.y + d.z * x.z + d.w * x.w;
      *p = d;
    }
    dGc += s * exp_d(gc);
  }
  load_tile<kDC, D, L>(sY, a.U + at, ld, live);            // U over dU
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  zero(dk);
  mm_nt<8, C, D, L, L>(dk, sY, sS, row0, lane);            // dKend = U dS'^T
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      dk[i][c] *= ee[i];
      const float x = dk[i][c] * sK[(row0 + i) * L + lane + 32 * c];
      dGt[i] -= x;
      dGc += x;
    }
  {                                                        // dP = tril(dO U^T); its decay factors go to dG
    float p[8][2];
    zero(p);
    mm_nt<8, 2, D, L, L>(p, sX, sY, row0, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int t = row0 + i, s = lane + 32 * c;
        const float m = s <= t ? exp_d(fmin(sG[t] - sG[s], 0.0)) : 0.f;
        const float x = s <= t ? p[i][c] * a.P[(nh * kDC + t) * kDC + s] : 0.f;
        dGt[i] += x;
        col[c] -= x;
        sP[t * kLP + s] = p[i][c] * m;
      }
  }
  __syncthreads();
  mm_nn<8, C, kDC, kLP, L>(dq, sP, sK, row0, lane);        // dq += dP K
  mm_tn<8, C, kDC, kLP, L>(dk, sP, sQ, row0, lane);        // dk += dP^T Q
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (row0 + i < live)
#pragma unroll
      for (int c = 0; c < C; ++c) a.dq[at + (int64_t)(row0 + i) * ld + lane + 32 * c] = dq[i][c];
  // ---- through W = (I + A)^-1 R: dR = inv^T dW, dA = -dR W^T
  float* sI = sS + kDC * L;                                // dW2 and the inverse share the state's buffer
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) sS[(row0 + i) * L + lane + 32 * c] = -w[i][c];
  load_tile<kDC, kDC, kLP>(sI, a.inv + nh * kDC * kDC, kDC, kDC);
  load_tile<kDC, D, L>(sX, a.dU + at, ld, live);           // dW1
  load_tile<kDC, D, L>(sY, a.W1 + nh * kDC * D, D, kDC);
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  float da[8][2];
  zero(da);
  zero(w);
  mm_tn<8, C, kDC, kLP, L>(w, sI, sX, row0, lane);         // dR1
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int t = row0 + i, col = lane + 32 * c;
      sX[t * L + col] = w[i][c];
      if (t < live) {
        const int64_t e = at + (int64_t)t * ld + col;
        dBt[i] += w[i][c] * a.v[e];
        a.dv[e] = bt[i] * w[i][c];
      }
    }
  __syncthreads();
  mm_nt<8, 2, D, L, L>(da, sX, sY, row0, lane);            // dR1 W1^T
  zero(w);
  mm_tn<8, C, kDC, kLP, L>(w, sI, sS, row0, lane);         // dR2
  __syncthreads();
  load_tile<kDC, D, L>(sY, a.W2 + nh * kDC * D, D, kDC);
  cp_commit();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int t = row0 + i, col = lane + 32 * c;
      sX[t * L + col] = w[i][c];
      const float x = w[i][c] * eg[i];
      dk[i][c] += bt[i] * x;
      const float y = x * sK[t * L + col];
      dBt[i] += y;
      dGt[i] += bt[i] * y;
    }
  cp_wait<0>();
  __syncthreads();
  mm_nt<8, 2, D, L, L>(da, sX, sY, row0, lane);            // + dR2 W2^T
  // ---- A = beta (K K^T) M below the diagonal
  {
    float kk[8][2];
    zero(kk);
    mm_nt<8, 2, D, L, L>(kk, sK, sK, row0, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int t = row0 + i, s = lane + 32 * c;
        const float m = s < t ? exp_d(fmin(sG[t] - sG[s], 0.0)) : 0.f, d = -da[i][c] * m;      // dA * M
        const float y = d * kk[i][c], x = bt[i] * y;
        dBt[i] += y;
        dGt[i] += x;
        col[c] -= x;
        sP[t * kLP + s] = bt[i] * d;                                                           // d(K K^T)
      }
  }
  cG[warp * kDC + lane] = col[0];                          // added over the warps in a fixed order below
  cG[warp * kDC + lane + 32] = col[1];
  __syncthreads();
  mm_nn<8, C, kDC, kLP, L>(dk, sP, sK, row0, lane);
  mm_tn<8, C, kDC, kLP, L>(dk, sP, sK, row0, lane);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (row0 + i < live)
#pragma unroll
      for (int c = 0; c < C; ++c) a.dk[at + (int64_t)(row0 + i) * ld + lane + 32 * c] = dk[i][c];
    const float s = warp_sum(dGt[i]), b = warp_sum(dBt[i]);
    if (lane == 0) { rG[row0 + i] = s; rB[row0 + i] = b; }
  }
  dGc = warp_sum(dGc);
  if (lane == 0) red[warp] = dGc;
  __syncthreads();
  if (warp == 0) {                                         // dg_t = sum of dG from t to the end of the chunk
    const int t = 2 * lane;
    float e0 = rG[t], e1 = rG[t + 1];
    for (int i = 0; i < kDThreads / 32; ++i) {
      e0 += cG[i * kDC + t];
      e1 += cG[i * kDC + t + 1];
      if (lane == 31) e1 += red[i];
    }
    float s = e0 + e1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float u = __shfl_down_sync(0xffffffffu, s, o);
      if (lane + o < 32) s += u;
    }
    if (t < live) { a.dg[(int64_t)(t0 + t) * a.H + h] = s; a.dbeta[(int64_t)(t0 + t) * a.H + h] = rB[t]; }
    if (t + 1 < live) { a.dg[(int64_t)(t0 + t + 1) * a.H + h] = s - e0; a.dbeta[(int64_t)(t0 + t + 1) * a.H + h] = rB[t + 1]; }
  }
}

}  // namespace llmt

using namespace llmt;

template <int D>
static int delta_fwd(const DeltaArgs& a, cudaStream_t st) {
  const int N = (a.T + kDC - 1) / kDC, s1 = PrepSmem<D>::kFloats * 4, s2 = ScanSmem<D>::kFloats * 4;
  static bool cfg = false;
  if (!cfg) {
    if (cudaFuncSetAttribute(delta_prep_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s1) != cudaSuccess ||
        cudaFuncSetAttribute(delta_scan_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2) != cudaSuccess)
      return -2;
    cfg = true;
  }
  delta_prep_kernel<D><<<dim3(N, a.H), kDThreads, s1, st>>>(a);
  delta_scan_fwd_kernel<D><<<dim3(a.H, D / kDV), kDThreads, s2, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
template <int D>
static int delta_bwd(const DeltaArgs& a, cudaStream_t st) {
  const int N = (a.T + kDC - 1) / kDC, s2 = ScanSmem<D>::kFloats * 4, s3 = GradSmem<D>::kFloats * 4;
  static bool cfg = false;
  if (!cfg) {
    if (cudaFuncSetAttribute(delta_scan_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2) != cudaSuccess ||
        cudaFuncSetAttribute(delta_grad_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3) != cudaSuccess)
      return -2;
    cfg = true;
  }
  delta_scan_bwd_kernel<D><<<dim3(a.H, D / kDV), kDThreads, s2, st>>>(a);
  delta_grad_kernel<D><<<dim3(N, a.H), kDThreads, s3, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// All tensors fp32 and contiguous; D 64 or 128 for keys and values. N = ceil(T / 64). W1, W2 [N, H, 64, D], P, inv [N, H, 64, 64],
// G [N, H, 64], S [N, H, D, D], U, o [T, H, D]. inv, S and U are for the backward: null when there is none.
extern "C" int llmt_delta_rule_fwd(const float* q, const float* k, const float* v, const float* beta, const float* g, double* G, float* W1, float* W2,
                                   float* P, float* inv, float* S, float* U, float* o, int T, int H, int D, cudaStream_t st) {
  if (T <= 0 || H <= 0) return 0;
  DeltaArgs a{};
  a.q = q; a.k = k; a.v = v; a.beta = beta; a.g = g; a.G = G; a.W1 = W1; a.W2 = W2; a.P = P; a.inv = inv; a.S = S; a.U = U; a.o = o; a.T = T; a.H = H;
  if (D == 128) return delta_fwd<128>(a, st);
  if (D == 64) return delta_fwd<64>(a, st);
  return -10;
}
extern "C" int llmt_delta_rule_bwd(const float* dout, const float* q, const float* k, const float* v, const float* beta, const double* G, const float* W1,
                                   const float* W2, const float* P, const float* inv, const float* S, const float* U, float* dS, float* dU, float* dq,
                                   float* dk, float* dv, float* dbeta, float* dg, int T, int H, int D, cudaStream_t st) {
  if (T <= 0 || H <= 0) return 0;
  DeltaArgs a{};
  a.dout = dout; a.q = q; a.k = k; a.v = v; a.beta = beta; a.T = T; a.H = H;
  a.G = const_cast<double*>(G); a.W1 = const_cast<float*>(W1); a.W2 = const_cast<float*>(W2); a.P = const_cast<float*>(P);
  a.inv = const_cast<float*>(inv); a.S = const_cast<float*>(S); a.U = const_cast<float*>(U);
  a.dS = dS; a.dU = dU; a.dq = dq; a.dk = dk; a.dv = dv; a.dbeta = dbeta; a.dg = dg;
  if (D == 128) return delta_bwd<128>(a, st);
  if (D == 64) return delta_bwd<64>(a, st);
  return -10;
}
