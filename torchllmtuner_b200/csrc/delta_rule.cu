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
// out 16-bit and TF32 operands. Operands sit in shared memory, a thread holds 8 x 8 (or 8 x 4, 4 x 4) results in registers (see mm).
// Counters at 2048 tokens x 32 heads x 128 (preparation, two scans, gradients): FMA pipes 46, 51, 50, 49 %, shared-memory reads 64, 45,
// 47, 41 %, issue slots 69, 44, 43, 60 %, DRAM 10 to 13 %, 12 % of the warps resident (23 % in the preparation): no pipe is full;
// two warps per scheduler (the tiles leave room for one block per SM) do not cover each other's chains of loads, FMAs and barriers. As tensor expressions (batched products, a triangular solve, a two-level scan
// over state maps, some 600 launches) forward + backward took 5.5 ms at 2048 tokens x 32 heads x 128, with 8 x 1, 16 x 1 and 8 x 4
// results (209 + 461 + 444 + 606 us for the four kernels) 1.72 ms, now 1.16 to 1.18 ms (150 + 250 + 256 + 509); the error against 64 bits
// is 1.2e-7 instead of 3.3e-7 (outputs; gradients 0.5 to 1.0 of it).
#include "common.cuh"
#include "kernels.h"

namespace llmt {

constexpr int kDC = 64;          // tokens per chunk
constexpr int kDV = 32;          // value columns of a scan block
constexpr int kThreads = 256;    // two teams of four warps: where two products do not depend on one another each team does one

// Tiles sit in shared memory without padding; the 16-byte pieces of a row are exchanged within each 128 bytes by XOR with sw(row).
// The eight lanes that one shared access serves together then read or write different banks in every form below (rows 4 or 8 apart
// at the same piece, neighbouring pieces of one row, or four pieces of two rows 8 apart). sw is linear over XOR: sw(r + i) =
// sw(r) ^ sw(i) where r and i have no bit in common.
__host__ __device__ constexpr int sw(int r) { return ((r >> 2) & 1) | ((r >> 1) & 4) | ((r >> 3) & 2); }
template <int LD>
__device__ __forceinline__ int at(int r, int c) { return r * LD + ((((c >> 2) ^ sw(r)) << 2) | (c & 3)); }

template <int R, int C>
__device__ __forceinline__ void zero(float (&acc)[R][C]) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[i][c] = 0.f;
}
__device__ __forceinline__ void get(float* b, const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  b[0] = v.x; b[1] = v.y; b[2] = v.z; b[3] = v.w;
}
__device__ __forceinline__ void set(float* p, const float* b) { *reinterpret_cast<float4*>(p) = make_float4(b[0], b[1], b[2], b[3]); }
// A thread's columns: c0 .. c0 + 3 and, with 8 of them, c0 + 16 .. c0 + 19.
__device__ __forceinline__ constexpr int col_of(int j) { return (j & 3) + (j >> 2) * 16; }

// c += a b for two neighbouring results in one instruction: half the issue slots (forward and backward scan 269 + 273 us -> 254 + 255).
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void fma2(float& c0, float& c1, uint64_t a, float b0, float b1) {
  uint64_t c = pack2(c0, c1);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(pack2(b0, b1)));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(c));
}

template <bool PAIRS>
__device__ __forceinline__ void fma_pair(float& c0, float& c1, float a, float b0, float b1) {
  if constexpr (PAIRS) fma2(c0, c1, pack2(a, a), b0, b1);
  else { c0 = fmaf(a, b0, c0); c1 = fmaf(a, b1, c1); }
}
// One thread's R x C results of a product over K terms from k0 (multiples of 4):
//   NN  acc[i][j] += sum_k A[r0 + i][k] B[k][col]     NT  ... A[r0 + i][k] B[col][k]     TN  ... A[k][r0 + i] B[k][col]
// Shared memory hands a warp 32 floats per clock, broadcast or not, and the FMA pipes take 128 per clock: a loaded float has to feed
// four FMAs, which is an 8 x 8 tile (R C / (R + C) = 4). 8 x 1 and 16 x 1 results (0.9) made the scans 3 times as long as their
// FMAs, 4 x 4 (2) 1.8 times. PAIRS helps where the code is small (the scans); the gradients, which stream through more code than the
// instruction cache holds, got slower with it (636 -> 675 us) and with deeper unrolling (696).
enum class Mm { NN, NT, TN };
template <Mm OP, int R, int C, int K, int LDA, int LDB, int UNROLL = 1, bool PAIRS = false>
__device__ __forceinline__ void mm(float (&acc)[R][C], const float* A, const float* B, int r0, int c0, int k0) {
  static_assert(K % 4 == 0 && (R == 4 || R == 8) && (C == 4 || C == 8), "product shape");
  const int ra = (r0 >> 2) & 7, ca = (c0 >> 2) & 7;
#pragma unroll UNROLL
  for (int kk = 0; kk < K; kk += 4) {
    const int k = k0 + kk, xk = (k >> 2) & 7, sk = sw(k & 31);
    const float* a0 = OP == Mm::TN ? A + k * LDA + ((r0 >> 2) & ~7) * 4 : A + r0 * LDA + (k & ~31);
    const float* b0 = OP == Mm::NT ? B + c0 * LDB + (k & ~31) : B + k * LDB + ((c0 >> 2) & ~7) * 4;
    const int xa = OP == Mm::TN ? ra ^ sk : sw(r0) ^ xk, xb = OP == Mm::NT ? sw(c0) ^ xk : ca ^ sk;
    float b[OP == Mm::NT ? C : 4][OP == Mm::NT ? 4 : C];   // [col][term], else [term][col]
    if constexpr (OP == Mm::NT) {
#pragma unroll
      for (int j = 0; j < C; ++j) get(b[j], b0 + col_of(j) * LDB + ((sw(col_of(j)) ^ xb) << 2));
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < C; j += 4) get(b[q] + j, b0 + q * LDB + ((sw(q) ^ xb ^ j) << 2));   // piece + 4 for the second four
    }
    if constexpr (OP == Mm::TN) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float x[R];
#pragma unroll
        for (int i = 0; i < R; i += 4) get(x + i, a0 + q * LDA + ((sw(q) ^ xa ^ (i >> 2)) << 2));
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int j = 0; j < C; j += 2) fma_pair<PAIRS>(acc[i][j], acc[i][j + 1], x[i], b[q][j], b[q][j + 1]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float x[4];
        get(x, a0 + i * LDA + ((sw(i) ^ xa) << 2));
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int j = 0; j < C; j += 2)
            fma_pair<PAIRS>(acc[i][j], acc[i][j + 1], x[q], OP == Mm::NT ? b[j][q] : b[q][j], OP == Mm::NT ? b[j + 1][q] : b[q][j + 1]);
      }
    }
  }
}
// The same with the contraction summed in blocks of 16: a chain of 64 or 128 roundings at the size of the result becomes 4 to 8.
template <Mm OP, int R, int C, int K, int LDA, int LDB>
__device__ __forceinline__ void mm_blocked(float (&acc)[R][C], const float* A, const float* B, int r0, int c0) {
#pragma unroll 1
  for (int k = 0; k < K; k += 16) {
    float t[R][C];
    zero(t);
    mm<OP, R, C, 16, LDA, LDB, 4>(t, A, B, r0, c0, k);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) acc[i][j] += t[i][j];
  }
}
// Piece j of row r0 + i where a thread owns rows r0 .. r0 + 7 (r0 a multiple of 8) and the columns of col_of from c0: four registers
// plus constants, where at() would cost half a dozen integer instructions each time.
template <int LD>
__device__ __forceinline__ int own(int r0, int c0, int i, int j) {
  return r0 * LD + ((c0 >> 2) & ~7) * 4 + i * LD + (((((c0 >> 2) & 7) ^ sw(r0)) ^ (sw(i) ^ (j & 4))) << 2);
}
// rows r0 .. r0 + 7 of the results into a tile
template <int C, int LD>
__device__ __forceinline__ void put(float* dst, const float (&v)[8][C], int r0, int c0) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < C; j += 4) set(dst + own<LD>(r0, c0, i, j), v[i] + j);
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// ROWS x COLS floats into shared memory; rows at or beyond `live` are zero-filled (their address is not read).
template <int ROWS, int COLS>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int64_t ld, int live) {
  constexpr int V = COLS / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < ROWS * V; i += kThreads) {
    const int r = i / V, c = (i % V) * 4;
    cp16(dst + at<COLS>(r, c), src + (int64_t)(r < live ? r : 0) * ld + c, r < live);
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
  float *W1, *W2, *P, *inv, *M;              // [N, H, 64, D], [N, H, 64, 64]; M the decay ratios e^(G_t - G_i), i <= t
  float *S, *U, *o;                          // [N, H, D, D] state at chunk starts, [T, H, D]
  const float* dout;
  float *dS, *dU;                            // [N, H, D, D] gradient of the state after the chunk, [T, H, D]
  float *dq, *dk, *dv, *dbeta, *dg;
  int T, H;
};

// ------------------------------------------------------------------------------------------ per chunk: A, P, inverse, W
// Two blocks per SM, so that one block's products run under the other's loads and its serial inverse.
template <int D>
struct PrepSmem {
  static constexpr int kBytes = (2 * kDC * D + 2 * kDC * kDC + 48 * 17 + 2 * kDC) * 4 + kDC * 8;
};
template <int D>
__global__ void __launch_bounds__(kThreads, 2) delta_prep_kernel(const DeltaArgs a) {
  constexpr int R = D / 16, LI = kDC;
  extern __shared__ __align__(16) float sm[];
  float *sK = sm, *sQ = sK + kDC * D, *sA = sQ + kDC * D, *sI = sA + kDC * kDC, *sT = sI + kDC * kDC;
  double* sG = reinterpret_cast<double*>(sT + 48 * 17);
  float *sB = reinterpret_cast<float*>(sG + kDC), *sE = sB + kDC;
  const int n = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rg = lane >> 3, cg = lane & 7;
  const int t0 = n * kDC, live = min(kDC, a.T - t0);
  const int64_t off = ((int64_t)t0 * a.H + h) * D, ld = (int64_t)a.H * D, nh = (int64_t)n * a.H + h;
  load_tile<kDC, D>(sK, a.k + off, ld, live);
  load_tile<kDC, D>(sQ, a.q + off, ld, live);
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
  if (threadIdx.x < kDC) {
    a.G[nh * kDC + threadIdx.x] = sG[threadIdx.x];
    sE[threadIdx.x] = exp_d(sG[threadIdx.x]);
  }
  {
    const int r0 = (warp >> 1) * 16 + rg * 4, c0 = (warp & 1) * 32 + cg * 4;
    float kk[4][4], qk[4][4];
    zero(kk); zero(qk);
    mm_blocked<Mm::NT, 4, 4, D, D, D>(kk, sK, sK, r0, c0);
    mm_blocked<Mm::NT, 4, 4, D, D, D>(qk, sQ, sK, r0, c0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = r0 + i;
      float x[4], y[4], m[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int s = c0 + c;
        m[c] = s <= t ? exp_d(fmin(sG[t] - sG[s], 0.0)) : 0.f;
        x[c] = s < t ? sB[t] * kk[i][c] * m[c] : 0.f;
        y[c] = qk[i][c] * m[c];
      }
      if (a.M != nullptr) set(a.M + (nh * kDC + t) * kDC + c0, m);
      set(sA + t * kDC + c0, x);
      set(a.P + (nh * kDC + t) * kDC + c0, y);
    }
  }
  for (int i = threadIdx.x; i < kDC * kDC; i += kThreads) sI[i] = 0.f;
  __syncthreads();
  load_tile<kDC, D>(sQ, a.v + off, ld, live);          // v over q, under the inverse
  cp_commit();
  // (I + A)^-1 by 16 x 16 blocks: the diagonal blocks by forward substitution, one column per thread ...
  if (threadIdx.x < kDC) {
    const int b = threadIdx.x / 16 * 16, j = threadIdx.x % 16;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      float s = r == j ? 1.f : 0.f;
#pragma unroll
      for (int i = 0; i < r; ++i) s -= sA[(b + r) * kDC + b + i] * x[i];
      x[r] = s;
      sI[at<LI>(b + r, b + j)] = s;
    }
  }
  __syncthreads();
  // ... then the blocks d below the diagonal: X_ij = -X_ii (sum_{j <= k < i} A_ik X_kj)
  const int er = threadIdx.x / 16, ec = threadIdx.x % 16;
  for (int d = 1; d < 4; ++d) {
    for (int bi = d; bi < 4; ++bi) {
      const int bj = bi - d;
      float s = 0.f;
      for (int bk = bj * 16; bk < bi * 16; bk += 16)
#pragma unroll
        for (int r = 0; r < 16; ++r) s += sA[(bi * 16 + er) * kDC + bk + r] * sI[at<LI>(bk + r, bj * 16 + ec)];
      sT[((bi - d) * 16 + er) * 17 + ec] = s;
    }
    __syncthreads();
    for (int bi = d; bi < 4; ++bi) {
      float s = 0.f;
#pragma unroll
      for (int r = 0; r < 16; ++r) s -= sI[at<LI>(bi * 16 + er, bi * 16 + r)] * sT[((bi - d) * 16 + r) * 17 + ec];
      sI[at<LI>(bi * 16 + er, (bi - d) * 16 + ec)] = s;
    }
    __syncthreads();
  }
  cp_wait<0>();
  __syncthreads();
  // right-hand sides in place: beta v, beta e^G k
  for (int i = threadIdx.x; i < kDC * D; i += kThreads) {
    const int r = i / D;                                   // a row's order does not matter here
    sQ[i] *= sB[r];
    sK[i] = sB[r] * sE[r] * sK[i];
  }
  if (a.inv != nullptr)
    for (int i = threadIdx.x; i < kDC * kDC / 4; i += kThreads) {
      const int r = i / (kDC / 4), c = i % (kDC / 4) * 4;
      *reinterpret_cast<float4*>(a.inv + (nh * kDC + r) * kDC + c) = *reinterpret_cast<const float4*>(sI + at<LI>(r, c));
    }
  __syncthreads();
  const int r0 = warp / (D / 32) * (4 * R) + rg * R, c0 = warp % (D / 32) * 32 + cg * 4;
  auto rhs = [&](const float* x, float* out) {
    float w[R][4];
    zero(w);
    mm_blocked<Mm::NN, R, 4, kDC, LI, D>(w, sI, x, r0, c0);
#pragma unroll
    for (int i = 0; i < R; ++i) set(out + (nh * kDC + r0 + i) * D + c0, w[i]);
  };
  rhs(sQ, a.W1);
  rhs(sK, a.W2);
}

// ------------------------------------------------------------------------------------------ walk over the chunks
// One block per (head, 32 value columns). A warp holds all 64 rows x 32 columns of a result (8 x 8 per thread) for its share of the
// contraction; the shares are added in shared memory. Tiles are single-buffered: a tile's successor is fetched as soon as its last
// product has read it, so every fetch runs under the products of the other tiles.
template <int D>
struct ScanSmem {
  static constexpr int kRed = 8 * kDC * kDV;               // shares
  static constexpr int kBytes = (3 * kDC * D + kDC * kDC + D * kDV + 3 * kDC * kDV + kRed + 2 * kDC + 4) * 4;
};
template <int KS>
__device__ __forceinline__ void add_shares(float* v, const float* red, int rows, int r, int c) {
  get(v, red + at<kDV>(r, c));
#pragma unroll
  for (int k = 1; k < KS; ++k) {
    float x[4];
    get(x, red + k * rows * kDV + at<kDV>(r, c));
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] += x[j];
  }
}
// 64 threads keep the next chunk's running log decays on their way and turn them into the chunk's decay factors (e^(G_C) has two
// places: it is read after the last barrier of a step)
struct ChunkDecay {
  double g, gc;
  __device__ __forceinline__ void fetch(const double* G, int64_t nh) {
    if (threadIdx.x < kDC) { g = G[nh * kDC + threadIdx.x]; gc = G[nh * kDC + kDC - 1]; }
  }
  __device__ __forceinline__ void publish(float* sEg, float* sEe, float* sEc) const {
    if (threadIdx.x < kDC) {
      sEg[threadIdx.x] = exp_d(g);
      sEe[threadIdx.x] = exp_d(gc - g);
      if (threadIdx.x == 0) *sEc = exp_d(gc);
    }
  }
};
template <int D>
__device__ __forceinline__ void store_state(float* dst, const float* sS, int64_t nh, int v0) {
  for (int i = threadIdx.x; i < D * kDV / 4; i += kThreads) {
    const int r = i / (kDV / 4), c = i % (kDV / 4) * 4;
    *reinterpret_cast<float4*>(dst + (nh * D + r) * D + v0 + c) = *reinterpret_cast<const float4*>(sS + at<kDV>(r, c));
  }
}
template <int D>
__global__ void __launch_bounds__(kThreads, 1) delta_scan_fwd_kernel(const DeltaArgs a) {
  constexpr int HALF = ScanSmem<D>::kRed / 2, KT = 256 / D;   // shares of a state-row result per team
  extern __shared__ __align__(16) float sm[];
  float *sW = sm, *sQ = sW + kDC * D, *sK = sQ + kDC * D, *sP = sK + kDC * D, *sS = sP + kDC * kDC;
  float *sW1 = sS + D * kDV, *sU = sW1 + kDC * kDV, *sE = sU + kDC * kDV, *sR = sE + kDC * kDV;
  float *sEg = sR + 2 * HALF, *sEe = sEg + kDC, *sEc = sEe + kDC;
  const int h = blockIdx.x, v0 = blockIdx.y * kDV, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, team = warp >> 2, w = warp & 3;
  const int N = (a.T + kDC - 1) / kDC;
  const int64_t ld = (int64_t)a.H * D;
  const int r0 = (lane >> 2) * 8, c0 = (lane & 3) * 4;
  const int sh = D == 128 ? (w & 1) * kDC : 0, sk = D == 128 ? w >> 1 : w;     // rows and share of a D x 32 result
  const int er = threadIdx.x / 8, ec = (threadIdx.x % 8) * 4;                  // row and columns when shares are added
  auto fetch_wq = [&](int n) {
    const int64_t nh = (int64_t)n * a.H + h;
    load_tile<kDC, D>(sW, a.W2 + nh * kDC * D, D, kDC);
    load_tile<kDC, kDV>(sW1, a.W1 + nh * kDC * D + v0, D, kDC);
    load_tile<kDC, D>(sQ, a.q + ((int64_t)n * kDC * a.H + h) * D, ld, min(kDC, a.T - n * kDC));
    cp_commit();
  };
  auto fetch_pk = [&](int n) {
    load_tile<kDC, kDC>(sP, a.P + ((int64_t)n * a.H + h) * kDC * kDC, kDC, kDC);
    load_tile<kDC, D>(sK, a.k + ((int64_t)n * kDC * a.H + h) * D, ld, min(kDC, a.T - n * kDC));
    cp_commit();
  };
  for (int i = threadIdx.x; i < D * kDV; i += kThreads) sS[i] = 0.f;
  ChunkDecay decay;
  decay.fetch(a.G, h);
  fetch_wq(0); fetch_pk(0);
  for (int n = 0; n < N; ++n) {
    const int64_t nh = (int64_t)n * a.H + h;
    const int t0 = n * kDC, live = min(kDC, a.T - t0);
    decay.publish(sEg, sEe, sEc + (n & 1));
    if (n + 1 < N) decay.fetch(a.G, nh + a.H);
    cp_wait<1>();                                          // W and Q tiles (P and K are the newer group)
    __syncthreads();                                       // they, the state and the decay factors are here
    if (a.S != nullptr) store_state<D>(a.S, sS, nh, v0);
    float acc[8][8];
    zero(acc);                                             // W2 S by the first team, q S by the second
    mm<Mm::NN, 8, 8, D / 4, D, kDV, 2, true>(acc, team == 0 ? sW : sQ, sS, r0, c0, w * (D / 4));
    if (team == 0) {
      put<8, kDV>(sR + w * kDC * kDV, acc, r0, c0);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float e = sEg[r0 + i];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] *= e;
      }
    }
    __syncthreads();                                       // shares of W2 S are here
#pragma unroll
    for (int r = er; r < kDC; r += kThreads / 8) {
      float u[4], x[4], e[4];
      add_shares<4>(u, sR, kDC, r, ec);
      get(x, sW1 + at<kDV>(r, ec));
#pragma unroll
      for (int j = 0; j < 4; ++j) { u[j] = x[j] - u[j]; e[j] = sEe[r] * u[j]; }
      set(sU + at<kDV>(r, ec), u);
      set(sE + at<kDV>(r, ec), e);
      if (r < live && a.U != nullptr) set(a.U + ((int64_t)(t0 + r) * a.H + h) * D + v0 + ec, u);
    }
    cp_wait<0>();
    __syncthreads();                                       // U complete, W and Q free, P and K here
    if (n + 1 < N) fetch_wq(n + 1);
    if (team == 0) {                                       // the chunk's sum first: one rounding at the size of the state
      zero(acc);
      mm<Mm::TN, 8, 8, kDC / KT, D, kDV, 2, true>(acc, sK, sE, sh + r0, c0, sk * (kDC / KT));
      put<8, kDV>(sR + sk * D * kDV, acc, sh + r0, c0);
    } else {
      mm<Mm::NN, 8, 8, kDC / 4, kDC, kDV, 2, true>(acc, sP, sU, r0, c0, w * (kDC / 4));
      put<8, kDV>(sR + HALF + w * kDC * kDV, acc, r0, c0);
    }
    __syncthreads();                                       // shares of O and of the state are here, P and K free
    if (n + 1 < N) fetch_pk(n + 1); else cp_commit();
#pragma unroll
    for (int r = er; r < kDC; r += kThreads / 8) {
      float x[4];
      add_shares<4>(x, sR + HALF, kDC, r, ec);
      if (r < live) set(a.o + ((int64_t)(t0 + r) * a.H + h) * D + v0 + ec, x);
    }
    const float f = sEc[n & 1];
#pragma unroll
    for (int r = er; r < D; r += kThreads / 8) {
      float x[4], y[4];
      add_shares<KT>(x, sR, D, r, ec);
      get(y, sS + at<kDV>(r, ec));
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = fmaf(f, y[j], x[j]);
      set(sS + at<kDV>(r, ec), y);
    }
  }
  cp_wait<0>();
}

// Backwards: dU = P^T dO + e^(G_C - G) (k dS'),  dS = e^(G_C) dS' + q^T (e^G dO) - W2^T dU.
template <int D>
__global__ void __launch_bounds__(kThreads, 1) delta_scan_bwd_kernel(const DeltaArgs a) {
  constexpr int KT = 256 / D;
  constexpr int Y1 = (kDC + D) / 8, Y0 = Y1 - kDC / 4;     // terms of k dS' per warp of the second and of the first team, which has P^T dO
  extern __shared__ __align__(16) float sm[];
  float *sW = sm, *sQ = sW + kDC * D, *sK = sQ + kDC * D, *sP = sK + kDC * D, *sS = sP + kDC * kDC;
  float *sO = sS + D * kDV, *sU = sO + kDC * kDV, *sE = sU + kDC * kDV, *sR = sE + kDC * kDV;
  float *sEg = sR + ScanSmem<D>::kRed, *sEe = sEg + kDC, *sEc = sEe + kDC;
  const int h = blockIdx.x, v0 = blockIdx.y * kDV, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, team = warp >> 2, w = warp & 3;
  const int N = (a.T + kDC - 1) / kDC;
  const int64_t ld = (int64_t)a.H * D;
  const int r0 = (lane >> 2) * 8, c0 = (lane & 3) * 4;
  const int sh = D == 128 ? (w & 1) * kDC : 0, sk = D == 128 ? w >> 1 : w;
  const int er = threadIdx.x / 8, ec = (threadIdx.x % 8) * 4;
  auto fetch_kp = [&](int n) {                             // first group of a step: K, P, dO
    const int live = min(kDC, a.T - n * kDC);
    const int64_t off = ((int64_t)n * kDC * a.H + h) * D;
    load_tile<kDC, D>(sK, a.k + off, ld, live);
    load_tile<kDC, kDC>(sP, a.P + ((int64_t)n * a.H + h) * kDC * kDC, kDC, kDC);
    load_tile<kDC, kDV>(sO, a.dout + off + v0, ld, live);
    cp_commit();
  };
  auto fetch_qw = [&](int n) {                             // second group: Q, W2
    load_tile<kDC, D>(sQ, a.q + ((int64_t)n * kDC * a.H + h) * D, ld, min(kDC, a.T - n * kDC));
    load_tile<kDC, D>(sW, a.W2 + ((int64_t)n * a.H + h) * kDC * D, D, kDC);
    cp_commit();
  };
  for (int i = threadIdx.x; i < D * kDV; i += kThreads) sS[i] = 0.f;
  ChunkDecay decay;
  decay.fetch(a.G, (int64_t)(N - 1) * a.H + h);
  fetch_kp(N - 1); fetch_qw(N - 1);
  for (int n = N - 1; n >= 0; --n) {
    const int64_t nh = (int64_t)n * a.H + h;
    const int t0 = n * kDC, live = min(kDC, a.T - t0);
    decay.publish(sEg, sEe, sEc + (n & 1));
    if (n > 0) decay.fetch(a.G, nh - a.H);
    cp_wait<1>();
    __syncthreads();
    store_state<D>(a.dS, sS, nh, v0);
    float acc[8][8];
    zero(acc);
    if (team == 1) mm<Mm::NN, 8, 8, Y1, D, kDV, 2, true>(acc, sK, sS, r0, c0, w * Y1);
    else if constexpr (Y0 > 0) mm<Mm::NN, 8, 8, Y0, D, kDV, 2, true>(acc, sK, sS, r0, c0, 4 * Y1 + w * Y0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float e = sEe[r0 + i];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] *= e;
    }
    if (team == 0) mm<Mm::TN, 8, 8, kDC / 4, kDC, kDV, 2, true>(acc, sP, sO, r0, c0, w * (kDC / 4));
    put<8, kDV>(sR + warp * kDC * kDV, acc, r0, c0);
    __syncthreads();                                       // shares of dU are here
#pragma unroll
    for (int r = er; r < kDC; r += kThreads / 8) {
      float d[4], e[4];
      add_shares<8>(d, sR, kDC, r, ec);
      if (r < live) set(a.dU + ((int64_t)(t0 + r) * a.H + h) * D + v0 + ec, d);
      get(e, sO + at<kDV>(r, ec));
#pragma unroll
      for (int j = 0; j < 4; ++j) { d[j] = -d[j]; e[j] *= sEg[r]; }
      set(sU + at<kDV>(r, ec), d);
      set(sE + at<kDV>(r, ec), e);
    }
    cp_wait<0>();
    __syncthreads();                                       // dU complete; K, P and dO free; Q and W here
    if (n > 0) fetch_kp(n - 1);
    zero(acc);                                             // q^T (e^G dO) by the first team, -W2^T dU by the second
    mm<Mm::TN, 8, 8, kDC / KT, D, kDV, 2, true>(acc, team == 0 ? sQ : sW, team == 0 ? sE : sU, sh + r0, c0, sk * (kDC / KT));
    put<8, kDV>(sR + (team * KT + sk) * D * kDV, acc, sh + r0, c0);
    __syncthreads();                                       // shares of the state are here; Q, W free
    if (n > 0) fetch_qw(n - 1); else cp_commit();
    const float f = sEc[n & 1];
#pragma unroll
    for (int r = er; r < D; r += kThreads / 8) {
      float x[4], y[4];
      add_shares<2 * KT>(x, sR, D, r, ec);
      get(y, sS + at<kDV>(r, ec));
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = fmaf(f, y[j], x[j]);
      set(sS + at<kDV>(r, ec), y);
    }
  }
  cp_wait<0>();
}

// ------------------------------------------------------------------------------------------ per chunk: input gradients
// The two teams take products of the same step side by side; a thread owns rows r0 .. r0 + 7 and C of D columns (or 4 of 64). The
// decay ratios come from the preparation: forming their 64 exponentials per thread here took 120 us more.
template <int D>
struct GradSmem {
  static constexpr int kBig = (D * D > kDC * D + kDC * kDC) ? D * D : kDC * D + kDC * kDC;   // a state, or dW2 and the inverse
  static constexpr int kBytes = (4 * kDC * D + kBig + kDC * kDC + 3 * kDC + (2 * 8 + 1) * kDC + 8) * 4 + kDC * 8;
};
template <int D>
__global__ void __launch_bounds__(kThreads, 1) delta_grad_kernel(const DeltaArgs a) {
  constexpr int C = D / 16, V = D / 4, PRE = D * V / kThreads;
  extern __shared__ __align__(16) float sm[];
  float *sK = sm, *sQ = sK + kDC * D, *sX = sQ + kDC * D, *sY = sX + kDC * D, *sS = sY + kDC * D, *sP = sS + GradSmem<D>::kBig;
  double* sG = reinterpret_cast<double*>(sP + kDC * kDC);
  float *sB = reinterpret_cast<float*>(sG + kDC), *sEg = sB + kDC, *sEe = sEg + kDC;
  float *rG = sEe + kDC, *rB = rG + 8 * kDC, *cG = rB + 8 * kDC, *red = cG + kDC;          // row sums [8 warps][64], column sums
  float* sI = sS + kDC * D;
  const int n = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, team = warp >> 2, w = warp & 3;
  const int t0 = n * kDC, live = min(kDC, a.T - t0);
  const int64_t off = ((int64_t)t0 * a.H + h) * D, ld = (int64_t)a.H * D, nh = (int64_t)n * a.H + h;
  const int r0 = (lane >> 2) * 8, c0 = w * (D / 4) + (lane & 3) * 4, s0 = w * 16 + (lane & 3) * 4;
  load_tile<kDC, D>(sX, a.dout + off, ld, live);           // dO
  load_tile<kDC, D>(sY, a.dU + off, ld, live);             // dU = dW1
  load_tile<D, D>(sS, a.S + nh * D * D, D, D);
  cp_commit();
  load_tile<kDC, D>(sQ, a.q + off, ld, live);
  load_tile<kDC, D>(sK, a.k + off, ld, live);
  cp_commit();
  if (threadIdx.x < kDC) {
    const double g = a.G[nh * kDC + threadIdx.x], gc = a.G[nh * kDC + kDC - 1];
    sG[threadIdx.x] = g;
    sEg[threadIdx.x] = exp_d(g);
    sEe[threadIdx.x] = exp_d(gc - g);
    sB[threadIdx.x] = (int)threadIdx.x < live ? a.beta[(int64_t)(t0 + threadIdx.x) * a.H + h] : 0.f;
  }
  float dGt[8], dBt[8];                                    // row sums of dG and dbeta (this thread's columns)
#pragma unroll
  for (int i = 0; i < 8; ++i) { dGt[i] = 0.f; dBt[i] = 0.f; }
  float dGc = 0.f;                                         // gradient of G at the end of the chunk (this thread's share)
  float4 ds[PRE];                                          // the state gradient is on its way during the first products
#pragma unroll
  for (int p = 0; p < PRE; ++p) ds[p] = reinterpret_cast<const float4*>(a.dS + nh * D * D)[threadIdx.x + p * kThreads];
  cp_wait<1>();
  __syncthreads();
  // ---- products with the state: dq = e^G (dO S^T) | -dW2 = dU S^T, which the second team keeps until the state's buffer is free
  float x1[8][C];
  zero(x1);
  mm<Mm::NT, 8, C, D, D, D>(x1, team == 0 ? sX : sY, sS, r0, c0, 0);
  __syncthreads();
  load_tile<kDC, D>(sY, a.U + off, ld, live);              // U over dU
  cp_commit();
  // ---- the state gradient takes the state's place; its product with the state is the gradient of the chunk's decay
  {
    float s = 0.f;
#pragma unroll
    for (int p = 0; p < PRE; ++p) {
      const int i = threadIdx.x + p * kThreads;
      float4* at4 = reinterpret_cast<float4*>(sS + at<D>(i / V, (i % V) * 4));
      const float4 x = *at4, d = ds[p];
      s += d.x * x.x + d.y * x.y + d.z * x.z + d.w * x.w;
      *at4 = d;
    }
    dGc += s * exp_d(sG[kDC - 1]);
  }
  cp_wait<0>();
  __syncthreads();
  // ---- dP = tril(dO U^T), its decay factors go to dG, and K K^T | dk = e^(G_C - G) (U dS'^T)
  float x2[8][C], kk[8][4], col[4] = {0.f, 0.f, 0.f, 0.f};   // col: column sums of dG over this thread's rows
  if (team == 0) {
    float p[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int j = 0; j < C; j += 4) {
        float q[4];
        get(q, sQ + own<D>(r0, c0, i, j));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          x1[i][j + c] *= sEg[r0 + i];
          dGt[i] += x1[i][j + c] * q[c];
        }
      }
    }
    zero(p);
    mm<Mm::NT, 8, 4, D, D, D>(p, sX, sY, r0, s0, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = r0 + i;
      float pt[4], m[4];
      get(pt, a.P + (nh * kDC + t) * kDC + s0);
      get(m, a.M + (nh * kDC + t) * kDC + s0);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float x = p[i][c] * pt[c];                   // P and M are zero above the diagonal
        dGt[i] += x;
        col[c] -= x;
        p[i][c] *= m[c];
      }
    }
    put<4, kDC>(sP, p, r0, s0);
    zero(kk);
    mm<Mm::NT, 8, 4, D, D, D>(kk, sK, sK, r0, s0, 0);
  } else {
    zero(x2);
    mm<Mm::NT, 8, C, D, D, D>(x2, sY, sS, r0, c0, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < C; j += 4) {
        float k[4];
        get(k, sK + own<D>(r0, c0, i, j));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          x2[i][j + c] *= sEe[r0 + i];
          const float x = x2[i][j + c] * k[c];
          dGt[i] -= x;
          dGc += x;
        }
      }
  }
  __syncthreads();                                         // dP here; dO, U and the state gradient are free
  load_tile<kDC, kDC>(sI, a.inv + nh * kDC * kDC, kDC, kDC);
  load_tile<kDC, D>(sX, a.dU + off, ld, live);             // dW1
  load_tile<kDC, D>(sY, a.W1 + nh * kDC * D, D, kDC);
  cp_commit();
  // ---- dq += dP K | dk += dP^T q
  if (team == 0) {
    mm<Mm::NN, 8, C, kDC, kDC, D>(x1, sP, sK, r0, c0, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (r0 + i < live)
#pragma unroll
        for (int j = 0; j < C; j += 4) set(a.dq + off + (int64_t)(r0 + i) * ld + c0 + col_of(j), x1[i] + j);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) x1[i][j] = -x1[i][j];
    put<C, D>(sS, x1, r0, c0);                             // dW2
    mm<Mm::TN, 8, C, kDC, kDC, D>(x2, sP, sQ, r0, c0, 0);
  }
  cp_wait<0>();
  __syncthreads();                                         // q is free
  load_tile<kDC, D>(sQ, a.W2 + nh * kDC * D, D, kDC);
  cp_commit();
  // ---- through W = (I + A)^-1 R: dR = inv^T dW for dW1 | dW2, then dA = -dR W^T
  zero(x1);
  mm<Mm::TN, 8, C, kDC, kDC, D>(x1, sI, team == 0 ? sX : sS, r0, c0, 0);
  __syncthreads();
  put<C, D>(team == 0 ? sX : sS, x1, r0, c0);
  if (team == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = r0 + i;
      if (t < live) {
#pragma unroll
        for (int j = 0; j < C; j += 4) {
          const int64_t e = off + (int64_t)t * ld + c0 + col_of(j);
          float v[4];
          get(v, a.v + e);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            dBt[i] += x1[i][j + c] * v[c];
            x1[i][j + c] *= sB[t];
          }
          set(a.dv + e, x1[i] + j);
        }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float b = sB[r0 + i], e = sEg[r0 + i];
#pragma unroll
      for (int j = 0; j < C; j += 4) {
        float k[4];
        get(k, sK + own<D>(r0, c0, i, j));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float x = x1[i][j + c] * e;
          x2[i][j + c] += b * x;
          const float y = x * k[c];
          dBt[i] += y;
          dGt[i] += b * y;
        }
      }
    }
  }
  cp_wait<0>();
  __syncthreads();
  {
    float da[8][4];
    zero(da);
    mm<Mm::NT, 8, 4, D, D, D>(da, team == 0 ? sX : sS, team == 0 ? sY : sQ, r0, s0, 0);
    if (team == 1) put<4, kDC>(sP, da, r0, s0);
    __syncthreads();
    if (team == 0) {                                       // A = beta (K K^T) M below the diagonal
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = r0 + i;
        float d2[4], m[4];
        get(d2, sP + own<kDC>(r0, s0, i, 0));
        get(m, a.M + (nh * kDC + t) * kDC + s0);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int s = s0 + c;
          const float d = s < t ? -(da[i][c] + d2[c]) * m[c] : 0.f;                                        // dA * M
          const float y = d * kk[i][c], x = sB[t] * y;
          dBt[i] += y;
          dGt[i] += x;
          col[c] -= x;
          da[i][c] = sB[t] * d;                                                                          // d(K K^T)
        }
      }
      put<4, kDC>(sP, da, r0, s0);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) col[c] += __shfl_xor_sync(0xffffffffu, col[c], o);
      }
      if (lane < 4) set(cG + s0, col);
    }
  }
  __syncthreads();
  // ---- dk += d(K K^T)^T K | dk += d(K K^T) K
  if (team == 0) {
    zero(x1);
    mm<Mm::TN, 8, C, kDC, kDC, D>(x1, sP, sK, r0, c0, 0);
    put<C, D>(sX, x1, r0, c0);
  } else {
    mm<Mm::NN, 8, C, kDC, kDC, D>(x2, sP, sK, r0, c0, 0);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float s = dGt[i], b = dBt[i];
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((lane & 3) == 0) { rG[warp * kDC + r0 + i] = s; rB[warp * kDC + r0 + i] = b; }
  }
  dGc = warp_sum(dGc);
  if (lane == 0) red[warp] = dGc;
  __syncthreads();
  if (team == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (r0 + i < live)
#pragma unroll
        for (int j = 0; j < C; j += 4) {
          float x[4];
          get(x, sX + own<D>(r0, c0, i, j));
#pragma unroll
          for (int c = 0; c < 4; ++c) x[c] += x2[i][j + c];
          set(a.dk + off + (int64_t)(r0 + i) * ld + c0 + col_of(j), x);
        }
  } else if (warp == 0) {                                  // dg_t = sum of dG from t to the end of the chunk
    const int t = 2 * lane;
    double e0 = cG[t], e1 = cG[t + 1];                     // rows and columns cancel: their sum keeps the bits of its terms
    float b0 = 0.f, b1 = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      e0 += rG[i * kDC + t];
      e1 += rG[i * kDC + t + 1];
      b0 += rB[i * kDC + t];
      b1 += rB[i * kDC + t + 1];
      if (lane == 31) e1 += red[i];
    }
    double s = e0 + e1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double u = __shfl_down_sync(0xffffffffu, s, o);
      if (lane + o < 32) s += u;
    }
    if (t < live) { a.dg[(int64_t)(t0 + t) * a.H + h] = (float)s; a.dbeta[(int64_t)(t0 + t) * a.H + h] = b0; }
    if (t + 1 < live) { a.dg[(int64_t)(t0 + t + 1) * a.H + h] = (float)(s - e0); a.dbeta[(int64_t)(t0 + t + 1) * a.H + h] = b1; }
  }
}

}  // namespace llmt

using namespace llmt;

template <int D>
static int delta_fwd(const DeltaArgs& a, cudaStream_t st) {
  const int N = (a.T + kDC - 1) / kDC, s1 = PrepSmem<D>::kBytes, s2 = ScanSmem<D>::kBytes;
  static bool cfg = false;
  if (!cfg) {
    if (cudaFuncSetAttribute(delta_prep_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s1) != cudaSuccess ||
        cudaFuncSetAttribute(delta_scan_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2) != cudaSuccess)
      return -2;
    cfg = true;
  }
  delta_prep_kernel<D><<<dim3(N, a.H), kThreads, s1, st>>>(a);
  delta_scan_fwd_kernel<D><<<dim3(a.H, D / kDV), kThreads, s2, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
template <int D>
static int delta_bwd(const DeltaArgs& a, cudaStream_t st) {
  const int N = (a.T + kDC - 1) / kDC, s2 = ScanSmem<D>::kBytes, s3 = GradSmem<D>::kBytes;
  static bool cfg = false;
  if (!cfg) {
    if (cudaFuncSetAttribute(delta_scan_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2) != cudaSuccess ||
        cudaFuncSetAttribute(delta_grad_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3) != cudaSuccess)
      return -2;
    cfg = true;
  }
  delta_scan_bwd_kernel<D><<<dim3(a.H, D / kDV), kThreads, s2, st>>>(a);
  delta_grad_kernel<D><<<dim3(N, a.H), kThreads, s3, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

static float* second_half(float* inv, int T, int H) { return inv == nullptr ? nullptr : inv + (int64_t)((T + kDC - 1) / kDC) * H * kDC * kDC; }

// All tensors fp32 and contiguous; D 64 or 128 for keys and values. N = ceil(T / 64). W1, W2 [N, H, 64, D], P [N, H, 64, 64],
// inv [2, N, H, 64, 64] (the inverses, then the decay ratios), G [N, H, 64], S [N, H, D, D], U, o [T, H, D]. inv, S and U are for
// the backward: null when there is none.
extern "C" int llmt_delta_rule_fwd(const float* q, const float* k, const float* v, const float* beta, const float* g, double* G, float* W1, float* W2,
                                   float* P, float* inv, float* S, float* U, float* o, int T, int H, int D, cudaStream_t st) {
  if (T <= 0 || H <= 0) return 0;
  DeltaArgs a{};
  a.q = q; a.k = k; a.v = v; a.beta = beta; a.g = g; a.G = G; a.W1 = W1; a.W2 = W2; a.P = P; a.inv = inv; a.M = second_half(inv, T, H); a.S = S; a.U = U; a.o = o; a.T = T; a.H = H;
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
  a.inv = const_cast<float*>(inv); a.M = second_half(a.inv, T, H); a.S = const_cast<float*>(S); a.U = const_cast<float*>(U);
  a.dS = dS; a.dU = dU; a.dq = dq; a.dk = dk; a.dv = dv; a.dbeta = dbeta; a.dg = dg;
  if (D == 128) return delta_bwd<128>(a, st);
  if (D == 64) return delta_bwd<64>(a, st);
  return -10;
}
