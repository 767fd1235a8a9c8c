// Flash-attention backward for head size 256 on tcgen05 / TMEM (reference call sites: llmtuner/models/qwen/qwen3/model.py:270-283,
// llmtuner/kernel/ops/varlen_attention.py:60-85; Qwen3.5's full-attention layers have 256-wide heads).
//
// At this width dK and dV of one 128-key tile alone fill the 512 tensor-memory columns, so the three gradients are three walks
// of one skeleton over (128 resident rows) x (64 streamed rows):
//     X = R1 B1^T        Y = R2 B2^T        OUT += f(X, Y) B3            (contractions over 256, 256 and 64)
//   dQ: rows = queries, stream = keys:     R1 = Q, B1 = K, R2 = dO, B2 = V,  f = dS,   B3 = K
//   dK: rows = keys,    stream = queries:  R1 = K, B1 = Q, R2 = V,  B2 = dO, f = dS^T, B3 = Q
//   dV: rows = keys,    stream = queries:  R1 = K, B1 = Q,                   f = P^T,  B3 = dO
// OUT takes 256 columns, X and Y two buffers of 64 columns each; f is written back over X as packed bf16 and is the A operand
// of the third product straight from tensor memory, so it costs no shared memory: 128 KB of resident rows, two 32 KB stages
// of B1 (needed until OUT) and one of B2 (free after Y) are 224 KB. dV has no second product and streams both operands in two
// stages. Eight products instead of the five of the one-kernel form for narrower heads, but every sum stays on the SM and in
// a fixed order: the gradients are bitwise reproducible.
// One launch holds all three walks (dK, dQ, then the shorter dV), heaviest tiles first, so that none of them has a tail of its own.
// Bound by the chain of an iteration, not by a pipe: reload of B2 (one stage: a TMA round trip) -> X, Y -> f -> OUT. Counters: tensor
// pipe active 42 %, issue slots 17 %, DRAM 8 %, and the warps wait on tensor memory and barriers. 4096 tokens in two documents,
// 16 / 4 heads: 381 us with the delta and partial-sum passes; the row-chunked form with library products and some 330 launches
// took 1.85 ms. Relative error against 64 bits 0.0025 (0.0030 before).
#include "attn_common.cuh"

namespace llmt {

constexpr int kWideHD = 256;
constexpr int kWideCols = 64;                          // streamed rows per iteration
constexpr int kWideRes = 128 * kWideHD * 2;            // a resident tile: 64 KB
constexpr int kWideStr = kWideCols * kWideHD * 2;      // a streamed tile: 32 KB
constexpr int kWideThreads = 64 + 256;                 // TMA warp, MMA warp, 8 compute warps (two per lane quarter, 32 columns each)
constexpr int kWideSmem = 2 * kWideRes + 3 * kWideStr + 4 * kWideCols * 4 + 256;   // exact: the kernel checks the alignment of its base

enum WideMode { kWideDQ = 0, kWideDK = 1, kWideDV = 2 };

struct WideArgs {
  const float *lse, *delta;
  __nv_bfloat16 *dq, *dk, *dv;
  float* part;               // [2][nsplit][Tk][Hkv][256] fp32 partial dK, dV when nsplit > 1
  const int *q_tiles, *k_tiles;
  int num_q_tiles, num_k_tiles, Hq, Hkv, Tq, Tk, nsplit, causal;
  int64_t dq_stride, dk_stride, dv_stride;
  float scale;
  int* status;
};

template <int MODE>
__device__ __forceinline__ void wide_walk(const CUtensorMap* mR1, const CUtensorMap* mR2, const CUtensorMap* mB1, const CUtensorMap* mB2,
                                          const WideArgs& a, int block, uint8_t* smem) {
  constexpr bool HAS_Y = MODE != kWideDV;
  constexpr int S2 = HAS_Y ? 1 : 2;                    // stages of the second stream
  uint8_t* sR1 = smem;
  uint8_t* sR2 = sR1 + kWideRes;                       // dV: the second stage pair of the streams starts here instead
  uint8_t* sB1 = HAS_Y ? sR2 + kWideRes : sR2;         // [2]
  uint8_t* sB2 = sB1 + 2 * kWideStr;                   // [S2]
  float* s_lse = reinterpret_cast<float*>(smem + 2 * kWideRes + 3 * kWideStr);   // [2][64]
  float* s_delta = s_lse + 2 * kWideCols;                                        // [2][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_delta + 2 * kWideCols);
  uint64_t* r_full = bars;
  uint64_t* b1_full = bars + 1;     // [2]
  uint64_t* b1_empty = bars + 3;    // [2]
  uint64_t* b2_full = bars + 5;     // [2]
  uint64_t* b2_empty = bars + 7;    // [2]
  uint64_t* x_full = bars + 9;      // [2]
  uint64_t* f_full = bars + 11;     // [2]
  uint64_t* out_done = bars + 13;
  uint64_t* stat_ready = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* status = a.status;

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int g = a.Hq / a.Hkv;
  // rows: first row of the resident tile, its head and live rows; the stream: first row, rows per head and heads to walk
  int row0, nrow, rhead, n_it, per_head = 1, str0, shead0;
  int klen, diag0 = 0, kk0 = 0, qlen = 0, off = 0, qs = 0, part_idx = 0;
  if constexpr (MODE == kWideDQ) {
    const int* tl = a.q_tiles + (block / a.Hq) * 8;
    rhead = block % a.Hq;
    row0 = tl[0]; nrow = tl[1]; str0 = tl[2]; klen = tl[3]; diag0 = tl[4];
    shead0 = rhead / g;
    const int kmax = a.causal ? min(klen, diag0 + nrow - 1) : klen;
    n_it = (kmax + kWideCols - 1) / kWideCols;
    per_head = n_it > 0 ? n_it : 1;
  } else {
    const int per_tile = a.Hkv * a.nsplit;
    const int* tl = a.k_tiles + (block / per_tile) * 8;
    rhead = (block % per_tile) / a.nsplit;
    part_idx = block % a.nsplit;
    row0 = tl[0]; nrow = tl[1]; kk0 = tl[2]; qlen = tl[4]; off = tl[5]; klen = tl[6];
    if (a.causal) { qs = kk0 - off; if (qs < 0) qs = 0; qs &= ~(kWideCols - 1); }
    str0 = tl[3] + qs;
    const int n_qt = (qlen > qs) ? (qlen - qs + kWideCols - 1) / kWideCols : 0;
    const int heads = g / a.nsplit;
    n_it = n_qt * heads;
    per_head = n_qt > 0 ? n_qt : 1;
    shead0 = rhead * g + part_idx * heads;
  }

  if (threadIdx.x == 0) {
    mbar_init(r_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&b1_full[s], 1); mbar_init(&b1_empty[s], 1); mbar_init(&b2_full[s], 1); mbar_init(&b2_empty[s], 1);
      mbar_init(&x_full[s], 1); mbar_init(&f_full[s], 256);
    }
    mbar_init(out_done, 1); mbar_init(stat_ready, 256);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tOut = tmem_base, tX = tmem_base + 256, tY = tmem_base + 384;   // X, Y: two buffers of 64 columns

  if (warp == 0) {
    // ------------------------------------------------------------------------------------ TMA producer
    if (lane == 0 && n_it > 0) {
      tma_prefetch_desc(mR1); tma_prefetch_desc(mB1); tma_prefetch_desc(mB2);
      mbar_arrive_expect_tx(r_full, HAS_Y ? 2 * kWideRes : kWideRes);
#pragma unroll
      for (int hf = 0; hf < 4; ++hf) {
        tma_load_3d(sR1 + hf * 16384, mR1, r_full, hf * 64, rhead, row0);
        if constexpr (HAS_Y) tma_load_3d(sR2 + hf * 16384, mR2, r_full, hf * 64, rhead, row0);
      }
      int armed1[2] = {-1, -1}, armed2[2] = {-1, -1};
      for (int it = 0; it < n_it; ++it) {
        const int head = shead0 + it / per_head, row = str0 + (it % per_head) * kWideCols;
        const int s = it & 1;
        const uint32_t ph = (it >> 1) & 1;
        if (!mbar_wait_bounded(&b1_empty[s], ph ^ 1, abort_flag, status, 4100 + s)) break;
        mbar_arrive_expect_tx(&b1_full[s], kWideStr);
        armed1[s] = (int)ph;
#pragma unroll
        for (int hf = 0; hf < 4; ++hf) tma_load_3d(sB1 + s * kWideStr + hf * 8192, mB1, &b1_full[s], hf * 64, head, row);
        const int s2 = S2 == 1 ? 0 : s;
        const uint32_t ph2 = S2 == 1 ? (it & 1) : ph;
        if (!mbar_wait_bounded(&b2_empty[s2], ph2 ^ 1, abort_flag, status, 4110 + s2)) break;
        mbar_arrive_expect_tx(&b2_full[s2], kWideStr);
        armed2[s2] = (int)ph2;
#pragma unroll
        for (int hf = 0; hf < 4; ++hf) tma_load_3d(sB2 + s2 * kWideStr + hf * 8192, mB2, &b2_full[s2], hf * 64, head, row);
      }
      if (*abort_flag) {
        // wait (bounded) for copies in flight before shared memory is released
        for (uint32_t i = 0; i < (1u << 16); ++i) if (mbar_try_wait(r_full, 0)) break;
        for (int s = 0; s < 2; ++s) {
          if (armed1[s] >= 0)
            for (uint32_t i = 0; i < (1u << 16); ++i) if (mbar_try_wait(&b1_full[s], (uint32_t)armed1[s])) break;
          if (armed2[s] >= 0)
            for (uint32_t i = 0; i < (1u << 16); ++i) if (mbar_try_wait(&b2_full[s], (uint32_t)armed2[s])) break;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------ MMA issuer
    // warp-uniform control flow, one lane issues (see uniform_warp)
    if (n_it > 0) {
      constexpr uint32_t idX = umma_idesc_bf16(128, kWideCols, false, false);
      constexpr uint32_t idOut = umma_idesc_bf16(128, kWideHD, false, true);
      const uint32_t loR1 = desc_lo(smem_u32(sR1), 16), loR2 = desc_lo(smem_u32(sR2), 16);
      const uint32_t lo1 = desc_lo(smem_u32(sB1), 16), lo2 = desc_lo(smem_u32(sB2), 16), lo3 = desc_lo(smem_u32(HAS_Y ? sB1 : sB2), kWideCols * 128);
      constexpr uint32_t kStep = kWideStr >> 4;
      const bool leader = elect_one();
      bool ok = mbar_wait_bounded(r_full, 0, abort_flag, status, 4200);
      // X (and Y) of iteration `it` into buffer it & 1. That buffer's previous content has been consumed: this warp has
      // waited for f of iteration it - 2 and issued its product, and products run in the order in which they are issued.
      auto issue_xy = [&](auto sc, int it) -> bool {
        constexpr int s = decltype(sc)::value;
        if (!mbar_wait_bounded(&b1_full[s], (it >> 1) & 1, abort_flag, status, 4210 + s)) return false;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < kWideHD / 16; ++ks)
            umma_bf16_ss(tX + s * kWideCols, desc_pack(loR1 + koff(ks, 128)), desc_pack(lo1 + s * kStep + koff(ks, kWideCols)), idX, ks ? 1u : 0u);
          if constexpr (!HAS_Y) umma_commit(&b1_empty[s]);
        }
        if constexpr (HAS_Y) {
          if (!mbar_wait_bounded(&b2_full[0], it & 1, abort_flag, status, 4220)) return false;
          tc_fence_after();
          if (leader) {
#pragma unroll
            for (int ks = 0; ks < kWideHD / 16; ++ks)
              umma_bf16_ss(tY + s * kWideCols, desc_pack(loR2 + koff(ks, 128)), desc_pack(lo2 + koff(ks, kWideCols)), idX, ks ? 1u : 0u);
            umma_commit(&b2_empty[0]);
          }
        }
        if (leader) umma_commit(&x_full[s]);
        return true;
      };
      auto step = [&](auto sc, auto nc, int it) -> bool {
        constexpr int s = decltype(sc)::value;
        if (it + 1 < n_it && !issue_xy(nc, it + 1)) return false;
        if (!mbar_wait_bounded(&f_full[s], (it >> 1) & 1, abort_flag, status, 4230 + s)) return false;
        if constexpr (!HAS_Y)
          if (!mbar_wait_bounded(&b2_full[s], (it >> 1) & 1, abort_flag, status, 4240 + s)) return false;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < kWideCols / 16; ++ks)   // f: 8 columns per 16 of the contraction, each half of it over its half of X
            umma_bf16_ts(tOut, tX + s * kWideCols + (ks >> 1) * 32 + (ks & 1) * 8, desc_pack(lo3 + s * kStep + mnoff(ks)), idOut,
                         ks ? 1u : (it ? 1u : 0u));
          umma_commit(HAS_Y ? &b1_empty[s] : &b2_empty[s]);
          if (it == n_it - 1) umma_commit(out_done);
        }
        return true;
      };
      using I0 = std::integral_constant<int, 0>;
      using I1 = std::integral_constant<int, 1>;
      if (ok) ok = issue_xy(I0{}, 0);
      for (int it = 0; it < n_it && ok; it += 2) {
        ok = step(I0{}, I1{}, it);
        if (ok && it + 1 < n_it) ok = step(I1{}, I0{}, it + 1);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------------------------ compute: a row and 32 columns per thread
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int tid = threadIdx.x - 64;
    const int half = tid >> 7;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const bool row_ok = row < nrow;
    const float sl2 = a.scale * kLog2e;
    bool ok = true;
    float row_lse = INFINITY, row_delta = 0.f;
    int row_limit = 0;
    if constexpr (MODE == kWideDQ) {
      if (row_ok) {
        row_lse = a.lse[(int64_t)rhead * a.Tq + row0 + row] * kLog2e;
        row_delta = a.delta[(int64_t)rhead * a.Tq + row0 + row];
        row_limit = a.causal ? min(klen, diag0 + row) : klen;
      }
    }
    // dK, dV: the statistics belong to the streamed queries; they are fetched one iteration ahead and published in shared memory
    auto load_stats = [&](int it, float& l, float& d) {
      const int h = shead0 + it / per_head, qi = qs + (it % per_head) * kWideCols + tid;
      const bool v = qi < qlen;
      const int64_t at = (int64_t)h * a.Tq + (str0 - qs) + qi;
      l = v ? a.lse[at] * kLog2e : INFINITY;
      d = v && HAS_Y ? a.delta[at] : 0.f;
    };
    if constexpr (MODE != kWideDQ) {
      if (n_it > 0) {
        if (tid < kWideCols) load_stats(0, s_lse[tid], s_delta[tid]);
        mbar_arrive(stat_ready);
      }
    }
    const int key_idx = kk0 + row;
    const bool key_ok = row_ok && key_idx < klen;
    for (int it = 0; it < n_it && ok; ++it) {
      const int b = it & 1;
      const uint32_t ph = (it >> 1) & 1;
      float next_l = INFINITY, next_d = 0.f;
      const bool have_next = it + 1 < n_it;
      if constexpr (MODE != kWideDQ) {
        if (have_next && tid < kWideCols) load_stats(it + 1, next_l, next_d);
        if (!mbar_wait_bounded(stat_ready, it & 1, abort_flag, status, 4330)) { ok = false; break; }
      }
      if (!mbar_wait_bounded(&x_full[b], ph, abort_flag, status, 4300 + b)) { ok = false; break; }
      tc_fence_after();
      uint32_t x[32], y[32];
      tmem_ld_32x32(tX + lane_off + b * kWideCols + half * 32, x);
      if constexpr (HAS_Y) tmem_ld_32x32(tY + lane_off + b * kWideCols + half * 32, y);
      tmem_wait_ld();
      const int c0 = (it % per_head) * kWideCols + half * 32;     // first column: key index (dQ) or query index past qs (dK, dV)
      bool full;
      if constexpr (MODE == kWideDQ) full = c0 - half * 32 + kWideCols <= (a.causal ? min(klen, diag0) : klen);
      else full = nrow == 128 && kk0 + 128 <= klen && qs + c0 - half * 32 + kWideCols <= qlen && (!a.causal || kk0 + 127 <= qs + c0 - half * 32 + off);
      uint32_t w[16];
      auto columns = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float lv[4], dl[4], f[4];
          if constexpr (MODE == kWideDQ) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { lv[e] = row_lse; dl[e] = row_delta; }
          } else {
            const float4 l4 = *reinterpret_cast<const float4*>(s_lse + b * kWideCols + half * 32 + i);
            lv[0] = l4.x; lv[1] = l4.y; lv[2] = l4.z; lv[3] = l4.w;
            if constexpr (HAS_Y) {
              const float4 d4 = *reinterpret_cast<const float4*>(s_delta + b * kWideCols + half * 32 + i);
              dl[0] = d4.x; dl[1] = d4.y; dl[2] = d4.z; dl[3] = d4.w;
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float p = ex2(__uint_as_float(x[i + e]) * sl2 - lv[e]);
            if constexpr (decltype(masked)::value) {
              bool vis;
              if constexpr (MODE == kWideDQ) vis = c0 + i + e < row_limit;
              else {
                const int qi = qs + c0 + i + e;
                vis = key_ok && qi < qlen && (!a.causal || key_idx <= qi + off);
              }
              p = vis ? p : 0.f;
            }
            f[e] = HAS_Y ? p * (__uint_as_float(y[i + e]) - dl[e]) : p;
          }
          w[i >> 1] = pack_bf16x2(f[0], f[1]);
          w[(i >> 1) + 1] = pack_bf16x2(f[2], f[3]);
        }
      };
      if (full) columns(std::false_type{}); else columns(std::true_type{});
      tmem_st_32x16(tX + lane_off + b * kWideCols + half * 32, w);   // over this thread's own part of X
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&f_full[b]);
      if constexpr (MODE != kWideDQ) {
        if (have_next) {
          // every thread has passed this iteration's stat_ready wait, so nobody still reads the other buffer
          if (tid < kWideCols) {
            s_lse[(b ^ 1) * kWideCols + tid] = next_l;
            s_delta[(b ^ 1) * kWideCols + tid] = next_d;
          }
          mbar_arrive(stat_ready);
        }
      }
    }
    if (ok && n_it > 0) ok = mbar_wait_bounded(out_done, 0, abort_flag, status, 4320);
    if (ok) {
      tc_fence_after();
      const float osc = MODE == kWideDV ? 1.f : a.scale;
      const bool partial = MODE != kWideDQ && a.nsplit > 1;
      __nv_bfloat16* o16 = nullptr;
      float* o32 = nullptr;
      if (partial)
        o32 = a.part + ((((int64_t)(MODE == kWideDV) * a.nsplit + part_idx) * a.Tk + row0 + row) * a.Hkv + rhead) * kWideHD;
      else if (MODE == kWideDQ) o16 = a.dq + (int64_t)(row0 + row) * a.dq_stride + (int64_t)rhead * kWideHD;
      else if (MODE == kWideDK) o16 = a.dk + (int64_t)(row0 + row) * a.dk_stride + (int64_t)rhead * kWideHD;
      else o16 = a.dv + (int64_t)(row0 + row) * a.dv_stride + (int64_t)rhead * kWideHD;
#pragma unroll 1
      for (int c = half * 4; c < half * 4 + 4; ++c) {
        uint32_t r[32];
        if (n_it > 0) {
          tmem_ld_32x32(tOut + lane_off + c * 32, r);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (!row_ok) continue;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r[8 * v + i]) * osc;
          if (partial) {
            float4* d = reinterpret_cast<float4*>(o32 + c * 32 + v * 8);
            d[0] = make_float4(f[0], f[1], f[2], f[3]);
            d[1] = make_float4(f[4], f[5], f[6], f[7]);
          } else {
            reinterpret_cast<uint4*>(o16 + c * 32)[v] =
                make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

__global__ void __launch_bounds__(kWideThreads, 1)
attn_bwd_wide_kernel(const __grid_constant__ CUtensorMap q128, const __grid_constant__ CUtensorMap do128,
                     const __grid_constant__ CUtensorMap k128, const __grid_constant__ CUtensorMap v128,
                     const __grid_constant__ CUtensorMap q64, const __grid_constant__ CUtensorMap do64,
                     const __grid_constant__ CUtensorMap k64, const __grid_constant__ CUtensorMap v64, const WideArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) report_status(a.status, kStatusBadArgument, 4001, (int)(smem_u32(smem_raw) & 1023u));
    return;
  }
  const int n_kv = a.num_k_tiles * a.Hkv * a.nsplit, n_q = a.num_q_tiles * a.Hq;
  int b = blockIdx.x;
  if (b < n_kv) { wide_walk<kWideDK>(&k128, &v128, &q64, &do64, a, b, smem_raw); return; }
  b -= n_kv;
  if (b < n_q) { wide_walk<kWideDQ>(&q128, &do128, &k64, &v64, a, b, smem_raw); return; }
  wide_walk<kWideDV>(&k128, &v128, &q64, &do64, a, b - n_q, smem_raw);
}

// dk, dv [rows, 256] bf16 = the sums over the splits of a group, in a fixed order.
__global__ void __launch_bounds__(256) attn_wide_reduce_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ dk,
                                                               __nv_bfloat16* __restrict__ dv, int64_t dk_stride, int64_t dv_stride,
                                                               int nsplit, int64_t Tk, int Hkv) {
  const int64_t n = Tk * Hkv * (kWideHD / 8);          // 16-byte outputs of one gradient
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < 2 * n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool is_v = i >= n;
    const int64_t j = is_v ? i - n : i, t = j / (Hkv * (kWideHD / 8)), rest = j % (Hkv * (kWideHD / 8));
    const float* p = part + (int64_t)(is_v ? nsplit : 0) * n * 8 + j * 8;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < nsplit; ++s) {
      const float4 u = reinterpret_cast<const float4*>(p + s * n * 8)[0], w = reinterpret_cast<const float4*>(p + s * n * 8)[1];
      f[0] += u.x; f[1] += u.y; f[2] += u.z; f[3] += u.w; f[4] += w.x; f[5] += w.y; f[6] += w.z; f[7] += w.w;
    }
    __nv_bfloat16* o = is_v ? dv + t * dv_stride : dk + t * dk_stride;
    reinterpret_cast<uint4*>(o)[rest] = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
  }
}

int sm_count();   // gemm.cu

}  // namespace llmt

using namespace llmt;

// Into how many parts the query heads of a key/value group are split over CTAs (1, 2 or 4): a dK tile walks all query rows of
// all its heads, so few tiles leave the chip waiting for the longest of them; the parts meet in fp32 partial sums.
extern "C" int llmt_attn_bwd_wide_splits(int num_k_tiles, int Hq, int Hkv) {
  int n = 1;
  while (n < 4 && (Hq / Hkv) % (2 * n) == 0 && (int64_t)num_k_tiles * Hkv * n * 2 < 3 * sm_count()) n *= 2;
  return n;
}

// q, dout [Tq, Hq, 256], k, v [Tk, Hkv, 256]. q_tiles / k_tiles as for the other attention kernels (one pass: no two key tiles
// overlap). part: fp32 scratch of 2 * nsplit * Tk * Hkv * 256 floats when nsplit > 1 (every key row must then belong to a tile).
extern "C" int llmt_attn_bwd_wide(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse, float* delta,
                                  void* dq, void* dk, void* dv, float* part, int nsplit, const int* q_tiles, int num_q_tiles, const int* k_tiles,
                                  int num_k_tiles, int Tq, int Tk, int Hq, int Hkv, int64_t q_stride, int64_t k_stride, int64_t v_stride,
                                  int64_t o_stride, int64_t do_stride, int64_t dq_stride, int64_t dk_stride, int64_t dv_stride, float scale,
                                  int causal, int* status, cudaStream_t st) {
  if (Hq <= 0 || Tq <= 0 || Tk <= 0) return 0;
  if (Hq % Hkv || nsplit < 1 || (Hq / Hkv) % nsplit || (nsplit > 1 && part == nullptr) || (q_stride & 7) || (k_stride & 7) || (v_stride & 7) ||
      (do_stride & 7) || (dq_stride & 7) || (dk_stride & 7) || (dv_stride & 7))
    return -10;
  if (const int rc = launch_delta(o, o_stride, dout, do_stride, delta, nullptr, Tq, Hq, kWideHD, st)) return rc;
  CUtensorMap q128, do128, k128, v128, q64, do64, k64, v64;
  if (make_thd_map(&q128, q, Tq, Hq, kWideHD, q_stride) || make_thd_map(&do128, dout, Tq, Hq, kWideHD, do_stride) ||
      make_thd_map(&k128, k, Tk, Hkv, kWideHD, k_stride) || make_thd_map(&v128, v, Tk, Hkv, kWideHD, v_stride) ||
      make_thd_map(&q64, q, Tq, Hq, kWideHD, q_stride, kWideCols) || make_thd_map(&do64, dout, Tq, Hq, kWideHD, do_stride, kWideCols) ||
      make_thd_map(&k64, k, Tk, Hkv, kWideHD, k_stride, kWideCols) || make_thd_map(&v64, v, Tk, Hkv, kWideHD, v_stride, kWideCols))
    return -11;
  static bool cfg = false;
  if (!cfg) { if (set_smem(attn_bwd_wide_kernel, kWideSmem)) return -2; cfg = true; }
  WideArgs a{};
  a.lse = lse; a.delta = delta;
  a.dq = (__nv_bfloat16*)dq; a.dk = (__nv_bfloat16*)dk; a.dv = (__nv_bfloat16*)dv; a.part = part;
  a.q_tiles = q_tiles; a.k_tiles = k_tiles; a.num_q_tiles = num_q_tiles; a.num_k_tiles = num_k_tiles;
  a.Hq = Hq; a.Hkv = Hkv; a.Tq = Tq; a.Tk = Tk; a.nsplit = nsplit; a.causal = causal;
  a.dq_stride = dq_stride; a.dk_stride = dk_stride; a.dv_stride = dv_stride; a.scale = scale; a.status = status;
  const int64_t grid = 2 * (int64_t)num_k_tiles * Hkv * nsplit + (int64_t)num_q_tiles * Hq;
  if (grid > 0) attn_bwd_wide_kernel<<<(unsigned)grid, kWideThreads, kWideSmem, st>>>(q128, do128, k128, v128, q64, do64, k64, v64, a);
  if (nsplit > 1) {
    const int64_t n = 2 * (int64_t)Tk * Hkv * (kWideHD / 8), cap = (int64_t)sm_count() * 8;
    const int64_t blocks = (n + 255) / 256;
    attn_wide_reduce_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(part, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, dk_stride, dv_stride,
                                                                                     nsplit, Tk, Hkv);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
