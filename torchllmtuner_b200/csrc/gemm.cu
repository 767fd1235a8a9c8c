// Persistent bf16 GEMM for sm_100a: TMA -> shared memory (128B swizzle) -> tcgen05.mma with the fp32
// accumulator in TMEM -> tcgen05.ld epilogue. One kernel covers the three products of a linear layer
// (reference call sites: llmtuner/models/qwen/qwen3/model.py:255-268 via nn.Linear, and the packed
// expert products of llmtuner/models/common/moe/experts.py:206-209,268 via torch._grouped_mm):
//   forward  y  = x  * W^T   A K-major,  B K-major
//   dgrad    dx = dy * W     A K-major,  B MN-major
//   wgrad    dW = dy^T * x   A MN-major, B MN-major
// so no operand is ever transposed in memory. The grouped form runs the same tiles over row segments
// of A (one per expert, 128-row aligned) against a stack of B matrices.
//
// Warp 0 issues TMA, warp 1 owns TMEM and issues MMAs, the next 8 (4 beside comm warps) drain the accumulator.
// The accumulator is double buffered in TMEM so the epilogue of tile i overlaps the MMAs of tile i+1.
#include <type_traits>
#include "comm.cuh"
#include "kernels.h"

namespace llmt {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = one 128-byte swizzle row
// COMM: the form launched with a SideJob or a fused tensor-parallel collective: TMA warp, MMA warp, 4 epilogue warps and the
// comm warps. Without it 8 epilogue warps, two per tensor-memory lane quarter with half of the columns each: one warp per
// scheduler waits out every tensor-memory and shared-memory latency of a chunk by itself (0.45 us per 64 columns), which
// shows wherever the k-loop is short: expert weight gradients (K = rows of one expert), small products, the last tile.
template <bool COMM>
struct GemmRoles {
  static constexpr int kEpiWarps = COMM ? 4 : 8;
  static constexpr int kCommBase = 64 + 32 * kEpiWarps;                       // first comm thread
  static constexpr int kThreads = kCommBase + (COMM ? kCommThreads : 0);
};

// CG: CTAs that work on one tile. 1: a 128 x BN tile per CTA. 2: a 256 x BN tile per cluster of two CTAs (cta_group::2): each
// CTA loads its 128 rows of A and its half of the B tile, the tensor cores of both SMs read both halves of B, and each CTA's
// tensor memory receives its 128 rows of the product. See use_pair() for when which is used.
template <int CG, int BN, bool COMM>
struct GemmCfg {
  static constexpr int kBRows = BN / CG;           // rows of B that this CTA loads
  static constexpr int kStages = (kBRows == 256) ? 4 : 6;
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBBytes = kBRows * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kTmemCols = 2 * BN;  // two accumulators
  static constexpr int kEpiBytes = GemmRoles<COMM>::kEpiWarps * 4096;  // staging of the epilogue: 32 rows of 128 bytes per warp
  static constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + 1024 /*align slack*/ + 256 /*barriers*/;
};

struct GroupedArgs {
  const int* seg_offsets;  // [G+1] row offsets into A / C, each a multiple of BM; nullptr = plain GEMM
  int num_groups;
};

template <int CG, int BN, bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM, int MODE, bool COMM>
__global__ void __launch_bounds__(GemmRoles<COMM>::kThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    void* __restrict__ Cptr, int M, int N, int K, int64_t ldc, GroupedArgs grp, SideJob side, TPFuse tp, int* status) {
  using Cfg = GemmCfg<CG, BN, COMM>;
  using Roles = GemmRoles<COMM>;
  static_assert(!COMM || (CG == 1 && MODE == 0), "collectives ride on plain single-CTA products");
  static_assert(CG == 1 || MODE != 1, "segments are 128-row aligned: a 256-row tile would straddle them");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + Cfg::kStages * Cfg::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi + Cfg::kEpiBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + Cfg::kStages;
  uint64_t* tfull = bars + 2 * Cfg::kStages;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* comm_word = abort_flag + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // In a pair the CTA of rank 0 leads: its full[] barriers count the bytes of both CTAs' loads, it alone issues the products,
  // and its tempty[] barriers collect the epilogue threads of both. empty[] and tfull[] exist in both CTAs and are signalled
  // together by the leader's commits.
  const uint32_t rank = CG == 2 ? cluster_ctarank() : 0u;
  const int unit = blockIdx.x / CG, num_units = gridDim.x / CG;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], CG * 32 * Roles::kEpiWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (CG == 2) { tmem_alloc_pair(tmem_slot, Cfg::kTmemCols); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_slot, Cfg::kTmemCols); tmem_relinquish(); }
  }
  tc_fence_before();
  if constexpr (CG == 2) cluster_sync();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // Tile enumeration. Plain: tile -> (m = t % num_m, n = t / num_m). Grouped: m tiles walk the 128-row
  // aligned segments; the segment index selects the B matrix (third TMA coordinate).
  // MODE 0: plain. MODE 1: rows of A/C are 128-aligned segments, segment g uses B[g] (third TMA coordinate).
  // MODE 2: one M x N product per segment, reduced over that segment's rows (the K dimension); C[g] is M x N.
  constexpr bool GROUPED = (MODE == 1);
  const int num_n = (N + BN - 1) / BN;
  // MODE 1: M is the capacity of the padded row buffer (a multiple of BM); only the tiles below the last segment's end
  // hold rows, the rest of a statically sized buffer is skipped.
  constexpr int TM = BM * CG;                      // rows of a tile
  int num_m = (M + TM - 1) / TM;
  if constexpr (MODE == 1) {
    const int used = grp.seg_offsets[grp.num_groups] / BM;
    num_m = used < num_m ? used : num_m;
  }
  const int tiles_per_group = num_m * num_n;
  const int num_tiles = (MODE == 2) ? tiles_per_group * grp.num_groups : tiles_per_group;
  const int num_kb_plain = (K + BK - 1) / BK;
  auto kb_range = [&](int t, int& k_begin) -> int {
    if constexpr (MODE == 2) {
      const int g = t / tiles_per_group;
      k_begin = grp.seg_offsets[g];
      return (grp.seg_offsets[g + 1] - k_begin + BK - 1) / BK;
    } else {
      k_begin = 0;
      return num_kb_plain;
    }
  };

  // Tile order inside one M x N problem: super-rows of kGroupM m-tiles are swept column by column, so the CTAs that
  // run concurrently cover a near-square patch (A and B tiles are both reused out of L2).
  constexpr int kGroupM = 16 / CG;
  // With a fused tensor-parallel collective (MODE 0 only) the rows are walked chunk by chunk instead: the all-gather
  // form starts with this rank's own chunk, the reduce-scatter form ends with it.
  const bool tp_on = COMM && tp.mode != kTPNone;
  const int tp_mpc = tp_on ? tp.chunk_rows / BM : 1;
  const int tp_tpc = tp_mpc * num_n;
  auto tp_chunk_of = [&](int tt) -> int { return (tp.rank + tt / tp_tpc + (tp.mode == kTPReduceScatter ? 1 : 0)) % tp.world; };
  auto tile_mn = [&](int tt, int& m0, int& n0) {
    if (tp_on) {   // the same super-row sweep, inside one chunk
      const int w = tt % tp_tpc;
      const int per_group = kGroupM * num_n;
      const int grp_i = w / per_group;
      const int first_m = grp_i * kGroupM;
      const int gm = (tp_mpc - first_m < kGroupM) ? (tp_mpc - first_m) : kGroupM;
      const int r = w - grp_i * per_group;
      m0 = (tp_chunk_of(tt) * tp_mpc + first_m + r % gm) * BM;
      n0 = (r / gm) * BN;
      return;
    }
    const int per_group = kGroupM * num_n;
    const int grp_i = tt / per_group;
    const int first_m = grp_i * kGroupM;
    const int gm = (num_m - first_m < kGroupM) ? (num_m - first_m) : kGroupM;
    const int r = tt - grp_i * per_group;
    m0 = (first_m + r % gm) * TM + (int)rank * BM;        // this CTA's rows
    n0 = (r / gm) * BN;
  };

  auto group_of_row = [&](int row) -> int {
    // first segment that ends beyond `row`. A bisection: the producer thread looks it up for every tile, and a scan over 128
    // segments (one dependent load each) took longer than the tile's loads could run ahead.
    int lo = 0, hi = grp.num_groups - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (grp.seg_offsets[mid + 1] > row) hi = mid;
      else lo = mid + 1;
    }
    return lo;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t armed = 0, armed_parity = 0;  // per-stage bookkeeping for the abort drain
      bool ok = true;
      int landed_chunk = -1;
      for (int t = unit; t < num_tiles && ok; t += num_units) {
        int m0, n0;
        tile_mn(t % tiles_per_group, m0, n0);
        const int nb = n0 + (int)rank * Cfg::kBRows;        // this CTA's rows of the B tile
        if (tp_on && tp.mode == kTPAllGather) {
          const int c = tp_chunk_of(t);
          if (c != landed_chunk) {
            if (!tp_wait_landed(tp, c, abort_flag, status)) break;
            landed_chunk = c;
          }
        }
        int g = 0;
        if constexpr (GROUPED) g = group_of_row(m0);
        int k_begin;
        const int num_kb = kb_range(t, k_begin);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(&empty[stage], phase ^ 1, abort_flag, status, 100 + stage)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * Cfg::kStageBytes;
          uint8_t* sb = sa + Cfg::kABytes;
          if (rank == 0) {
            mbar_arrive_expect_tx(&full[stage], CG * Cfg::kStageBytes);
            armed |= 1u << stage;
            armed_parity = (armed_parity & ~(1u << stage)) | (phase << stage);
          }
          const int k0 = k_begin + kb * BK;
          if constexpr (CG == 2) {
            // a load of the second CTA may be counted before the leader has armed the phase: the transaction count may dip
            // below zero meanwhile, and the leader's own arrival keeps the phase from completing
            const uint32_t bar = cluster_map_u32(smem_u32(&full[stage]), 0);
            if constexpr (!A_MN) tma_load_2d_pair(sa, &tmA, bar, k0, m0);
            else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * (BK * 128), &tmA, bar, m0 + 64 * j, k0);
            }
            if constexpr (!B_MN) tma_load_2d_pair(sb, &tmB, bar, k0, nb);
            else {
#pragma unroll
              for (int j = 0; j < Cfg::kBRows / 64; ++j) tma_load_2d_pair(sb + j * (BK * 128), &tmB, bar, nb + 64 * j, k0);
            }
            if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
            continue;
          }
          if constexpr (!A_MN) {
            tma_load_2d(sa, &tmA, &full[stage], k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * (BK * 128), &tmA, &full[stage], m0 + 64 * j, k0);
          }
          if constexpr (!B_MN) {
            if constexpr (GROUPED) tma_load_3d(sb, &tmB, &full[stage], k0, n0, g);
            else tma_load_2d(sb, &tmB, &full[stage], k0, n0);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) {
              if constexpr (GROUPED) tma_load_3d(sb + j * (BK * 128), &tmB, &full[stage], n0 + 64 * j, k0, g);
              else tma_load_2d(sb + j * (BK * 128), &tmB, &full[stage], n0 + 64 * j, k0);
            }
          }
          if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (*abort_flag) {
        // Let copies that are still in flight land before this CTA's shared memory is released.
        for (int s = 0; s < Cfg::kStages; ++s) {
          if (!(armed & (1u << s))) continue;
          const uint32_t par = (armed_parity >> s) & 1u;
          for (uint32_t i = 0; i < (1u << 16); ++i)
            if (mbar_try_wait(&full[s], par)) break;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(TM, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int t = unit; t < num_tiles && ok; t += num_units) {
        if (!mbar_wait_bounded<CG == 2>(&tempty[acc], acc_phase ^ 1, abort_flag, status, 200 + acc)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        int k_begin;
        const int num_kb = kb_range(t, k_begin);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(&full[stage], phase, abort_flag, status, 300 + stage)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * Cfg::kStageBytes);
          const uint32_t sb = sa + Cfg::kABytes;
          const uint32_t la = desc_lo(sa, A_MN ? BK * 128 : 16), lb = desc_lo(sb, B_MN ? BK * 128 : 16);
          const uint32_t acc0 = kb ? 1u : 0u;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = desc_pack(la + (A_MN ? k * 128 : k * 2));
            const uint64_t db = desc_pack(lb + (B_MN ? k * 128 : k * 2));
            if constexpr (CG == 2) umma_bf16_ss_pair(d_tmem, da, db, idesc, k ? 1u : acc0);
            else umma_bf16_ss(d_tmem, da, db, idesc, k ? 1u : acc0);
          }
          // frees the stage (of both CTAs) once these MMAs have read it
          if constexpr (CG == 2) umma_commit_pair(&empty[stage]);
          else umma_commit(&empty[stage]);
          if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if constexpr (CG == 2) umma_commit_pair(&tfull[acc]);
        else umma_commit(&tfull[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (COMM && warp >= 2 + Roles::kEpiWarps) {
    // ------------------------------------------------------------------ comm warps (only launched with a SideJob)
    if (tp_on) {
      if (tp.mode == kTPAllGather) tp_allgather_comm(tp, threadIdx.x - Roles::kCommBase, comm_word, status);
      else tp_reducescatter_comm(tp, threadIdx.x - Roles::kCommBase, comm_word, status);
    } else {
      run_side_job(side, (long long)blockIdx.x * kCommThreads + (threadIdx.x - Roles::kCommBase), (long long)gridDim.x * kCommThreads, status);
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..)
    // A thread reads one row of the accumulator, so storing from registers touches 32 rows per instruction with 16 bytes each.
    // Every warp instead turns 32 rows x 128 bytes around in shared memory (16-byte chunks XORed with the row: no bank
    // conflicts) and writes, and when accumulating reads, whole 128-byte lines. What is added is added in fp32.
    const int quarter = warp & 3;  // TMEM lane quarter this warp may read
    constexpr int kCols = BN * 4 / Roles::kEpiWarps;       // columns of the tile that this warp drains, from col_w on
    const int col_w = ((warp - 2) >> 2) * kCols;
    uint8_t* stg = epi + (warp - 2) * 4096;
    constexpr int kOutBytes = OUT_F32 ? 4 : 2;
    constexpr bool kStageF32 = OUT_F32 || ACCUM;
    constexpr int kChunk = kStageF32 ? 32 : 64;            // columns per 128-byte staging row
    const bool vec_ok = ((reinterpret_cast<uintptr_t>(Cptr) | (uint64_t)(ldc * kOutBytes)) & 15) == 0;
    const int rr0 = lane >> 3, cc = lane & 7;              // this lane's row (of every 4) and 16-byte chunk when reading back
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = unit; t < num_tiles; t += num_units) {
      int m0, n0;
      tile_mn(t % tiles_per_group, m0, n0);
      const int row_limit = M;  // MODE 1: padded rows are written too (their inputs are zero)
      int k_begin;
      const bool empty_k = kb_range(t, k_begin) == 0;  // MODE 2 segment without rows: the product is zero
      const int64_t c_base = (MODE == 2) ? (int64_t)(t / tiles_per_group) * M * ldc : 0;
      const int row0 = m0 + quarter * 32;
      if constexpr (ACCUM) {        // fetch this warp's rows of C into L2 while their product is still being computed
        const int pr = min(row0 + lane, row_limit - 1);
        const uint8_t* line = reinterpret_cast<const uint8_t*>(Cptr) + (c_base + (int64_t)pr * ldc + n0 + col_w) * kOutBytes;
        for (int o = 0; o < min(kCols, N - n0 - col_w) * kOutBytes; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(line + o));
      }
      if (!mbar_wait_bounded(&tfull[acc], acc_phase, abort_flag, status, 400 + acc)) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN + col_w;
      const int n_chunks = (min(kCols, N - n0 - col_w) + kChunk - 1) / kChunk;   // <= 0: these columns lie outside
      const bool tile_vec = vec_ok && ((c_base * kOutBytes) & 15) == 0;
#pragma unroll 1
      for (int c = 0; c < n_chunks; ++c) {
        uint32_t r[kChunk];
        tmem_ld_32x32(t_row + c * kChunk, r);
        if constexpr (kChunk == 64) tmem_ld_32x32(t_row + c * kChunk + 32, r + 32);
        const int col0 = n0 + col_w + c * kChunk;
        if (tile_vec && (N & 7) == 0) {
          constexpr int kPer = kStageF32 ? 4 : 8;          // columns per 16 staged bytes
          const int col = col0 + cc * kPer;
          const bool col_ok = col < N;
          const int64_t at = c_base + (int64_t)(row0 + rr0) * ldc + col;
          using OldT = typename std::conditional<OUT_F32, uint4, uint2>::type;
          OldT old[8];                                     // what the product is added to: raw, converted where it is used
          if constexpr (ACCUM) {
            // clamped instead of skipped: eight unconditional loads are in flight together, a branch around each would
            // leave them one after another
            const int64_t cat = c_base + (col_ok ? col : n0);   // n0 < N
#pragma unroll
            for (int it = 0; it < 8; ++it)
              old[it] = *reinterpret_cast<const OldT*>(reinterpret_cast<const uint8_t*>(Cptr) +
                                                       (cat + (int64_t)min(row0 + rr0 + it * 4, row_limit - 1) * ldc) * kOutBytes);
          }
          tmem_wait_ld();
          if (empty_k) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) r[j] = 0u;
          }
          if constexpr (!kStageF32) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = pack_bf16x2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          }
          __syncwarp();                                    // the previous chunk has been read back by every lane
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int rr = it * 4 + rr0;
            uint4 v = *reinterpret_cast<const uint4*>(stg + rr * 128 + ((cc ^ (rr & 7)) << 4));
            if (!(col_ok && row0 + rr < row_limit)) continue;
            if constexpr (kStageF32) {
              float4 o = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
              if constexpr (ACCUM && OUT_F32) {
                o.x += __uint_as_float(old[it].x); o.y += __uint_as_float(old[it].y);
                o.z += __uint_as_float(old[it].z); o.w += __uint_as_float(old[it].w);
              } else if constexpr (ACCUM) {
                const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&old[it].x));
                const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&old[it].y));
                o.x += a.x; o.y += a.y; o.z += b.x; o.w += b.y;
              }
              if constexpr (OUT_F32) {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(Cptr) + at + (int64_t)it * 4 * ldc) = o;
              } else {
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(Cptr) + at + (int64_t)it * 4 * ldc) =
                    make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w));
              }
            } else {
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(Cptr) + at + (int64_t)it * 4 * ldc) = v;
            }
          }
        } else {                                           // outputs off a 16-byte boundary, widths that are no multiple of 8
          tmem_wait_ld();
          const int row = row0 + lane;
          if (row < row_limit) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
              if (col0 + j >= N) break;
              const int64_t at = c_base + (int64_t)row * ldc + col0 + j;
              float o = empty_k ? 0.f : __uint_as_float(r[j]);
              if constexpr (OUT_F32) {
                float* dst = reinterpret_cast<float*>(Cptr) + at;
                if constexpr (ACCUM) o += *dst;
                *dst = o;
              } else {
                __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(Cptr) + at;
                if constexpr (ACCUM) o += __bfloat162float(*dst);
                *dst = __float2bfloat16_rn(o);
              }
            }
          }
        }
      }
      tc_fence_before();
      if constexpr (CG == 2) mbar_arrive_cluster(cluster_map_u32(smem_u32(&tempty[acc]), 0));
      else mbar_arrive(&tempty[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      if (tp_on && tp.mode == kTPReduceScatter) tp_tile_done(tp, tp_chunk_of(t), (uint32_t)tp_tpc * 4u, lane);
    }
  }

  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync();   // neither CTA leaves while the other's products or barriers still refer to it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CG == 2) tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
    else tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// ---------------------------------------------------------------------------------------------
// host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) return (EncodeTiledFn) nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// bf16 tensor map with a 128-byte swizzle. dims/strides are innermost-first; strides in bytes for dims 1..rank-1.
int make_tmap_typed(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                    const uint32_t* box, int is_f32);
int make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                   const uint32_t* box) {
  return make_tmap_typed(out, base, rank, dims, strides_bytes, box, 0);
}
// Same for fp32 elements when `is_f32` (inner box of at most 32 elements = one 128-byte swizzle row).
int make_tmap_typed(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                    const uint32_t* box, int is_f32) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return -1;
  // The encoder is a driver call and needs the primary context bound to the calling thread; a fresh thread (the
  // autograd engine's) has none until its first runtime call.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(nullptr);
    ctx_bound = true;
  }
  cuuint64_t gdim[5], gstr[5];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i > 0) gstr[i - 1] = strides_bytes[i - 1];
  }
  CUresult r = enc(out, is_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr, bx, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (r == CUDA_SUCCESS) ? 0 : (int)r;
}

int sm_count() {
  static int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  return n;
}

// Whether a plain product takes pair tiles (256 x 256 on two SMs) or single ones (128 x 256 on one). Both give an SM the same
// share of a full wave, so the one with fewer waves wins; at equal waves the pair is the faster one, because each SM reads
// 8 KB instead of 12 KB of shared memory per 128 clocks of tensor work (single tiles measured 1.06 to 1.3 times the time:
// 8192 x 12288 x 4096 504 us against 541 us, 8192 x 4096 x 4096 164 against 216, cuBLAS 529 and 176). At most 128 rows leave
// the second CTA without work.
static bool use_pair(int64_t M, int64_t N, int max_ctas) {
  if (M <= BM || max_ctas == 1) return false;
  const int64_t sms = sm_count(), n = (N + 255) / 256;
  const int64_t pair = ((M + 255) / 256 * n + sms / 2 - 1) / (sms / 2), single = ((M + 127) / 128 * n + sms - 1) / sms;
  return 100 * pair <= 107 * single;
}

template <int CG, int BN, bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM, int MODE, bool COMM = false>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, int64_t ldc, GroupedArgs grp,
                  int* status, int max_ctas, cudaStream_t stream, const SideJob* side = nullptr, const TPFuse* tpf = nullptr) {
  const bool with_tp = tpf != nullptr && tpf->mode != kTPNone;
  const bool with_side = (side != nullptr && side->kind != kSideNone) || with_tp;
  if constexpr (CG == 1 && MODE == 0 && !COMM)
    if (with_side)
      return launch<CG, BN, A_MN, B_MN, OUT_F32, ACCUM, MODE, true>(ta, tb, C, M, N, K, ldc, grp, status, max_ctas, stream, side, tpf);
  using Cfg = GemmCfg<CG, BN, COMM>;
  constexpr int kThreads = GemmRoles<COMM>::kThreads;
  auto kern = gemm_tcgen05_kernel<CG, BN, A_MN, B_MN, OUT_F32, ACCUM, MODE, COMM>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) return -2;
    configured = true;
  }
  const int tiles = ((M + BM * CG - 1) / (BM * CG)) * ((N + BN - 1) / BN) * (MODE == 2 ? grp.num_groups : 1);
  int grid = tiles < sm_count() / CG ? tiles : sm_count() / CG;
  if (max_ctas > 0 && grid > max_ctas / CG) grid = max_ctas / CG;
  if (grid < 1) return 0;
  if constexpr (CG == 2) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid * 2);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, ta, tb, C, M, N, K, ldc, grp, SideJob{}, TPFuse{}, status) == cudaSuccess ? 0 : -3;
  }
  SideJob none{};
  TPFuse no_tp{};
  if (with_side && max_ctas <= 0) grid = sm_count();   // every SM carries comm warps, even past the last tile
  kern<<<grid, kThreads, Cfg::kSmemBytes, stream>>>(
      ta, tb, C, M, N, K, ldc, grp, (side != nullptr && !with_tp) ? *side : none, with_tp ? *tpf : no_tp, status);
  return (cudaGetLastError() == cudaSuccess) ? 0 : -3;
}

template <int CG, int BN>
static int dispatch_plain(bool a_mn, bool b_mn, bool out_f32, bool accum, const CUtensorMap& ta, const CUtensorMap& tb,
                          void* C, int M, int N, int K, int64_t ldc, int* status, int max_ctas, cudaStream_t s,
                          const SideJob* side, const TPFuse* tpf = nullptr) {
  GroupedArgs grp{nullptr, 0};
#define LLMT_CASE(AM, BMN, F32, ACC)                                                            \
  if (a_mn == AM && b_mn == BMN && out_f32 == F32 && accum == ACC)                              \
    return launch<CG, BN, AM, BMN, F32, ACC, 0>(ta, tb, C, M, N, K, ldc, grp, status, max_ctas, s, side, tpf);
  LLMT_CASE(false, false, false, false)
  LLMT_CASE(false, false, true, false)
  LLMT_CASE(false, true, false, false)
  LLMT_CASE(false, true, true, false)
  LLMT_CASE(false, true, false, true)
  LLMT_CASE(true, true, false, false)
  LLMT_CASE(true, true, true, false)
  LLMT_CASE(true, true, false, true)
  LLMT_CASE(true, true, true, true)
#undef LLMT_CASE
  return -4;  // combination not instantiated
}

}  // namespace llmt

using namespace llmt;

// C[M,N] (+)= A * B with bf16 inputs and fp32 accumulation.
//   a_mn == 0: A stored [M][K] (row stride lda elements); a_mn == 1: A stored [K][M].
//   b_mn == 0: B stored [N][K] (row stride ldb);          b_mn == 1: B stored [K][N].
// Requirements: base pointers 16-byte aligned, lda/ldb multiples of 8 elements.
static int gemm_impl(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc, int a_mn,
                     int b_mn, int out_f32, int accumulate, int* status, int max_ctas, cudaStream_t stream, const SideJob* side,
                     const TPFuse* tpf = nullptr) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (lda & 7) || (ldb & 7) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -10;
  const bool bn256 = N > 128;
  const bool fused = (side != nullptr && side->kind != kSideNone) || (tpf != nullptr && tpf->mode != kTPNone);
  const bool pair = bn256 && !fused && use_pair(M, N, max_ctas);
  const uint32_t bn = bn256 && !pair ? 256 : 128;          // rows of B per load
  CUtensorMap ta, tb;
  {
    uint64_t dims[2], str[1];
    uint32_t box[2];
    if (!a_mn) { dims[0] = K; dims[1] = M; box[0] = 64; box[1] = BM; }
    else       { dims[0] = M; dims[1] = K; box[0] = 64; box[1] = BK; }
    str[0] = (uint64_t)lda * 2;
    if (int rc = make_tmap_bf16(&ta, A, 2, dims, str, box)) return -1100 - rc;
    if (!b_mn) { dims[0] = K; dims[1] = N; box[0] = 64; box[1] = bn; }
    else       { dims[0] = N; dims[1] = K; box[0] = 64; box[1] = BK; }
    str[0] = (uint64_t)ldb * 2;
    if (make_tmap_bf16(&tb, B, 2, dims, str, box)) return -12;
  }
  if (pair) return dispatch_plain<2, 256>(a_mn, b_mn, out_f32, accumulate, ta, tb, C, M, N, K, ldc, status, max_ctas, stream, nullptr);
  if (bn256) return dispatch_plain<1, 256>(a_mn, b_mn, out_f32, accumulate, ta, tb, C, M, N, K, ldc, status, max_ctas, stream, side, tpf);
  return dispatch_plain<1, 128>(a_mn, b_mn, out_f32, accumulate, ta, tb, C, M, N, K, ldc, status, max_ctas, stream, side, tpf);
}

extern "C" int llmt_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                              int64_t ldc, int a_mn, int b_mn, int out_f32, int accumulate, int* status, int max_ctas,
                              cudaStream_t stream) {
  return gemm_impl(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_f32, accumulate, status, max_ctas, stream, nullptr);
}

// Same product, with a slice of a peer-memory collective carried by the comm warps of every CTA (see comm.cuh).
extern "C" int llmt_gemm_bf16_fused(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                                    int64_t ldc, int a_mn, int b_mn, int out_f32, int accumulate, int job_kind, int job_nsrc,
                                    const void* const* job_src, void* job_dst, long long job_n, int job_accumulate,
                                    const uint32_t* wait_flags, int n_wait, uint32_t wait_value, int* status,
                                    cudaStream_t stream) {
  SideJob j{};
  j.kind = job_kind;
  j.nsrc = job_nsrc;
  for (int i = 0; i < kMaxPeers; ++i) j.src[i] = (i < job_nsrc) ? job_src[i] : nullptr;
  j.dst = job_dst;
  j.n = job_n;
  j.accumulate = job_accumulate;
  j.wait_flags = wait_flags;
  j.n_wait = n_wait;
  j.wait_value = wait_value;
  if (job_kind != kSideNone && (job_nsrc < 1 || job_nsrc > kMaxPeers)) return -10;
  return gemm_impl(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_f32, accumulate, status, 0, stream, &j);
}

// Tensor-parallel fused forms (see comm.cuh). mode 1: C[M,N] = gather(A) * B where `A` is the local gathered matrix
// [M,K] that the comm warps fill from `peer_src` (every rank's chunk); mode 2: `C` is this rank's symmetric bf16 partial
// matrix [M,N] (ldc == N), `out` [M/world, N] receives the reduced chunk (+ residual). A is row-major in both.
// `accumulate` (only with b_mn) adds the product to what C already holds before the partial is published.
extern "C" int llmt_gemm_bf16_tp(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                                 int64_t ldc, int b_mn, int accumulate, int mode, int world, int rank, uint32_t epoch,
                                 const void* const* peer_src, const uint32_t* flags, uint32_t* const* peer_flags,
                                 uint32_t* counters, float* acc, void* out, const void* residual, int* status,
                                 cudaStream_t stream) {
  if (world < 2 || world > kMaxPeers || rank < 0 || rank >= world || M % world) return -10;
  const int chunk_rows = M / world;
  if (chunk_rows % BM || (mode != kTPAllGather && mode != kTPReduceScatter)) return -10;
  if (mode == kTPReduceScatter && (ldc != N || (N & 7))) return -10;
  if (mode == kTPAllGather && lda != K) return -10;
  TPFuse t{};
  t.mode = mode; t.world = world; t.rank = rank; t.chunk_rows = chunk_rows; t.epoch = epoch;
  for (int i = 0; i < world; ++i) { t.peer_src[i] = peer_src[i]; t.peer_flags[i] = peer_flags[i]; }
  t.local_dst = const_cast<void*>(A);
  t.chunk_bytes = (long long)chunk_rows * K * 2;
  t.flags = flags; t.counters = counters;
  t.acc = acc; t.out = reinterpret_cast<__nv_bfloat16*>(out); t.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  t.n_cols = N;
  return gemm_impl(A, B, C, M, N, K, lda, ldb, ldc, 0, b_mn, 0, accumulate, status, 0, stream, nullptr, &t);
}

// Grouped forward/dgrad: rows of A (and C) are cut into `num_groups` segments at seg_offsets (device int32,
// [G+1], multiples of 128, seg_offsets[G] == M_padded); segment g multiplies B[g].
//   b_mn == 0: B stored [G][N][K];  b_mn == 1: B stored [G][K][N] (with `accumulate`: C += ..., added in fp32).
extern "C" int llmt_grouped_gemm_bf16(const void* A, const void* B, void* C, const int* seg_offsets, int num_groups,
                                      int M_padded, int N, int K, int64_t lda, int64_t ldc, int b_mn, int out_f32, int accumulate,
                                      int* status, cudaStream_t stream) {
  if (M_padded <= 0 || N <= 0 || num_groups <= 0) return 0;
  if (K <= 0 || (lda & 7) || (M_padded % BM) || (reinterpret_cast<uintptr_t>(A) & 15)) return -10;
  const bool bn256 = N > 128;
  const uint32_t bn = bn256 ? 256 : 128;
  CUtensorMap ta, tb;
  {
    uint64_t dims[3], str[2];
    uint32_t box[3];
    dims[0] = K; dims[1] = M_padded; box[0] = 64; box[1] = BM;
    str[0] = (uint64_t)lda * 2;
    if (int rc = make_tmap_bf16(&ta, A, 2, dims, str, box)) return -1100 - rc;
    if (!b_mn) { dims[0] = K; dims[1] = N; box[0] = 64; box[1] = bn; str[0] = (uint64_t)K * 2; }
    else       { dims[0] = N; dims[1] = K; box[0] = 64; box[1] = BK; str[0] = (uint64_t)N * 2; }
    dims[2] = num_groups; box[2] = 1;
    str[1] = (uint64_t)N * K * 2;
    if (make_tmap_bf16(&tb, B, 3, dims, str, box)) return -12;
  }
  GroupedArgs grp{seg_offsets, num_groups};
  if (out_f32 || (accumulate && !b_mn)) return -4;
  if (accumulate) {                                    // dx += dy_i W_i of a second projection of the same rows
    if (bn256) return launch<1, 256, false, true, false, true, 1>(ta, tb, C, M_padded, N, K, ldc, grp, status, 0, stream);
    return launch<1, 128, false, true, false, true, 1>(ta, tb, C, M_padded, N, K, ldc, grp, status, 0, stream);
  }
  if (bn256) {
    if (b_mn) return launch<1, 256, false, true, false, false, 1>(ta, tb, C, M_padded, N, K, ldc, grp, status, 0, stream);
    return launch<1, 256, false, false, false, false, 1>(ta, tb, C, M_padded, N, K, ldc, grp, status, 0, stream);
  }
  if (b_mn) return launch<1, 128, false, true, false, false, 1>(ta, tb, C, M_padded, N, K, ldc, grp, status, 0, stream);
  return launch<1, 128, false, false, false, false, 1>(ta, tb, C, M_padded, N, K, ldc, grp, status, 0, stream);
}

// Grouped wgrad: C[g] (M x N, row stride N) (+)= A_g^T * B_g where A is stored [rows][M], B is stored [rows][N] and
// segment g covers rows [seg_offsets[g], seg_offsets[g+1]) (multiples of 128; padded rows must hold zeros).
extern "C" int llmt_grouped_wgrad_bf16(const void* A, const void* B, void* C, const int* seg_offsets, int num_groups,
                                       int rows_padded, int M, int N, int64_t lda, int64_t ldb, int out_f32,
                                       int accumulate, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || num_groups <= 0) return 0;
  if ((lda & 7) || (ldb & 7) || (rows_padded % BM) || rows_padded <= 0) return -10;
  const bool bn256 = N > 128;
  CUtensorMap ta, tb;
  {
    uint64_t dims[2], str[1];
    uint32_t box[2];
    dims[0] = M; dims[1] = rows_padded; box[0] = 64; box[1] = BK; str[0] = (uint64_t)lda * 2;
    if (int rc = make_tmap_bf16(&ta, A, 2, dims, str, box)) return -1100 - rc;
    dims[0] = N; dims[1] = rows_padded; box[0] = 64; box[1] = BK; str[0] = (uint64_t)ldb * 2;
    if (make_tmap_bf16(&tb, B, 2, dims, str, box)) return -12;
  }
  GroupedArgs grp{seg_offsets, num_groups};
  const int K = rows_padded;      // single-CTA tiles: with the few k-blocks of one expert the pair form measured slower (164 us
                                  // against 141 us per 128 x 768 x 2048 gradient over 32768 rows, 62 us to write it)
#define LLMT_W(BNV, F32, ACC) \
  if (bn256 == (BNV == 256) && (bool)out_f32 == F32 && (bool)accumulate == ACC) \
    return launch<1, BNV, true, true, F32, ACC, 2>(ta, tb, C, M, N, K, (int64_t)N, grp, status, 0, stream);
  LLMT_W(256, false, false) LLMT_W(256, true, false) LLMT_W(256, false, true) LLMT_W(256, true, true)
  LLMT_W(128, false, false) LLMT_W(128, true, false) LLMT_W(128, false, true) LLMT_W(128, true, true)
#undef LLMT_W
  return -4;
}
