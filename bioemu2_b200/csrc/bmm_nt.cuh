// Batched C[b] = scale * A[b] * B[b]^T with both operands K-major bf16, fp32
// accumulation in tensor memory and bf16 output.
//
// This is the per-channel contraction of triangle multiplication
// (t[d][i][j] = sum_k a[d][i][k] * b[d][j][k]) and the MSA-depth contraction of
// the outer product mean.  Persistent kernel, one CTA per SM:
//   warp 0      TMA producer   (A and B K-slabs of 64 through a shared-memory ring)
//   warp 1      MMA issuer     (tcgen05.mma 128 x BN x 16, two accumulator buffers in TMEM)
//   warps 2..5  epilogue       (TMEM -> registers -> bf16 -> global)
#pragma once
#include <climits>

#include "row_tile.cuh"

namespace b200 {

struct BmmParams {
  void* C;                   // bf16, or fp32 when out_f32
  long long c_batch_stride;  // elements
  int ldc;                   // elements
  int m_valid, n_valid;      // rows / columns of C that exist (n_valid % 8 == 0)
  int tiles_m, tiles_n, batch;
  int k_blocks;              // K / 64, rounded up (TMA zero-fills the tail)
  float scale;
  const float* scale_ptr;    // optional per-batch device scalar multiplied into scale
  const float* bias;         // optional per-column bias added after scaling
  int out_f32;
  // Outer-product store: with opm_ntok > 0, C row r = (i, c) and column q = (j, d) (c, d < 32) go to
  // C[((i * opm_ntok + j) * 32 + c) * 32 + d]: every pair (i, j) gets its 32x32 outer product contiguous.
  int opm_ntok;
  // With residual != nullptr the value read from it at the destination offset is added.
  const void* residual;
  // Bulk output: the scaled (+ bias) tile leaves through 16 KB staging tiles ([128 rows][128 B]: 32 fp32 or 64
  // bf16 columns) and the C tensor map, 1 = stored, 2 = added into C (the residual is C itself, which the
  // epilogue then never reads), 3 = stored with the rows as groups of 32, {column, row in group, group, batch}.
  int tma_c;
  // Split operands stored once as (hi | lo): a K block at or past the fold is loaded from that many blocks before, which
  // makes the operand hi | hi | lo.  INT_MAX: none.
  int a_fold, b_fold;
  // Operands stored as hi and lo planes part_batch batch slices apart, each part_blocks K blocks wide: A is read hi, hi, lo,
  // B hi, lo, hi.  0: none.
  int part_blocks, part_batch;
  // kEpiGateSplit: row r of A is pair (line, pos) = (r / mask_pitch, r % mask_pitch), kept where pos < mask_n and
  // mask[line * mask_line + pos * mask_pos] != 0.
  const uint8_t* mask;
  int mask_pitch, mask_n;
  long long mask_line, mask_pos;
  int a_shared, b_shared;    // 1: every batch item multiplies the same A / B (its tensor map has a single batch slice)
};

// The epilogues are separate instantiations: with all of them in one kernel the plain one, which triangle multiplication's
// contraction lives on, took 27.8 us instead of 21.7 at N = 384.
enum BmmEpilogue : int {
  kEpiDirect = 0,  // scale, bias, residual; stores by the threads themselves
  kEpiBulk = 1,    // scale, bias; bulk stores through C's tensor map
  // Bulk, the tile multiplied element by element with fp32 factors (a per-token gate) before it is stored or added.  They
  // come by TMA during the product's K loop (read by the lanes from their rows: 16 against 9 us without the gate for
  // 2048 x 768 x 768, 23 against 13 for K = 3072).
  kEpiMul = 2,
  kEpiAdd = 6,     // the same with addends of C's type: an fp32 residual that is not C itself, or a bf16 C that is to be rounded once
  kEpiSwiglu = 3,  // bulk bf16: the columns are pairs of 64-column blocks (a | b), C gets silu(a) * b, half as many columns
  kEpiSwigluSplit = 4,  // the same from split operands: C gets (hi | lo) of silu(a) * b, see kEpiGateSplit
  // kEpiBulk with eight epilogue warps, each group of four draining half of the tile's columns: a short product's tile is
  // its epilogue (K = 128: 2 K blocks of 64 against 128 columns of TMEM reads, staging and stores a lane).
  kEpiBulkWide = 7,
  // Gated operands of the accurate triangle contraction, from split operands: the weights' 256 rows are p and g of 128
  // channels and take the M side, so a lane is a channel and its columns are consecutive pairs -- the order in which the
  // contraction reads them.  C gets hi and lo of p * sigmoid(g) (masked pairs zero) as rows part *
  // 128 + channel of column tile tn.  (Projection to fp32 and a gate kernel over it: 26 + 33 us for 40000 pairs.)  Both split
  // epilogues keep fp32: expf and the refined quotient.  Transition of 40000 rows / triangle multiplication of 200 tokens, us:
  // with the compiler's division, whose rare cases are a branch per value, 98 / 117, refined 82 / 108, with the hardware's
  // exponential and reciprocal alone 79 / 104 (a rounded argument costs the exponential 2^-18 of its value at 64).
  kEpiGateSplit = 8,
  kEpiOuter = 5,   // outer products of 32 x 32, one pair's 2 KB in one piece
};

template <int EPI>
inline constexpr bool kTwoGroups = EPI == kEpiSwigluSplit || EPI == kEpiBulkWide || EPI == kEpiGateSplit;
template <int EPI>
inline constexpr bool kBulk = EPI == kEpiBulk || EPI == kEpiBulkWide;
template <int EPI>
inline constexpr bool kTileOperand = EPI == kEpiMul || EPI == kEpiAdd;

template <int BN, int EPI>
struct BmmCfg {
  static constexpr int BM = 128;
  static constexpr int BK = 64;
  static constexpr int STAGES = kTwoGroups<EPI> ? (BN == 256 ? 3 : 5) : kTileOperand<EPI> || BN == 256 ? 4 : 6;
  static constexpr uint32_t A_BYTES = BM * BK * 2;
  static constexpr uint32_t B_BYTES = BN * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr uint32_t MUL_OFFSET = STAGES * STAGE_BYTES;     // the factors' or addends' [128 rows][32 columns] tiles
  static constexpr uint32_t MUL_BYTES = kTileOperand<EPI> ? BN * 128 * 4 : 0;
  static constexpr uint32_t BAR_OFFSET = MUL_OFFSET + MUL_BYTES;
  static constexpr uint32_t BIAS_OFFSET = BAR_OFFSET + 1024;       // the tile's BN bias values
  static constexpr uint32_t OUT_OFFSET = BAR_OFFSET + 2048;        // [128 rows][128 B] tiles for bulk output
  static constexpr int OUT_TILES = kTwoGroups<EPI> ? 4 : 2;
  static constexpr uint32_t SMEM_BYTES = OUT_OFFSET + OUT_TILES * 16384 + 1024;  // + alignment slack
  // The split SwiGLU's arithmetic keeps four warps busy for longer than the product (40000 x 1024 x 384: 105 us): it
  // has eight, each group of four with one of the tile's two 64-column groups.
  static constexpr int EPI_THREADS = kTwoGroups<EPI> ? 256 : 128;
  static constexpr int GROUPS = EPI_THREADS / 128;
  static constexpr int THREADS = 64 + EPI_THREADS;
};

template <int BN, int EPI>
__global__ void __launch_bounds__(BmmCfg<BN, EPI>::THREADS, 1)
bmm_nt_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
              const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmM, BmmParams p) {
  using Cfg = BmmCfg<BN, EPI>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFFSET);
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* acc_full = empty + Cfg::STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* mul_full = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mul_full + 1);
  float* bias_s = reinterpret_cast<float*>(smem + Cfg::BIAS_OFFSET);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int tiles_per_batch = p.tiles_m * p.tiles_n;
  const int total_tiles = tiles_per_batch * p.batch;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], Cfg::EPI_THREADS);
    }
    mbar_init(mul_full, 1);
    fence_mbar_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
    if (EPI != kEpiDirect && EPI != kEpiOuter) prefetch_tmap(&tmC);
    if (kTileOperand<EPI>) prefetch_tmap(&tmM);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
        const int b = tile / tiles_per_batch;
        const int rem = tile - b * tiles_per_batch;
        const int tm = rem / p.tiles_n;
        const int tn = rem - tm * p.tiles_n;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          mbar_wait(&empty[stage], phase ^ 1, 1);
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          mbar_arrive_expect_tx(&full[stage], Cfg::STAGE_BYTES);
          int ka = kb < p.a_fold ? kb : kb - p.a_fold, kbb = kb < p.b_fold ? kb : kb - p.b_fold;
          int ab = p.a_shared ? 0 : b, bb = p.b_shared ? 0 : b;
          if (p.part_blocks > 0) {
            const int part = kb / p.part_blocks;
            ka = kbb = kb - part * p.part_blocks;
            if (part == 2) ab += p.part_batch;
            if (part == 1) bb += p.part_batch;
          }
          tma_load_3d(sa, &tmA, &full[stage], ka * 64, tm * 128, ab);
          tma_load_3d(sa + Cfg::A_BYTES, &tmB, &full[stage], kbb * 64, tn * BN, bb);
          if (++stage == Cfg::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the tile and K loops and waits on the barriers; one elected lane issues the products and
    // the commits (a converged warp issues a tcgen05.mma several times faster than a lone thread of a diverged one).
    {
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(128, EPI == kEpiGateSplit ? 128 : BN);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it) {
        const int acc = it & 1;
        mbar_wait(&acc_empty[acc], ((it >> 1) & 1) ^ 1, 2);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          mbar_wait(&full[stage], phase, 3);
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t sb = sa + Cfg::A_BYTES;
          const uint32_t a_lo = desc_lo(sa), b_lo = desc_lo(sb);
          if (leader) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if constexpr (EPI == kEpiGateSplit) {
                umma_bf16_ss2(d_tmem, b_lo + 2 * k, kDescHiSw128, a_lo + 2 * k, kDescHiSw128, idesc, (kb | k) != 0);
                umma_bf16_ss2(d_tmem + 128, b_lo + 1024 + 2 * k, kDescHiSw128, a_lo + 2 * k, kDescHiSw128, idesc, (kb | k) != 0);
              } else {
                umma_bf16_ss2(d_tmem, a_lo + 2 * k, kDescHiSw128, b_lo + 2 * k, kDescHiSw128, idesc, (kb | k) != 0);
              }
            }
            umma_commit(&empty[stage]);
          }
          __syncwarp();
          if (++stage == Cfg::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (leader) umma_commit(&acc_full[acc]);
        __syncwarp();
      }
    }
  } else {
    const int quarter = warp & 3;  // TMEM lanes this warp may read: 32*quarter .. +31
    int it = 0;
    auto load_factors = [&](int tile) {
      const int rem = tile % tiles_per_batch;
      const int tm = rem / p.tiles_n, tn = rem - tm * p.tiles_n;
      if (EPI == kEpiAdd && !p.out_f32) {  // [128 rows][64 columns] of C itself
        mbar_arrive_expect_tx(mul_full, Cfg::MUL_BYTES / 2);
#pragma unroll
        for (int c = 0; c < BN / 64; ++c)
          tma_load_3d(smem + Cfg::MUL_OFFSET + c * 16384, &tmM, mul_full, tn * BN + c * 64, tm * 128, tile / tiles_per_batch);
        return;
      }
      mbar_arrive_expect_tx(mul_full, Cfg::MUL_BYTES);
#pragma unroll
      for (int c = 0; c < BN / 32; ++c)
        tma_load_2d(smem + Cfg::MUL_OFFSET + c * 16384, &tmM, mul_full, tn * BN + c * 32, tm * 128);
    };
    if (kTileOperand<EPI> && threadIdx.x == 64 && int(blockIdx.x) < total_tiles) load_factors(blockIdx.x);
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it) {
      const int b = tile / tiles_per_batch;
      const int rem = tile - b * tiles_per_batch;
      const int tm = rem / p.tiles_n;
      const int tn = rem - tm * p.tiles_n;
      const int acc = it & 1;
      const int grp = Cfg::GROUPS == 1 ? 0 : (warp - 2) >> 2;
      constexpr int GCOLS = BN / Cfg::GROUPS;            // columns a group drains
      if ((kBulk<EPI> || kTileOperand<EPI>) && p.bias) {
        // Read by every lane from shared memory (by every lane from global memory: 25 against 17 us without a bias for
        // 2048 x 4608 x 768).  The previous tile's values have been read before its last barrier; the first barrier
        // of this one makes the new ones visible.
#pragma unroll
        for (int i = 0; i < GCOLS; i += 128) {
          const int k = grp * GCOLS + i + quarter * 32 + lane, col = tn * BN + k;
          if (GCOLS >= 128 || quarter * 32 < GCOLS) bias_s[k] = col < p.n_valid ? p.bias[col] : 0.f;
        }
      }
      uint32_t keep[2];  // kEpiGateSplit: bit j = column j of the group's first / second 32 is kept
      if constexpr (EPI == kEpiGateSplit) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int pair = tm * 128 + grp * 64 + c * 32 + lane;
          const int line = pair / p.mask_pitch, pos = pair - line * p.mask_pitch;
          const bool k = pair < p.m_valid && pos < p.mask_n && p.mask[line * p.mask_line + pos * p.mask_pos] != 0;
          keep[c] = __ballot_sync(0xffffffffu, k);
        }
      }
      if (kTileOperand<EPI>) mbar_wait(mul_full, it & 1, 5);
      mbar_wait(&acc_full[acc], (it >> 1) & 1, 4);
      tc_fence_after_sync();
      const int row = tm * 128 + quarter * 32 + lane;
      const float scale = p.scale_ptr ? p.scale * p.scale_ptr[b] : p.scale;
      if constexpr (EPI == kEpiSwiglu) {
        // 32 output columns at a time from the matching columns of both blocks; a staging tile is 64 output columns
        const int r = quarter * 32 + lane;
        const bool leader = threadIdx.x == 64;
#pragma unroll
        for (int c = 0; c < BN / 64; ++c) {
          const int a_col = (c >> 1) * 128 + (c & 1) * 32;
          uint32_t va[32], vb[32];
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + a_col), va);
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + a_col + 64), vb);
          uint8_t* stage = smem + Cfg::OUT_OFFSET + ((it * (BN / 128) + (c >> 1)) & 1) * 16384;
          if ((c & 1) == 0) {
            if (leader) tma_store_wait_read1();  // the store that last used this staging tile has read it
            named_bar_sync(1, 128);
          }
          tmem_ld_wait();
          if (c + 1 == BN / 64) {
            tc_fence_before_sync();
            mbar_arrive(&acc_empty[acc]);
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float a = __uint_as_float(va[g * 8 + e]);
              x[e] = a * sigmoid_fast(a) * __uint_as_float(vb[g * 8 + e]);
            }
            *reinterpret_cast<uint4*>(stage + sw128_offset(r, (c & 1) * 4 + g)) =
                make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
          }
          if (c & 1) {
            fence_proxy_async_smem();
            named_bar_sync(1, 128);
            const int col = tn * (BN / 2) + (c >> 1) * 64;
            if (leader) {
              if (col < p.n_valid / 2) tma_store_3d(&tmC, stage, col, tm * 128, b);
              tma_store_commit();  // an empty group too: the waits count groups
            }
          }
        }
        continue;
      }
      if constexpr (EPI == kEpiSwigluSplit) {
        // The hi and the lo part of the group's 64 output columns in a staging tile each.
        static_assert(BN == 256 || EPI != kEpiSwigluSplit, "a column group per warp group");
        const int r = quarter * 32 + lane;
        const bool leader = (threadIdx.x & 127) == 64;
        uint8_t* stage = smem + Cfg::OUT_OFFSET + grp * 32768;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int a_col = grp * 128 + c * 32;
          uint32_t va[32], vb[32];
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + a_col), va);
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + a_col + 64), vb);
          tmem_ld_wait();
          if (c == 1) {
            tc_fence_before_sync();
            mbar_arrive(&acc_empty[acc]);
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float a = __uint_as_float(va[e]);
            va[e] = __float_as_uint(times_sigmoid(a, a) * __uint_as_float(vb[e]));
          }
          if (c == 0) {
            if (leader) tma_store_wait_read0();  // the stores that last used the staging tiles have read them
            named_bar_sync(1 + grp, 128);
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              split_pair(__uint_as_float(va[g * 8 + 2 * e]), __uint_as_float(va[g * 8 + 2 * e + 1]), hi[e], lo[e]);
            *reinterpret_cast<uint4*>(stage + sw128_offset(r, c * 4 + g)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(stage + 16384 + sw128_offset(r, c * 4 + g)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
          if (c == 1) {
            fence_proxy_async_smem();
            named_bar_sync(1 + grp, 128);
            const int col = tn * (BN / 2) + grp * 64;
            if (leader && col < p.n_valid / 2) {
              tma_store_3d(&tmC, stage, col, tm * 128, b);
              tma_store_3d(&tmC, stage + 16384, p.n_valid / 2 + col, tm * 128, b);
              tma_store_commit();
            }
          }
        }
        continue;
      }
      if constexpr (EPI == kEpiGateSplit) {
        static_assert(BN == 256 || EPI != kEpiGateSplit, "p and g of 128 channels");
        const int r = quarter * 32 + lane;  // channel
        const bool leader = (threadIdx.x & 127) == 64;
        uint8_t* stage = smem + Cfg::OUT_OFFSET + grp * 32768;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t va[32], vb[32];
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + grp * 64 + c * 32), va);
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + 128 + grp * 64 + c * 32), vb);
          tmem_ld_wait();
          if (c == 1) {
            tc_fence_before_sync();
            mbar_arrive(&acc_empty[acc]);
          }
#pragma unroll
          for (int e = 0; e < 32; ++e)  // an AND masks: a selection would be a branch around each value (114 us for the op)
            va[e] = __float_as_uint(times_sigmoid(__uint_as_float(va[e]), __uint_as_float(vb[e]))) & (0u - ((keep[c] >> e) & 1u));
          if (c == 0) {
            if (leader) tma_store_wait_read0();  // the stores that last used the staging tiles have read them
            named_bar_sync(1 + grp, 128);
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              split_pair(__uint_as_float(va[g * 8 + 2 * e]), __uint_as_float(va[g * 8 + 2 * e + 1]), hi[e], lo[e]);
            *reinterpret_cast<uint4*>(stage + sw128_offset(r, c * 4 + g)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(stage + 16384 + sw128_offset(r, c * 4 + g)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
        }
        fence_proxy_async_smem();
        named_bar_sync(1 + grp, 128);
        const int pair0 = tm * 128 + grp * 64;
        if (leader && pair0 < p.m_valid) {
          tma_store_3d(&tmC, stage, pair0, 0, tn);
          tma_store_3d(&tmC, stage + 16384, pair0, 128, tn);
          tma_store_commit();
        }
        continue;
      }
      if constexpr (kBulk<EPI> || kTileOperand<EPI>) {
        // 32 columns at a time into one of two swizzled staging tiles; warp 2's first lane sends each tile off.
        const int r = quarter * 32 + lane;
        const bool leader = (threadIdx.x & 127) == 64;
        const int c1 = tm * 128, c2 = b;  // tensor map {column, row, batch}
        const int cps = p.out_f32 ? 1 : 2;  // 32-column chunks per staging tile
        uint32_t va[32], vb[32];
        constexpr int CHUNKS = GCOLS / 32;
        const uint32_t t_addr = tmem_addr(tmem_base, quarter * 32, acc * BN + grp * GCOLS);
        uint8_t* stages = smem + Cfg::OUT_OFFSET + grp * 32768;
        tmem_ld_32x32(t_addr, va);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
          uint32_t(&v)[32] = (c & 1) ? vb : va;
          const int st = p.out_f32 ? c : (c >> 1);  // staging tile number within the output tile
          uint8_t* stage = stages + ((it * (CHUNKS / cps) + st) & 1) * 16384;
          if (p.out_f32 || (c & 1) == 0) {
            if (leader) tma_store_wait_read1();  // the store that last used this staging tile has read it
            named_bar_sync(1 + grp, 128);
          }
          tmem_ld_wait();
          if (c + 1 < CHUNKS) {
            tmem_ld_32x32(t_addr + (c + 1) * 32, (c & 1) ? va : vb);
          } else {
            tc_fence_before_sync();
            mbar_arrive(&acc_empty[acc]);
          }
          const uint8_t* factors = smem + Cfg::MUL_OFFSET + c * 16384;
          if (p.out_f32) {
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              float4 x;
              x.x = __uint_as_float(v[g * 4 + 0]) * scale;
              x.y = __uint_as_float(v[g * 4 + 1]) * scale;
              x.z = __uint_as_float(v[g * 4 + 2]) * scale;
              x.w = __uint_as_float(v[g * 4 + 3]) * scale;
              if (p.bias) {
                const float4 bv = *reinterpret_cast<const float4*>(bias_s + grp * GCOLS + c * 32 + g * 4);
                x.x += bv.x; x.y += bv.y; x.z += bv.z; x.w += bv.w;
              }
              if (EPI == kEpiMul) {
                const float4 mv = *reinterpret_cast<const float4*>(factors + sw128_offset(r, g));
                x.x *= mv.x; x.y *= mv.y; x.z *= mv.z; x.w *= mv.w;
              }
              if (EPI == kEpiAdd) {
                const float4 av = *reinterpret_cast<const float4*>(factors + sw128_offset(r, g));
                x.x += av.x; x.y += av.y; x.z += av.z; x.w += av.w;
              }
              *reinterpret_cast<float4*>(stage + sw128_offset(r, g)) = x;
            }
          } else {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              float x[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[g * 8 + e]) * scale;
              if (p.bias) {
                const float4 b0 = *reinterpret_cast<const float4*>(bias_s + grp * GCOLS + c * 32 + g * 8);
                const float4 b1 = *reinterpret_cast<const float4*>(bias_s + grp * GCOLS + c * 32 + g * 8 + 4);
                x[0] += b0.x; x[1] += b0.y; x[2] += b0.z; x[3] += b0.w;
                x[4] += b1.x; x[5] += b1.y; x[6] += b1.z; x[7] += b1.w;
              }
              if (EPI == kEpiMul) {
                const float4 m0 = *reinterpret_cast<const float4*>(factors + sw128_offset(r, g * 2));
                const float4 m1 = *reinterpret_cast<const float4*>(factors + sw128_offset(r, g * 2 + 1));
                x[0] *= m0.x; x[1] *= m0.y; x[2] *= m0.z; x[3] *= m0.w;
                x[4] *= m1.x; x[5] *= m1.y; x[6] *= m1.z; x[7] *= m1.w;
              }
              if (EPI == kEpiAdd) {
                const uint4 a4 = *reinterpret_cast<const uint4*>(smem + Cfg::MUL_OFFSET + (c >> 1) * 16384 + sw128_offset(r, (c & 1) * 4 + g));
                const uint32_t aw[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) x[2 * e] += bf16lo(aw[e]), x[2 * e + 1] += bf16hi(aw[e]);
              }
              *reinterpret_cast<uint4*>(stage + sw128_offset(r, (c & 1) * 4 + g)) = make_uint4(
                  pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
            }
          }
          if (p.out_f32 || (c & 1) == 1) {
            const int tcol0 = tn * BN + grp * GCOLS + st * 32 * cps;
            fence_proxy_async_smem();
            named_bar_sync(1 + grp, 128);
            if (leader) {
              if (tcol0 >= p.n_valid) {
              } else if (p.tma_c == 2)
                tma_reduce_add_3d(&tmC, stage, tcol0, c1, c2);
              else if (p.tma_c == 3)
                tma_store_4d(&tmC, stage, tcol0, 0, tm * 4, b);
              else
                tma_store_3d(&tmC, stage, tcol0, c1, c2);
              tma_store_commit();  // an empty group too: the waits count groups
            }
          }
        }
        // every thread has read its part before the last barrier above
        if (kTileOperand<EPI> && leader && tile + int(gridDim.x) < total_tiles) load_factors(tile + gridDim.x);
        continue;
      }
      if constexpr (EPI == kEpiOuter) {
        // A warp's 32 lanes x 32 columns are one pair's outer product, 2 KB in one piece: through one of the warp's four
        // buffers and out as a bulk copy (16-byte stores of the lanes' 64-byte rows: 98 us against 49 for 256 x 256 pairs).
        // The lanes of a quarter-warp write their four 16-byte units in rotated order, which keeps them on different banks.
        const int i = tm * 4 + quarter;
        uint8_t* buf = smem + Cfg::OUT_OFFSET + quarter * 8192;
        uint32_t va[32], vb[32];
        tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN), va);
#pragma unroll
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t(&v)[32] = (c & 1) ? vb : va;
          tmem_ld_wait();
          if (c + 1 < BN / 32) {
            tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + (c + 1) * 32), (c & 1) ? va : vb);
          } else {
            tc_fence_before_sync();
            mbar_arrive(&acc_empty[acc]);
          }
          uint4 w[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[g * 8 + e]) * scale;
            w[g] = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
          }
          const int j = (tn * BN >> 5) + c;
          if (i * 32 < p.m_valid && j * 32 < p.n_valid) {
            uint8_t* row = buf + (c & 3) * 2048 + lane * 64;
            if (lane == 0) tma_store_wait_read3();  // the copy that last used this buffer has read it
            __syncwarp();
            const int rot = (lane >> 1) & 3;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const int u = (g + rot) & 3;
              *reinterpret_cast<uint4*>(row + u * 16) = u == 0 ? w[0] : u == 1 ? w[1] : u == 2 ? w[2] : w[3];
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0)
              bulk_store(static_cast<__nv_bfloat16*>(p.C) + ((long long)i * p.opm_ntok + j) * 1024, buf + (c & 3) * 2048, 2048);
          }
          if (lane == 0) tma_store_commit();  // an empty group too: the waits count groups
        }
        continue;
      }
      if constexpr (EPI == kEpiDirect) {
      const size_t esz = p.out_f32 ? 4 : 2;
      uint8_t* cbase = static_cast<uint8_t*>(p.C) + (long long)b * p.c_batch_stride * esz;
      // 32 columns at a time; the next chunk's TMEM load and (when a residual is added) its residual row
      // segment are requested before the current chunk is processed.
      const uint8_t* rbase = p.residual ? static_cast<const uint8_t*>(p.residual) + (long long)b * p.c_batch_stride * esz
                                        : nullptr;
      auto chunk_off = [&](int c) -> long long {  // element offset of (row, first column of chunk c)
        const int col0 = tn * BN + c * 32;
        return (long long)row * p.ldc + col0;
      };
      auto load_res = [&](int c, float (&rz)[32]) {
        const long long off0 = chunk_off(c);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float t8[8];
          const bool ok = rbase && row < p.m_valid && (tn * BN + c * 32 + g * 8) < p.n_valid;
          if (ok) {
            if (p.out_f32)
              load8<true>(rbase + (off0 + g * 8) * 4, 0, t8);
            else
              load8<false>(rbase + (off0 + g * 8) * 2, 0, t8);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) rz[g * 8 + e] = ok ? t8[e] : 0.f;
        }
      };
      uint32_t va[32], vb[32];
      float ra[32], rb[32];
      tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN), va);
      load_res(0, ra);
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t(&v)[32] = (c & 1) ? vb : va;
        float(&rz)[32] = (c & 1) ? rb : ra;
        tmem_ld_wait();
        if (c + 1 < BN / 32) {
          tmem_ld_32x32(tmem_addr(tmem_base, quarter * 32, acc * BN + (c + 1) * 32), (c & 1) ? va : vb);
          load_res(c + 1, (c & 1) ? ra : rb);
        }
        if (row < p.m_valid) {
          const int col0 = tn * BN + c * 32;
          const long long off0 = chunk_off(c);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int col = col0 + g * 8;
            if (col < p.n_valid) {
              float x[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] = fmaf(__uint_as_float(v[g * 8 + e]), scale, rz[g * 8 + e]);
              if (p.bias) {
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] += p.bias[col + e];
              }
              if (p.out_f32)
                store8<true>(cbase + (off0 + g * 8) * 4, 0, x);
              else
                store8<false>(cbase + (off0 + g * 8) * 2, 0, x);
            }
          }
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&acc_empty[acc]);
      }
    }
  }

  if (warp >= 2 && (EPI == kEpiOuter ? lane == 0 : EPI != kEpiDirect && (threadIdx.x & 127) == 64)) tma_store_wait0();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200
