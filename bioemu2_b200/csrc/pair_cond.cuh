// The pairwise conditioning of the diffusion module in one pass over the pair tensor:
//
//   z = W . LayerNorm(x1 | x2);   z += T_t(z) for each transition t,   T(z) = fc3( silu(fc1(h)) * fc2(h) ), h = LayerNorm(z)
//
// for 128 + 128 -> 128 channels and transitions 128 -> 256 -> 128.  A tile is 128 pair rows.  z of a tile lives in tensor memory from
// the first product to the last: fc3 accumulates onto it, so the residual costs nothing, and the LayerNorms in between read it
// from there (a lane is a row).  Their result X and the SwiGLU's H go back to tensor memory, as the A operands of the products.
// All weights (64 KB and 192 KB a transition) stream from L2 through one ring of 16 KB units in the order in which the products
// take them.
//
//   warps 0-7    two groups of four: LayerNorm of 64 channels of z each (a row's halves meet in shared memory), the
//                SwiGLU of the even / odd chunks of 64 hidden units, 64 channels of the finished tile to TMA
//   warps 8-13   producers: LayerNorm of the next tile's source rows into the operand S
//   warp  14     issues all products
//   warp  15     TMA of the weights
//
// As ln_linear_kernel and two transition_kernel passes z went through memory five times more: 151 us at 384 x 384 pairs, 264 at
// 512 x 512; here 96 and 165 (the two sources and the result alone: 35 and 62 us).  The chain of a tile bounds it (LayerNorm 1.8, four
// chunks of SwiGLU and products 6 thousand clocks, twice, of 22); by the counters no pipe does: tensor pipe 34 % active, issue slots
// 39 %, the threads' accesses to shared memory 28 %, DRAM 22 %.  With X and H in shared memory it took 123 us.  Tried: 16 warps on the
// LayerNorm and SwiGLU at 80 registers (126 us: the producers then have one row a thread in flight), a warp a source row (142: more
// shuffles, which share the shared memory's path), the output stored by the lanes (110).
// At 128 registers a thread it spills 140 bytes for fp32 sources and 168 for bf16.
#pragma once
#include "row_tile.cuh"

namespace b200 {

constexpr int kPairCondMaxTransitions = 2;

struct PairCondParams {
  const void* x1;  // [rows][128] fp32 or bf16
  const void* x2;
  const float* ln_w;  // [256], may be nullptr
  const float* ln_b;
  const float* t_ln_w[kPairCondMaxTransitions];  // [128]
  const float* t_ln_b[kPairCondMaxTransitions];
  long long rows;
  int num_tiles;
  int transitions;  // 1 .. kPairCondMaxTransitions
  float eps;
};

struct PairCondMaps {
  CUtensorMap out;                           // [rows][128] fp32
  CUtensorMap w0;                            // [128][256]
  CUtensorMap w13[kPairCondMaxTransitions];  // [512][128]: 64 rows of fc1, 64 of fc2 a chunk
  CUtensorMap w3[kPairCondMaxTransitions];   // [128][256]
};

namespace pair_cond {
constexpr int CHUNKS = 4, UNITS = 5;
constexpr uint32_t S_OFF = 0;                                 // two sources x 32 KB
constexpr uint32_t W_OFF = 2 * kOperandTile;                  // ring of units, [128 rows][64 K]
constexpr uint32_t STAGE_OFF = W_OFF + UNITS * kOperandHalf;  // the finished tile, four times [128 rows][32 channels] fp32
constexpr uint32_t XCH_OFF = STAGE_OFF + 2 * kOperandTile;    // mean and squares of the rows' halves, [2 groups][128 rows] x 2 fp32
constexpr uint32_t LN_OFF = XCH_OFF + 2048;                     // the transitions' weight and half bias, [128] fp32 each
constexpr uint32_t BAR_OFF = LN_OFF + kPairCondMaxTransitions * 1024;
constexpr uint32_t SMEM_BYTES = BAR_OFF + 512 + 1024;
constexpr int COMPUTE = 256, PRODUCERS = 192, THREADS = COMPUTE + PRODUCERS + 64;
}  // namespace pair_cond

template <bool F32>
__global__ void __launch_bounds__(512, 1)
pair_cond_kernel(const __grid_constant__ PairCondMaps maps, const __grid_constant__ PairCondParams p) {
  using namespace pair_cond;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* s_full = bars;           // count PRODUCERS
  uint64_t* s_empty = bars + 1;      // commit
  uint64_t* x_full = bars + 2;       // count COMPUTE
  uint64_t* x_empty = bars + 3;      // commit
  uint64_t* d1_full = bars + 4;      // [2] commit
  uint64_t* h_full = bars + 6;       // [2] count 128: D1 has been read, H written over it
  uint64_t* z_full = bars + 8;       // commit: after the input projection and after each transition
  uint64_t* z_empty = bars + 9;      // count COMPUTE: the finished tile has been read
  uint64_t* w_full = bars + 10;      // [UNITS] TMA
  uint64_t* w_empty = w_full + UNITS;  // [UNITS] commit
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_empty + UNITS);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(s_full, PRODUCERS);
    mbar_init(s_empty, 1);
    mbar_init(x_full, COMPUTE);
    mbar_init(x_empty, 1);
    mbar_init(z_full, 1);
    mbar_init(z_empty, COMPUTE);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&d1_full[i], 1);
      mbar_init(&h_full[i], 128);
    }
    for (int i = 0; i < UNITS; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], 1);
    }
    fence_mbar_init();
    prefetch_tmap(&maps.w0);
    prefetch_tmap(&maps.out);
    prefetch_tmap(&maps.w13[0]);
    prefetch_tmap(&maps.w3[0]);
  }
  if (warp == 14) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  float* ln = reinterpret_cast<float*>(smem + LN_OFF);
  for (int i = threadIdx.x; i < p.transitions * 128; i += THREADS) {
    ln[(i >> 7) * 256 + (i & 127)] = p.t_ln_w[i >> 7][i & 127];
    ln[(i >> 7) * 256 + 128 + (i & 127)] = 0.5f * p.t_ln_b[i >> 7][i & 127];
  }
  __syncthreads();
  // TMEM columns: D1[b] at b * 128 (fc1 chunk 0..63, fc2 chunk 64..127) with H[b] over its first 32, z, X.
  constexpr uint32_t TM_Z = 256, TM_X = 384;

  const int T = p.transitions;
  int my_tiles = 0;
  for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x) ++my_tiles;

  if (warp == 15) {
    // ------------------------------------------------------------------ weights, in the issuer's order
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      auto unit = [&](const CUtensorMap* tm, int k, int row) {
        mbar_wait(&w_empty[stage], phase ^ 1, 120);
        mbar_arrive_expect_tx(&w_full[stage], kOperandHalf);
        tma_load_2d(smem + W_OFF + stage * kOperandHalf, tm, &w_full[stage], k, row);
        if (++stage == UNITS) stage = 0, phase ^= 1;
      };
      for (int i = 0; i < my_tiles; ++i) {
        for (int j = 0; j < 4; ++j) unit(&maps.w0, j * 64, 0);
        for (int t = 0; t < T; ++t)
          for (int c = 0; c <= CHUNKS; ++c) {  // fc1 | fc2 of chunk c, then fc3 of the chunk before it
            if (c < CHUNKS) {
              unit(&maps.w13[t], 0, c * 128);
              unit(&maps.w13[t], 64, c * 128);
            }
            if (c > 0) unit(&maps.w3[t], (c - 1) * 64, 0);
          }
      }
    }
  } else if (warp == 14) {
    // ------------------------------------------------------------------ issuer (the whole warp waits, one elected lane issues)
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(128, 128);
    const uint32_t smem_base = smem_u32(smem);
    int stage = 0;
    uint32_t phase = 0;
    auto unit_wait = [&]() -> uint32_t {  // the ring's next unit as the B operand
      mbar_wait(&w_full[stage], phase, 121);
      tc_fence_after_sync();
      return desc_lo(smem_base + W_OFF + stage * kOperandHalf);
    };
    auto unit_done = [&] {
      if (leader) umma_commit(&w_empty[stage]);
      __syncwarp();
      if (++stage == UNITS) stage = 0, phase ^= 1;
    };
    auto commit = [&](uint64_t* bar) {
      if (leader) umma_commit(bar);
      __syncwarp();
    };
    int n = 0, g = 0;  // transitions and chunks so far
    for (int i = 0; i < my_tiles; ++i) {
      mbar_wait(s_full, i & 1, 122);
      mbar_wait(z_empty, (i & 1) ^ 1, 123);
      for (int j = 0; j < 4; ++j) {
        const uint32_t b_lo = unit_wait(), a_lo = desc_lo(smem_base + S_OFF + j * kOperandHalf);
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ss2(tmem_base + TM_Z, a_lo + 2 * k, kDescHiSw128, b_lo + 2 * k, kDescHiSw128, idesc, (j | k) != 0);
        }
        unit_done();
      }
      commit(s_empty);
      commit(z_full);
      // GEMM1 of chunk c, then GEMM2 of chunk c - 1, from one warp, so that they run in this order: GEMM1 of chunk c + 1 writes over
      // the H that GEMM2 of chunk c - 1 reads.
      for (int t = 0; t < T; ++t, ++n) {
        mbar_wait(x_full, n & 1, 124);
        for (int c = 0; c <= CHUNKS; ++c) {
          if (c < CHUNKS) {
            const uint32_t d1 = tmem_base + ((g + c) & 1) * 128;
            for (int j = 0; j < 2; ++j) {
              const uint32_t b_lo = unit_wait();
              if (leader) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  umma_bf16_ts2(d1, tmem_base + TM_X + j * 32 + k * 8, b_lo + 2 * k, kDescHiSw128, idesc, (j | k) != 0);
              }
              unit_done();
            }
            commit(&d1_full[(g + c) & 1]);
            if (c == CHUNKS - 1) commit(x_empty);
          }
          if (c > 0) {
            const int gc = g + c - 1;
            mbar_wait(&h_full[gc & 1], (gc >> 1) & 1, 126);
            const uint32_t b_lo = unit_wait(), h = tmem_base + (gc & 1) * 128;
            if (leader) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_bf16_ts2(tmem_base + TM_Z, h + k * 8, b_lo + 2 * k, kDescHiSw128, idesc, true);
            }
            unit_done();
          }
        }
        commit(z_full);
        g += CHUNKS;
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ producers: 16 threads a row, 12 rows at a time
    const int pt = threadIdx.x - COMPUTE;
    const int c0 = (pt & 15) * 8, rbase = pt >> 4;
    float gamma[2][8], beta[2][8];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        gamma[k][e] = p.ln_w ? p.ln_w[k * 128 + c0 + e] : 1.0f;
        beta[k][e] = p.ln_b ? p.ln_b[k * 128 + c0 + e] : 0.0f;
      }
    constexpr int U = 2, GROUPS = 6;  // rows (q * U + u) * 12 + rbase, those below 128
    float xa[U][2][8], xb[U][2][8];
    auto load = [&](int tile, int q, float (&x)[U][2][8]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = (q * U + u) * 12 + rbase;
        const long long row = (long long)tile * 128 + r;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (r < 128 && row < p.rows && tile < p.num_tiles) {
            load8<F32>(static_cast<const uint8_t*>(k ? p.x2 : p.x1) + row * 128 * (long long)zbytes<F32>(), c0, x[u][k]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[u][k][e] = 0.f;
          }
        }
      }
    };
    auto emit = [&](int q, float (&x)[U][2][8]) {
      float sm[U], sq[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        sm[u] = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int e = 0; e < 8; ++e) sm[u] += x[u][k][e];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < U; ++u) sm[u] += __shfl_xor_sync(0xffffffffu, sm[u], o);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float mean = sm[u] * (1.0f / 256);
        sq[u] = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            x[u][k][e] -= mean;
            sq[u] = fmaf(x[u][k][e], x[u][k][e], sq[u]);
          }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < U; ++u) sq[u] += __shfl_xor_sync(0xffffffffu, sq[u], o);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float rstd = rsqrtf(sq[u] * (1.0f / 256) + p.eps);
        const int r = (q * U + u) * 12 + rbase;
        if (r >= 128) continue;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] = fmaf(x[u][k][e] * rstd, gamma[k][e], beta[k][e]);
          *reinterpret_cast<uint4*>(smem + S_OFF + k * kOperandTile + ((pt & 15) >> 3) * kOperandHalf + sw128_offset(r, pt & 7)) =
              make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
        }
      }
    };
    int it = 0;
    load(blockIdx.x, 0, xa);
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      load(tile, 1, xb);
      mbar_wait(s_empty, (it & 1) ^ 1, 127);
#pragma unroll
      for (int q = 0; q < GROUPS; q += 2) {
        emit(q, xa);
        if (q + 2 < GROUPS) load(tile, q + 2, xa);
        else load(tile + gridDim.x, 0, xa);
        emit(q + 1, xb);
        if (q + 3 < GROUPS) load(tile, q + 3, xb);
      }
      fence_proxy_async_smem();
      mbar_arrive(s_full);
    }
  } else {
    // ------------------------------------------------------------------ LayerNorm of z, SwiGLU, output
    const int grp = warp >> 2, quarter = warp & 3;  // channels 64 * grp ..; chunks of parity grp
    const int r = quarter * 32 + lane;              // row of the tile == TMEM lane
    const bool leader = (threadIdx.x & 127) == 0;
    uint8_t* stage = smem + STAGE_OFF + grp * kOperandTile;
    float2* xch = reinterpret_cast<float2*>(smem + XCH_OFF);
    const uint32_t z_addr = tmem_addr(tmem_base, quarter * 32, TM_Z + grp * 64);
    const uint32_t d1_addr = tmem_addr(tmem_base, quarter * 32, grp * 128);
    int tile = blockIdx.x, n = 0;
    for (int i = 0; i < my_tiles; ++i, tile += gridDim.x) {
      for (int t = 0; t < T; ++t, ++n) {
        mbar_wait(z_full, (i * (T + 1) + t) & 1, 129);
        tc_fence_after_sync();
        {
          float v[64];
          tmem_ld_32x32_f(z_addr, v);
          tmem_ld_32x32_f(z_addr + 32, v + 32);
          tmem_ld_wait();
          // A half's sum of squares about its own mean, then one exchange: mean and variance of the row are those of its halves, d on
          // either side of the mean (T. Chan, G. Golub, R. LeVeque, "Updating formulae and a pairwise algorithm for computing sample
          // variances", 1979).  The mean of the squares less the square of the mean has no digits left where a row's mean is a
          // thousand times its deviation (it took 94.9 us at 384 x 384 pairs where this takes 95.6).
          float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, q0[4] = {0.f, 0.f, 0.f, 0.f}, q1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int e = 0; e < 64; e += 2) add_f32x2(s0[(e >> 1) & 3], s1[(e >> 1) & 3], v[e], v[e + 1]);
          const float mu = (((s0[0] + s1[0]) + (s0[1] + s1[1])) + ((s0[2] + s1[2]) + (s0[3] + s1[3]))) * (1.0f / 64);
#pragma unroll
          for (int e = 0; e < 64; e += 2) {
            add_f32x2(v[e], v[e + 1], -mu, -mu);
            fma_f32x2(q0[(e >> 1) & 3], q1[(e >> 1) & 3], v[e], v[e + 1], v[e], v[e + 1], q0[(e >> 1) & 3], q1[(e >> 1) & 3]);
          }
          const float sq = ((q0[0] + q1[0]) + (q0[1] + q1[1])) + ((q0[2] + q1[2]) + (q0[3] + q1[3]));
          xch[grp * 128 + r] = make_float2(mu, sq);
          named_bar_sync(3, COMPUTE);
          const float2 other = xch[(grp ^ 1) * 128 + r];
          const float d = 0.5f * (other.x - mu);
          // half of the LayerNorm: see the SwiGLU below
          const float rstd = 0.5f * rsqrtf((sq + other.y) * (1.0f / kD) + d * d + p.eps);
          const float shift = -d * rstd;
          mbar_wait(x_empty, (n & 1) ^ 1, 130);
          tc_fence_after_sync();
          const float4* gw = reinterpret_cast<const float4*>(ln + t * 256 + grp * 64);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t o[16];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float4 w4 = gw[half * 8 + q], b4 = gw[32 + half * 8 + q];
              const float* x = v + half * 32 + q * 4;
              o[q * 2] = pack_bf16x2(fmaf(fmaf(x[0], rstd, shift), w4.x, b4.x), fmaf(fmaf(x[1], rstd, shift), w4.y, b4.y));
              o[q * 2 + 1] = pack_bf16x2(fmaf(fmaf(x[2], rstd, shift), w4.z, b4.z), fmaf(fmaf(x[3], rstd, shift), w4.w, b4.w));
            }
            tmem_st_32x16(tmem_addr(tmem_base, quarter * 32, TM_X + grp * 32 + half * 16), o);
          }
          tmem_st_wait();
          tc_fence_before_sync();
          mbar_arrive(x_full);
        }
        // With a' = fc1(h) / 2 and b' = fc2(h) / 2 from the halved operand: silu(a) b = u + u tanh(a'), u = 2 a' b'.
        for (int c = grp; c < CHUNKS; c += 2) {
          const int g = n * CHUNKS + c;
          mbar_wait(&d1_full[grp], (g >> 1) & 1, 131);
          tc_fence_after_sync();
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            uint32_t av[32], bv[32], o[16];
            tmem_ld_32x32(d1_addr + half * 32, av);
            tmem_ld_32x32(d1_addr + 64 + half * 32, bv);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float a0 = __uint_as_float(av[2 * e]), a1 = __uint_as_float(av[2 * e + 1]);
              const float u0 = (a0 + a0) * __uint_as_float(bv[2 * e]), u1 = (a1 + a1) * __uint_as_float(bv[2 * e + 1]);
              o[e] = pack_bf16x2(fmaf(u0, tanh_approx(a0), u0), fmaf(u1, tanh_approx(a1), u1));
            }
            tmem_st_32x16(d1_addr + half * 16, o);  // over fc1 columns read before
          }
          tmem_st_wait();
          tc_fence_before_sync();
          mbar_arrive(&h_full[grp]);
        }
      }
      // the finished tile, through staging tiles and TMA (stored by the lanes, a row each: 2,800 clocks a tile)
      if (leader) tma_store_wait_read0();  // the previous tile's stores have read the staging tiles
      named_bar_sync(1 + grp, 128);
      mbar_wait(z_full, (i * (T + 1) + T) & 1, 128);
      tc_fence_after_sync();
      float v[64];
      tmem_ld_32x32_f(z_addr, v);
      tmem_ld_32x32_f(z_addr + 32, v + 32);
      tmem_ld_wait();
      tc_fence_before_sync();
      mbar_arrive(z_empty);
#pragma unroll
      for (int q = 0; q < 16; ++q)
        *reinterpret_cast<float4*>(stage + (q >> 3) * kOperandHalf + sw128_offset(r, q & 7)) =
            make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
      fence_proxy_async_smem();
      named_bar_sync(1 + grp, 128);
      if (leader) {
        tma_store_2d(&maps.out, stage, grp * 64, tile * 128);
        tma_store_2d(&maps.out, stage + kOperandHalf, grp * 64 + 32, tile * 128);
        tma_store_commit();
      }
    }
    if (leader) tma_store_wait0();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 14) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200
