// The per-token parts of a conditioned transformer block of 128 channels on either side of its attention, in one kernel each:
//
//   cond_in_kernel    cond = W_c silu(LayerNorm(c)) + b_c;  y = lns (LN(x) (1 + alpha1) + beta1);  q | k | v | gate = W y + b
//   cond_out_kernel   x1 = x + gamma1 (W_o og);  y = lns (LN(x1) (1 + alpha2) + beta2);
//                     out = x1 + gamma2 fc3( silu(fc1(y)) * fc2(y) )
//
// The six conditioning vectors of a token (3 KB as fp32) never leave the SM: each kernel computes those it needs, in fp32 tensor
// memory, from the 512 bytes of c.  A tile is 128 tokens, a tensor-memory lane a token; operands that the lanes produce (y, the
// SwiGLU's H) go back to tensor memory.  Weights stream from L2 through a ring of 16 KB units in the order of the products.
//
//   warps 0-7    two groups of four, 64 channels each: adaptive LayerNorm, gates, SwiGLU of the even / odd chunks, output
//   warps 8-13   producers: silu(LayerNorm(c)) into the operand S, a tile ahead
//   warp  14     issues all products
//   warp  15     TMA of weights and of the tiles of x and og
//
// 32,768 tokens: as nine kernels (LayerNorm of c, the projection to 100 MB of conditioning, two adaptive LayerNorms, the products, the
// transition, two gated residuals) 104 us beside the attention, most of it reading and writing the conditioning; here 24 + 34.
// Bound by the chain of a tile (about 16 and 22
// thousand clocks) with at most two tiles a CTA to overlap, the first behind its own loads.  At 128 registers a thread both spill (the
// 64 channels of a row a thread beside alpha and beta): 136 bytes in cond_in, 116 in cond_out for an fp32 c, 76 and 84 for bf16.
// Tried: twelve rows of c a thread on their way at once (more spills: 297 us for three layers instead of 277), the output
// projections through one staging tile a group (284).
#pragma once
#include "row_tile.cuh"

namespace b200 {

struct CondBlockParams {
  const void* c;        // [rows][128] fp32 or bf16
  const float* ln_c_w;  // [128] or nullptr
  const float* ln_c_b;
  const float* b_cond;  // [6 * 128]: alpha1 | beta1 | gamma1 | alpha2 | beta2 | gamma2
  const float* b_qkvg;  // [512] (cond_in_kernel)
  long long rows;
  int num_tiles;
  int chunks;           // hidden units / 64 (cond_out_kernel)
  float lns, eps;
};

struct CondInMaps {
  CUtensorMap w_cond;  // [768][128]
  CUtensorMap w_qkvg;  // [512][128]
  CUtensorMap x;       // [rows][128] fp32
  CUtensorMap qkvg;    // [rows][512] bf16
};

struct CondOutMaps {
  CUtensorMap w_cond, w_o;  // w_o [128][128]
  CUtensorMap w13, w3;      // [2 * hidden][128], [128][hidden]
  CUtensorMap og;           // [rows][128] bf16
  CUtensorMap x, out;       // [rows][128] fp32
};

namespace cond_block {
constexpr int COMPUTE = 256, PRODUCERS = 192, THREADS = 512;

// Shared memory with a ring of UNITS and T_TILES [128][64] bf16 tiles (cond_in: two output tiles a group, cond_out: the og operand).
template <int UNITS_, int T_TILES>
struct Layout {
  static constexpr int UNITS = UNITS_;
  static constexpr uint32_t S_OFF = 0;                              // 32 KB
  static constexpr uint32_t X_OFF = S_OFF + kOperandTile;           // x (later x1, the output) fp32: four times [128 rows][32 channels]
  static constexpr uint32_t W_OFF = X_OFF + 2 * kOperandTile;       // units, [128 rows][64 K]
  static constexpr uint32_t T_OFF = W_OFF + UNITS * kOperandHalf;
  static constexpr uint32_t B_OFF = T_OFF + T_TILES * kOperandHalf;  // biases, fp32 [768]
  static constexpr uint32_t XCH_OFF = B_OFF + 768 * 4;               // [2][2 groups][128] fp32
  static constexpr uint32_t BAR_OFF = XCH_OFF + 2048;
  static constexpr uint32_t SMEM_BYTES = BAR_OFF + 512 + 1024;
};
using InLayout = Layout<3, 4>;
using OutLayout = Layout<5, 2>;

// The ring as its loader and its consumer see it.
template <int UNITS>
struct Ring {
  uint8_t* base;
  uint64_t *full, *empty;
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step() {
    if (++stage == UNITS) stage = 0, phase ^= 1;
  }
  __device__ __forceinline__ void load(const CUtensorMap* tm, int k, int row) {
    mbar_wait(&empty[stage], phase ^ 1, 140);
    mbar_arrive_expect_tx(&full[stage], kOperandHalf);
    tma_load_2d(base + stage * kOperandHalf, tm, &full[stage], k, row);
    step();
  }
  __device__ __forceinline__ uint32_t wait() {  // the next unit as a B operand
    mbar_wait(&full[stage], phase, 141);
    tc_fence_after_sync();
    return desc_lo(smem_u32(base + stage * kOperandHalf));
  }
  __device__ __forceinline__ void done(bool leader) {
    if (leader) umma_commit(&empty[stage]);
    __syncwarp();
    step();
  }
};

constexpr uint32_t kIdesc = make_idesc_bf16(128, 128);

// 128 x 128 x 128 with A in shared memory (two 64-channel halves) or in tensor memory, B the ring's next two units.
template <int UNITS>
__device__ __forceinline__ void product_ss(Ring<UNITS>& ring, uint32_t d, uint32_t a_smem, bool leader) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t b_lo = ring.wait(), a_lo = desc_lo(a_smem + j * kOperandHalf);
    if (leader) {
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_bf16_ss2(d, a_lo + 2 * k, kDescHiSw128, b_lo + 2 * k, kDescHiSw128, kIdesc, (j | k) != 0);
    }
    ring.done(leader);
  }
}
template <int UNITS>
__device__ __forceinline__ void product_ts(Ring<UNITS>& ring, uint32_t d, uint32_t a_tmem, bool leader) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t b_lo = ring.wait();
    if (leader) {
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_bf16_ts2(d, a_tmem + j * 32 + k * 8, b_lo + 2 * k, kDescHiSw128, kIdesc, (j | k) != 0);
    }
    ring.done(leader);
  }
}
__device__ __forceinline__ void commit(uint64_t* bar, bool leader) {
  if (leader) umma_commit(bar);
  __syncwarp();
}

// silu(LayerNorm(c)) of the CTA's tiles, 16 threads a row, 12 rows at a time.
template <bool CF32>
__device__ __forceinline__ void produce_cond(const CondBlockParams& p, uint8_t* s, uint64_t* s_full, uint64_t* s_empty) {
  const int pt = threadIdx.x - COMPUTE;
  const int c0 = (pt & 15) * 8, rbase = pt >> 4;
  float gamma[8], beta[8];
  load_gamma_beta(p.ln_c_w, p.ln_c_b, pt, gamma, beta);
  constexpr int U = 3, GROUPS = 4;  // rows (q * U + u) * 12 + rbase, those below 128
  float xa[U][8], xb[U][8];
  auto load = [&](int tile, int q, float (&x)[U][8]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = (q * U + u) * 12 + rbase;
      const long long row = (long long)tile * 128 + r;
      if (r < 128 && row < p.rows && tile < p.num_tiles) {
        load8<CF32>(static_cast<const uint8_t*>(p.c) + row * 128 * (long long)zbytes<CF32>(), c0, x[u]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[u][e] = 0.f;
      }
    }
  };
  auto emit = [&](int q, float (&x)[U][8]) {
    float sum[U];
#pragma unroll
    for (int u = 0; u < U; ++u) sum[u] = ((x[u][0] + x[u][1]) + (x[u][2] + x[u][3])) + ((x[u][4] + x[u][5]) + (x[u][6] + x[u][7]));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float mean = sum[u] * (1.0f / kD);
      sum[u] = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        x[u][e] -= mean;
        sum[u] = fmaf(x[u][e], x[u][e], sum[u]);
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = (q * U + u) * 12 + rbase;
      if (r >= 128) continue;
      const float rstd = rsqrtf(sum[u] * (1.0f / kD) + p.eps);
      float y[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        y[e] = fmaf(x[u][e] * rstd, gamma[e], beta[e]);
        y[e] *= sigmoid_fast(y[e]);
      }
      *reinterpret_cast<uint4*>(s + ((pt & 15) >> 3) * kOperandHalf + sw128_offset(r, pt & 7)) =
          make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
    }
  };
  int it = 0;
  load(blockIdx.x, 0, xa);
  load(blockIdx.x, 1, xb);
  for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
    mbar_wait(s_empty, (it & 1) ^ 1, 142);
#pragma unroll
    for (int q = 0; q < GROUPS; q += 2) {
      emit(q, xa);
      load(q + 2 < GROUPS ? tile : tile + gridDim.x, (q + 2) % GROUPS, xa);
      emit(q + 1, xb);
      load(q + 3 < GROUPS ? tile : tile + gridDim.x, (q + 3) % GROUPS, xb);
    }
    fence_proxy_async_smem();
    mbar_arrive(s_full);
  }
}

// Mean and 1 / std of a row whose two halves of 64 channels two threads (groups 0 and 1) hold; v leaves centred.
__device__ __forceinline__ float center_row(float (&v)[64], float* xch, int grp, int r, float eps) {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 64; ++e) s[e & 3] += v[e];
  const float sum = (s[0] + s[1]) + (s[2] + s[3]);
  xch[grp * 128 + r] = sum;
  named_bar_sync(3, COMPUTE);
  const float mean = (sum + xch[(grp ^ 1) * 128 + r]) * (1.0f / kD);
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] = 0.f;
#pragma unroll
  for (int e = 0; e < 64; ++e) {
    v[e] -= mean;
    s[e & 3] = fmaf(v[e], v[e], s[e & 3]);
  }
  const float sq = (s[0] + s[1]) + (s[2] + s[3]);
  xch[256 + grp * 128 + r] = sq;
  named_bar_sync(3, COMPUTE);
  return rsqrtf((sq + xch[256 + (grp ^ 1) * 128 + r]) * (1.0f / kD) + eps);
}

// y = lns (v rstd (1 + alpha) + beta) of a thread's 64 channels as the packed A operand at x_tmem; alpha and beta are read from
// tensor memory (their biases from shared memory).
__device__ __forceinline__ void adaptive_norm(const float (&v)[64], float rstd, float lns, uint32_t alpha, uint32_t beta, const float* b_alpha,
                                              const float* b_beta, uint32_t x_tmem) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t o[16];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = half * 32 + k * 16;
      float al[16], be[16];
      tmem_ld_32x16_f(alpha + c, al);
      tmem_ld_32x16_f(beta + c, be);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 ba = *reinterpret_cast<const float4*>(b_alpha + c + q * 4), bb = *reinterpret_cast<const float4*>(b_beta + c + q * 4);
        const float y0 = lns * fmaf(v[c + q * 4 + 0] * rstd, 1.0f + (al[q * 4 + 0] + ba.x), be[q * 4 + 0] + bb.x);
        const float y1 = lns * fmaf(v[c + q * 4 + 1] * rstd, 1.0f + (al[q * 4 + 1] + ba.y), be[q * 4 + 1] + bb.y);
        const float y2 = lns * fmaf(v[c + q * 4 + 2] * rstd, 1.0f + (al[q * 4 + 2] + ba.z), be[q * 4 + 2] + bb.z);
        const float y3 = lns * fmaf(v[c + q * 4 + 3] * rstd, 1.0f + (al[q * 4 + 3] + ba.w), be[q * 4 + 3] + bb.w);
        o[k * 8 + q * 2] = pack_bf16x2(y0, y1);
        o[k * 8 + q * 2 + 1] = pack_bf16x2(y2, y3);
      }
    }
    tmem_st_32x16(x_tmem + half * 16, o);
  }
  tmem_st_wait();
}
}  // namespace cond_block

// TMEM columns: alpha1 0..127, beta1 128..255, then two of the four outputs' products at a time over them; y 256..319.
template <bool CF32>
__global__ void __launch_bounds__(512, 1)
cond_in_kernel(const __grid_constant__ CondInMaps maps, const __grid_constant__ CondBlockParams p) {
  using namespace cond_block;
  using L = InLayout;
  constexpr int UNITS = L::UNITS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* s_full = bars;        // count PRODUCERS
  uint64_t* s_empty = bars + 1;   // commit
  uint64_t* x_full = bars + 2;    // TMA
  uint64_t* x_empty = bars + 3;   // count COMPUTE
  uint64_t* ab_full = bars + 4;   // commit
  uint64_t* y_full = bars + 5;    // count COMPUTE
  uint64_t* q_full = bars + 6;    // [2] commit, twice a tile each
  uint64_t* q_empty = bars + 8;   // [2] count COMPUTE
  uint64_t* w_full = bars + 10;   // [UNITS]
  uint64_t* w_empty = w_full + UNITS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_empty + UNITS);
  float* bias = reinterpret_cast<float*>(smem + L::B_OFF);  // alpha1, beta1, q | k | v | gate

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(s_full, PRODUCERS);
    mbar_init(s_empty, 1);
    mbar_init(x_full, 1);
    mbar_init(x_empty, COMPUTE);
    mbar_init(ab_full, 1);
    mbar_init(y_full, COMPUTE);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], COMPUTE);
    }
    for (int i = 0; i < UNITS; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], 1);
    }
    fence_mbar_init();
    prefetch_tmap(&maps.w_cond);
    prefetch_tmap(&maps.w_qkvg);
    prefetch_tmap(&maps.x);
    prefetch_tmap(&maps.qkvg);
  }
  if (warp == 14) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  for (int i = threadIdx.x; i < 768; i += THREADS) bias[i] = i < 256 ? p.b_cond[i] : p.b_qkvg[i - 256];
  __syncthreads();
  constexpr uint32_t TM_Y = 256;
  int my_tiles = 0;
  for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x) ++my_tiles;

  if (warp == 15) {
    if (lane == 0) {
      Ring<UNITS> ring{smem + L::W_OFF, w_full, w_empty};
      for (int i = 0; i < my_tiles; ++i) {
        mbar_wait(x_empty, (i & 1) ^ 1, 143);
        mbar_arrive_expect_tx(x_full, 2 * kOperandTile);
        for (int k = 0; k < 4; ++k)
          tma_load_2d(smem + L::X_OFF + k * kOperandHalf, &maps.x, x_full, k * 32, (blockIdx.x + i * gridDim.x) * 128);
        for (int n = 0; n < 2; ++n)
          for (int j = 0; j < 2; ++j) ring.load(&maps.w_cond, j * 64, n * 128);
        for (int n = 0; n < 4; ++n)
          for (int j = 0; j < 2; ++j) ring.load(&maps.w_qkvg, j * 64, n * 128);
      }
    }
  } else if (warp == 14) {
    const bool leader = elect_one();
    Ring<UNITS> ring{smem + L::W_OFF, w_full, w_empty};
    const uint32_t s = smem_u32(smem + L::S_OFF);
    for (int i = 0; i < my_tiles; ++i) {
      mbar_wait(s_full, i & 1, 144);
      if (i > 0) {
        mbar_wait(&q_empty[0], 1, 145);  // the last two outputs of the tile before have been read
        mbar_wait(&q_empty[1], 1, 146);
      }
      product_ss(ring, tmem_base, s, leader);
      product_ss(ring, tmem_base + 128, s, leader);
      commit(s_empty, leader);
      commit(ab_full, leader);
      mbar_wait(y_full, i & 1, 147);
      for (int n = 0; n < 4; ++n) {
        if (n >= 2) mbar_wait(&q_empty[n & 1], 0, 148);
        product_ts(ring, tmem_base + (n & 1) * 128, tmem_base + TM_Y, leader);
        commit(&q_full[n & 1], leader);
      }
    }
  } else if (warp >= 8) {
    produce_cond<CF32>(p, smem + L::S_OFF, s_full, s_empty);
  } else {
    const int grp = warp >> 2, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const bool leader = (threadIdx.x & 127) == 0;
    uint8_t* stages = smem + L::T_OFF + grp * kOperandTile;  // two tiles in turn
    float* xch = reinterpret_cast<float*>(smem + L::XCH_OFF);
    const uint32_t tm = tmem_addr(tmem_base, quarter * 32, grp * 64);
    int tile = blockIdx.x;
    for (int i = 0; i < my_tiles; ++i, tile += gridDim.x) {
      {
        float v[64];
        mbar_wait(x_full, i & 1, 149);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const float4 f = *reinterpret_cast<const float4*>(smem + L::X_OFF + (grp * 2 + (q >> 3)) * kOperandHalf + sw128_offset(r, q & 7));
          v[q * 4] = f.x, v[q * 4 + 1] = f.y, v[q * 4 + 2] = f.z, v[q * 4 + 3] = f.w;
        }
        mbar_arrive(x_empty);
        const float rstd = center_row(v, xch, grp, r, p.eps);
        mbar_wait(ab_full, i & 1, 150);
        tc_fence_after_sync();
        adaptive_norm(v, rstd, p.lns, tm, tm + 128, bias + grp * 64, bias + 128 + grp * 64,
                      tmem_addr(tmem_base, quarter * 32, TM_Y + grp * 32));
        tc_fence_before_sync();
        mbar_arrive(y_full);
      }
#pragma unroll 1
      for (int n = 0; n < 4; ++n) {
        uint8_t* stage = stages + (n & 1) * kOperandHalf;
        if (leader) tma_store_wait_read1();  // the store before the last has read the staging tile
        named_bar_sync(1 + grp, 128);
        mbar_wait(&q_full[n & 1], (n >> 1) & 1, 151);
        tc_fence_after_sync();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float f[32];
          tmem_ld_32x32_f(tm + (n & 1) * 128 + half * 32, f);
          tmem_ld_wait();
          if (half == 1) {
            tc_fence_before_sync();
            mbar_arrive(&q_empty[n & 1]);
          }
          const float* b = bias + 256 + n * 128 + grp * 64 + half * 32;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 b0 = *reinterpret_cast<const float4*>(b + q * 8), b1 = *reinterpret_cast<const float4*>(b + q * 8 + 4);
            *reinterpret_cast<uint4*>(stage + sw128_offset(r, half * 4 + q)) =
                make_uint4(pack_bf16x2(f[q * 8] + b0.x, f[q * 8 + 1] + b0.y), pack_bf16x2(f[q * 8 + 2] + b0.z, f[q * 8 + 3] + b0.w),
                           pack_bf16x2(f[q * 8 + 4] + b1.x, f[q * 8 + 5] + b1.y), pack_bf16x2(f[q * 8 + 6] + b1.z, f[q * 8 + 7] + b1.w));
          }
        }
        fence_proxy_async_smem();
        named_bar_sync(1 + grp, 128);
        if (leader) {
          tma_store_2d(&maps.qkvg, stage, n * 128 + grp * 64, tile * 128);
          tma_store_commit();
        }
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

// TMEM columns: gamma1 0..127 and W_o og 128..255, alpha2 256..383 and beta2 384..511; then y 0..63, fc3's sum 128..255 and the
// SwiGLU's chunks D1[b] at 256 + b * 128, each with its H over the first 32 columns; at last gamma2 0..127.
template <bool CF32>
__global__ void __launch_bounds__(512, 1)
cond_out_kernel(const __grid_constant__ CondOutMaps maps, const __grid_constant__ CondBlockParams p) {
  using namespace cond_block;
  using L = OutLayout;
  constexpr int UNITS = L::UNITS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* s_full = bars;          // count PRODUCERS
  uint64_t* s_empty = bars + 1;     // commit
  uint64_t* x_full = bars + 2;      // TMA: x and og
  uint64_t* x_empty = bars + 3;     // count 2: the groups' output stores have read the tile
  uint64_t* og_empty = bars + 4;    // commit
  uint64_t* p1_full = bars + 5;     // commit: gamma1, W_o og
  uint64_t* p2_full = bars + 6;     // commit: alpha2, beta2
  uint64_t* y_full = bars + 7;      // count COMPUTE
  uint64_t* d1_full = bars + 8;     // [2] commit
  uint64_t* h_full = bars + 10;     // [2] count 128
  uint64_t* out_full = bars + 12;   // commit: fc3's sum, gamma2
  uint64_t* out_empty = bars + 13;  // count COMPUTE
  uint64_t* og_full = bars + 14;    // TMA
  uint64_t* w_full = bars + 15;     // [UNITS]
  uint64_t* w_empty = w_full + UNITS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_empty + UNITS);
  float* bias = reinterpret_cast<float*>(smem + L::B_OFF);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(s_full, PRODUCERS);
    mbar_init(s_empty, 1);
    mbar_init(x_full, 1);
    mbar_init(x_empty, 2);
    mbar_init(og_empty, 1);
    mbar_init(p1_full, 1);
    mbar_init(p2_full, 1);
    mbar_init(y_full, COMPUTE);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&d1_full[i], 1);
      mbar_init(&h_full[i], 128);
    }
    mbar_init(out_full, 1);
    mbar_init(out_empty, COMPUTE);
    mbar_init(og_full, 1);
    for (int i = 0; i < UNITS; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], 1);
    }
    fence_mbar_init();
    prefetch_tmap(&maps.w_cond);
    prefetch_tmap(&maps.w_o);
    prefetch_tmap(&maps.og);
    prefetch_tmap(&maps.x);
    prefetch_tmap(&maps.w13);
    prefetch_tmap(&maps.w3);
    prefetch_tmap(&maps.out);
  }
  if (warp == 14) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  for (int i = threadIdx.x; i < 768; i += THREADS) bias[i] = p.b_cond[i];
  __syncthreads();
  constexpr uint32_t TM_OUT = 128, TM_AB = 256;
  const int chunks = p.chunks;
  int my_tiles = 0;
  for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x) ++my_tiles;

  if (warp == 15) {
    if (lane == 0) {
      Ring<UNITS> ring{smem + L::W_OFF, w_full, w_empty};
      for (int i = 0; i < my_tiles; ++i) {
        const int row = (blockIdx.x + i * gridDim.x) * 128;
        mbar_wait(og_empty, (i & 1) ^ 1, 152);
        mbar_arrive_expect_tx(og_full, kOperandTile);
        for (int j = 0; j < 2; ++j) tma_load_2d(smem + L::T_OFF + j * kOperandHalf, &maps.og, og_full, j * 64, row);
        for (int j = 0; j < 2; ++j) ring.load(&maps.w_cond, j * 64, 2 * 128);
        for (int j = 0; j < 2; ++j) ring.load(&maps.w_o, j * 64, 0);
        mbar_wait(x_empty, (i & 1) ^ 1, 153);
        mbar_arrive_expect_tx(x_full, 2 * kOperandTile);
        for (int k = 0; k < 4; ++k) tma_load_2d(smem + L::X_OFF + k * kOperandHalf, &maps.x, x_full, k * 32, row);
        for (int n = 3; n < 5; ++n)
          for (int j = 0; j < 2; ++j) ring.load(&maps.w_cond, j * 64, n * 128);
        for (int c = 0; c <= chunks; ++c) {  // fc1 | fc2 of chunk c (after the last: gamma2), fc3 of the chunk before it
          for (int j = 0; j < 2; ++j) ring.load(c < chunks ? &maps.w13 : &maps.w_cond, j * 64, c < chunks ? c * 128 : 5 * 128);
          if (c > 0) ring.load(&maps.w3, (c - 1) * 64, 0);
        }
      }
    }
  } else if (warp == 14) {
    const bool leader = elect_one();
    Ring<UNITS> ring{smem + L::W_OFF, w_full, w_empty};
    const uint32_t s = smem_u32(smem + L::S_OFF);
    int g = 0;  // chunks so far
    for (int i = 0; i < my_tiles; ++i) {
      mbar_wait(s_full, i & 1, 154);
      mbar_wait(out_empty, (i & 1) ^ 1, 155);
      product_ss(ring, tmem_base, s, leader);
      mbar_wait(og_full, i & 1, 156);
      product_ss(ring, tmem_base + 128, smem_u32(smem + L::T_OFF), leader);
      commit(og_empty, leader);
      commit(p1_full, leader);
      product_ss(ring, tmem_base + TM_AB, s, leader);
      product_ss(ring, tmem_base + TM_AB + 128, s, leader);
      commit(p2_full, leader);
      mbar_wait(y_full, i & 1, 157);
      // GEMM1 of chunk c, then GEMM2 of chunk c - 1, from one warp, so that they run in this order: GEMM1 of chunk c + 1 writes over
      // the H that GEMM2 of chunk c - 1 reads, gamma2 over the y that the last GEMM1 reads.
      for (int c = 0; c <= chunks; ++c) {
        if (c < chunks) {
          product_ts(ring, tmem_base + TM_AB + ((g + c) & 1) * 128, tmem_base, leader);
          commit(&d1_full[(g + c) & 1], leader);
        } else {
          product_ss(ring, tmem_base, s, leader);
          commit(s_empty, leader);
        }
        if (c > 0) {
          const int q = g + c - 1;
          mbar_wait(&h_full[q & 1], (q >> 1) & 1, 158);
          const uint32_t b_lo = ring.wait(), h = tmem_base + TM_AB + (q & 1) * 128;
          if (leader) {
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16_ts2(tmem_base + TM_OUT, h + k * 8, b_lo + 2 * k, kDescHiSw128, kIdesc, (c > 1 || k > 0) ? 1u : 0u);
          }
          ring.done(leader);
        }
      }
      commit(out_full, leader);
      g += chunks;
    }
  } else if (warp >= 8) {
    produce_cond<CF32>(p, smem + L::S_OFF, s_full, s_empty);
  } else {
    const int grp = warp >> 2, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const bool leader = (threadIdx.x & 127) == 0;
    uint8_t* xt = smem + L::X_OFF + grp * kOperandTile;  // the group's 64 channels
    float* xch = reinterpret_cast<float*>(smem + L::XCH_OFF);
    const uint32_t tm = tmem_addr(tmem_base, quarter * 32, grp * 64);
    const uint32_t d1 = tmem_addr(tmem_base, quarter * 32, TM_AB + grp * 128);
    int tile = blockIdx.x, g0 = 0;
    for (int i = 0; i < my_tiles; ++i, tile += gridDim.x, g0 += chunks) {
      {  // x1 = x + gamma1 (W_o og), kept in the tile; y into tensor memory
        float v[64];
        mbar_wait(x_full, i & 1, 159);
        mbar_wait(p1_full, i & 1, 160);
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float ga[16], o[16];
          tmem_ld_32x16_f(tm + k * 16, ga);
          tmem_ld_32x16_f(tm + 128 + k * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float4* px = reinterpret_cast<float4*>(xt + (k >> 1) * kOperandHalf + sw128_offset(r, (k & 1) * 4 + q));
            const float4 bg = *reinterpret_cast<const float4*>(bias + 2 * 128 + grp * 64 + k * 16 + q * 4);
            float4 f = *px;
            f.x = fmaf(ga[q * 4] + bg.x, o[q * 4], f.x), f.y = fmaf(ga[q * 4 + 1] + bg.y, o[q * 4 + 1], f.y);
            f.z = fmaf(ga[q * 4 + 2] + bg.z, o[q * 4 + 2], f.z), f.w = fmaf(ga[q * 4 + 3] + bg.w, o[q * 4 + 3], f.w);
            *px = f;
            v[k * 16 + q * 4] = f.x, v[k * 16 + q * 4 + 1] = f.y, v[k * 16 + q * 4 + 2] = f.z, v[k * 16 + q * 4 + 3] = f.w;
          }
        }
        const float rstd = center_row(v, xch, grp, r, p.eps);  // (its barriers: both groups have read gamma1, which y goes over)
        mbar_wait(p2_full, i & 1, 161);
        tc_fence_after_sync();
        // half of y: see the SwiGLU below
        adaptive_norm(v, rstd, 0.5f * p.lns, tm + TM_AB, tm + TM_AB + 128, bias + 3 * 128 + grp * 64, bias + 4 * 128 + grp * 64,
                      tmem_addr(tmem_base, quarter * 32, grp * 32));
        tc_fence_before_sync();
        mbar_arrive(y_full);
      }
      // With a' = fc1(y) / 2 and b' = fc2(y) / 2 from the halved operand: silu(a) b = u + u tanh(a'), u = 2 a' b'.
      for (int c = (g0 & 1) ^ grp; c < chunks; c += 2) {
        const int g = g0 + c;
        mbar_wait(&d1_full[grp], (g >> 1) & 1, 162);
        tc_fence_after_sync();
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t av[32], bv[32], o[16];
          tmem_ld_32x32(d1 + half * 32, av);
          tmem_ld_32x32(d1 + 64 + half * 32, bv);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float a0 = __uint_as_float(av[2 * e]), a1 = __uint_as_float(av[2 * e + 1]);
            const float u0 = (a0 + a0) * __uint_as_float(bv[2 * e]), u1 = (a1 + a1) * __uint_as_float(bv[2 * e + 1]);
            o[e] = pack_bf16x2(fmaf(u0, tanh_approx(a0), u0), fmaf(u1, tanh_approx(a1), u1));
          }
          tmem_st_32x16(d1 + half * 16, o);  // over fc1 columns read before
        }
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(&h_full[grp]);
      }
      // out = x1 + gamma2 h
      mbar_wait(out_full, i & 1, 163);
      tc_fence_after_sync();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float ga[16], o[16];
        tmem_ld_32x16_f(tm + k * 16, ga);
        tmem_ld_32x16_f(tm + TM_OUT + k * 16, o);
        tmem_ld_wait();
        if (k == 3) {
          tc_fence_before_sync();
          mbar_arrive(out_empty);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float4* px = reinterpret_cast<float4*>(xt + (k >> 1) * kOperandHalf + sw128_offset(r, (k & 1) * 4 + q));
          const float4 bg = *reinterpret_cast<const float4*>(bias + 5 * 128 + grp * 64 + k * 16 + q * 4);
          float4 f = *px;
          f.x = fmaf(ga[q * 4] + bg.x, o[q * 4], f.x), f.y = fmaf(ga[q * 4 + 1] + bg.y, o[q * 4 + 1], f.y);
          f.z = fmaf(ga[q * 4 + 2] + bg.z, o[q * 4 + 2], f.z), f.w = fmaf(ga[q * 4 + 3] + bg.w, o[q * 4 + 3], f.w);
          *px = f;
        }
      }
      fence_proxy_async_smem();
      named_bar_sync(1 + grp, 128);
      if (leader) {
        for (int k = 0; k < 2; ++k) tma_store_2d(&maps.out, xt + k * kOperandHalf, grp * 64 + k * 32, tile * 128);
        tma_store_commit();
        tma_store_wait_read0();
        mbar_arrive(x_empty);
      }
      __syncwarp();
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
