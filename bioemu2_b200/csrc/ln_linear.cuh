// out = W . LayerNorm(x1 | x2) [+ residual], rows of 128 (one source) or 128 + 128 channels (two sources) -> 128 channels fp32:
// the input projection of the pairwise conditioning and the recycling update of the pair tensor.
//
// Both are HBM-bound: as a LayerNorm pass writing bf16 rows and a product reading them, the normalised tensor went through
// memory twice (two sources, N = 384: 97 + 23 us for 226 MB that have to move, 35 us).  Here the LayerNorm writes the product's
// operand in shared memory.  A tile is 128 rows; W stays resident.
//   warps 0-3   epilogue: accumulator (+ residual) -> swizzled staging tiles -> TMA store
//   warps 4-11  producers: 16 threads per row, two (one source: four) rows in flight per thread beside those being normalised
//   warp  12    control: TMA of W, MMA issue
#pragma once
#include "row_tile.cuh"

namespace b200 {

struct LnLinearParams {
  const void* x1;         // [rows][128] fp32 or bf16
  const void* x2;         // [rows][128], second half of the row (two-source form)
  const float* ln_w;      // [128 * sources], may be nullptr
  const float* ln_b;
  const float* residual;  // [rows][128] fp32 or nullptr
  long long rows;
  int num_tiles;
  float eps;
};

template <int SRC>
struct LnLinearCfg {
  static constexpr uint32_t W_OFF = 0;                                // SRC x 32 KB
  static constexpr uint32_t X_OFF = SRC * kOperandTile;               // 2 stages x SRC x 32 KB
  static constexpr uint32_t STAGE_OFF = X_OFF + 2 * SRC * kOperandTile;  // two [128 rows][128 B] output tiles
  static constexpr uint32_t BAR_OFF = STAGE_OFF + 2 * kOperandHalf;
  static constexpr uint32_t SMEM_BYTES = BAR_OFF + 256 + 1024;
  static constexpr int THREADS = 416;
};

template <bool F32, int SRC>
__global__ void __launch_bounds__(416, 1)
ln_linear_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmO, LnLinearParams p) {
  using Cfg = LnLinearCfg<SRC>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* x_full = w_full + 1;       // [2] count 256
  uint64_t* x_empty = x_full + 2;      // [2] commit
  uint64_t* acc_full = x_empty + 2;    // [2] commit
  uint64_t* acc_empty = acc_full + 2;  // [2] count 128
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&x_full[i], 256);
      mbar_init(&x_empty[i], 1);
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 128);
    }
    fence_mbar_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmO);
  }
  if (warp == 12) tmem_alloc(tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 12) {
    const bool leader = elect_one();
    if (leader) {
      mbar_arrive_expect_tx(w_full, SRC * kOperandTile);
      for (int h = 0; h < 2 * SRC; ++h) tma_load_2d(smem + Cfg::W_OFF + h * kOperandHalf, &tmW, w_full, h * 64, 0);
    }
    __syncwarp();
    mbar_wait(w_full, 0, 100);
    constexpr uint32_t idesc = make_idesc_bf16(128, 128);
    const uint32_t w_s = smem_u32(smem + Cfg::W_OFF);
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int s = it & 1;
      mbar_wait(&x_full[s], (it >> 1) & 1, 101);
      mbar_wait(&acc_empty[s], ((it >> 1) & 1) ^ 1, 102);
      tc_fence_after_sync();
      const uint32_t x_s = smem_u32(smem + Cfg::X_OFF + s * SRC * kOperandTile);
      if (leader) {
#pragma unroll
        for (int k = 0; k < SRC; ++k)
          umma_k128(tmem_base + s * 128, x_s + k * kOperandTile, w_s + k * kOperandTile, idesc, k > 0);
        umma_commit(&x_empty[s]);
        umma_commit(&acc_full[s]);
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ producers
    const int pt = threadIdx.x - 128;
    const int c0 = (pt & 15) * 8, rbase = pt >> 4;
    float gamma[SRC][8], beta[SRC][8];
#pragma unroll
    for (int k = 0; k < SRC; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        gamma[k][i] = p.ln_w ? p.ln_w[k * 128 + c0 + i] : 1.0f;
        beta[k][i] = p.ln_b ? p.ln_b[k * 128 + c0 + i] : 0.0f;
      }
    constexpr int U = SRC == 1 ? 4 : 2;  // rows of a thread's group: half of its rows, as far as they fit its registers
    float xa[U][SRC][8], xb[U][SRC][8];
    auto load = [&](int tile, int q, float (&x)[U][SRC][8]) {  // rows (q*U + u)*16 + rbase of the tile
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long row = (long long)tile * 128 + (q * U + u) * 16 + rbase;
#pragma unroll
        for (int k = 0; k < SRC; ++k) {
          if (row < p.rows && tile < p.num_tiles) {
            load8<F32>(static_cast<const uint8_t*>(k ? p.x2 : p.x1) + row * 128 * (long long)zbytes<F32>(), c0, x[u][k]);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[u][k][i] = 0.f;
          }
        }
      }
    };
    auto emit = [&](uint8_t* dst, int q, float (&x)[U][SRC][8]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float sm = 0.f;
#pragma unroll
        for (int k = 0; k < SRC; ++k)
#pragma unroll
          for (int i = 0; i < 8; ++i) sm += x[u][k][i];
        const float mean = group16_sum(sm) * (1.0f / (128 * SRC));
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < SRC; ++k)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            x[u][k][i] -= mean;
            ss = fmaf(x[u][k][i], x[u][k][i], ss);
          }
        const float rstd = rsqrtf(group16_sum(ss) * (1.0f / (128 * SRC)) + p.eps);
        const int r = (q * U + u) * 16 + rbase;
#pragma unroll
        for (int k = 0; k < SRC; ++k) {
          float y[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) y[i] = fmaf(x[u][k][i] * rstd, gamma[k][i], beta[k][i]);
          *reinterpret_cast<uint4*>(dst + k * kOperandTile + ((pt & 15) >> 3) * kOperandHalf + sw128_offset(r, pt & 7)) =
              make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
        }
      }
    };
    int it = 0;
    load(blockIdx.x, 0, xa);
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int s = it & 1;
      uint8_t* dst = smem + Cfg::X_OFF + s * SRC * kOperandTile;
      load(tile, 1, xb);
      mbar_wait(&x_empty[s], ((it >> 1) & 1) ^ 1, 103);
#pragma unroll
      for (int q = 0; q < 8 / U; q += 2) {
        emit(dst, q, xa);
        if (q + 2 < 8 / U) load(tile, q + 2, xa);
        else load(tile + gridDim.x, 0, xa);
        emit(dst, q + 1, xb);
        if (q + 3 < 8 / U) load(tile, q + 3, xb);
      }
      fence_proxy_async_smem();
      mbar_arrive(&x_full[s]);
    }
  } else {
    // ------------------------------------------------------------------ epilogue: lane = row, 32 channels at a time
    const int r = warp * 32 + lane;
    const bool leader = threadIdx.x == 0;
    int it = 0;
    float res[4][8];  // the next 32 channels of the residual, loaded a chunk ahead
    auto load_res = [&](int tile, int c) {
      const long long row = (long long)tile * 128 + r;
      const bool there = p.residual && row < p.rows && tile < p.num_tiles;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if (there) {
          ld_global_v8(p.residual + row * 128 + c * 32 + g * 8, res[g]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) res[g][e] = 0.f;
        }
      }
    };
    load_res(blockIdx.x, 0);
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int acc = it & 1;
      mbar_wait(&acc_full[acc], (it >> 1) & 1, 104);
      tc_fence_after_sync();
      uint32_t va[32], vb[32];
      tmem_ld_32x32(tmem_addr(tmem_base, warp * 32, acc * 128), va);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t(&v)[32] = (c & 1) ? vb : va;
        uint8_t* stage = smem + Cfg::STAGE_OFF + (c & 1) * kOperandHalf;
        tmem_ld_wait();
        if (c < 3) {
          tmem_ld_32x32(tmem_addr(tmem_base, warp * 32, acc * 128 + (c + 1) * 32), (c & 1) ? va : vb);
        } else {
          tc_fence_before_sync();
          mbar_arrive(&acc_empty[acc]);
        }
        if (leader) tma_store_wait_read1();  // the store that last used this staging tile has read it
        named_bar_sync(1, 128);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = res[g][e] + __uint_as_float(v[g * 8 + e]);
          *reinterpret_cast<float4*>(stage + sw128_offset(r, g * 2)) = make_float4(x[0], x[1], x[2], x[3]);
          *reinterpret_cast<float4*>(stage + sw128_offset(r, g * 2 + 1)) = make_float4(x[4], x[5], x[6], x[7]);
        }
        if (c < 3) load_res(tile, c + 1);
        else load_res(tile + gridDim.x, 0);
        fence_proxy_async_smem();
        named_bar_sync(1, 128);
        if (leader) {
          tma_store_2d(&tmO, stage, c * 32, tile * 128);
          tma_store_commit();
        }
      }
    }
    if (leader) tma_store_wait0();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 12) {
    __syncwarp();
    tmem_dealloc(tmem_base, 256);
  }
}

}  // namespace b200
