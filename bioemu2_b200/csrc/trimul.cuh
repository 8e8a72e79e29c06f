// Triangle multiplication, the two kernels either side of the per-channel
// contraction (which is bmm_nt_kernel):
//
//   trimul_in_kernel   h = LN_in(z);  ab = mask * p_in(h) * sigmoid(g_in(h))
//                      written channel-major, a[d][line][pos] / b[d][line][pos] (bf16, pitch Np),
//                      so that the contraction reads K-major rows.  The product is computed
//                      transposed -- weights are the M operand, the pair tile the N operand -- so
//                      a TMEM lane is an output channel and each thread stores contiguous pairs.
//   trimul_out_kernel  out = p_out(LN_out(t)) * sigmoid(g_out(LN_in(z))) [+ z]
//                      reading t channel-major and writing the pair-major result.
//
// "line/pos": outgoing contracts the column index, a[d][i][k] = ab[i,k,d]; incoming contracts the
// row index, a[d][i][k] = ab[k,i,d].  A tile is two runs of 64 consecutive `pos`, each on one `line`.
#pragma once
#include "row_tile.cuh"

namespace b200 {

// Geometry is given as lines x positions over a (possibly rectangular, possibly strided) slab of the pair
// tensor: pair (line, pos) sits at z + line*z_line_stride + pos*z_pos_stride (bytes), its mask byte at
// mask + line*m_line_stride + pos*m_pos_stride.  Outgoing: line = row, pos = column; incoming: line =
// column, pos = row.
struct TriMulInParams {
  const void* z;           // z stream (fp32 or bf16), 128 channels per pair
  const uint8_t* mask;     // non-zero = valid
  const float* ln_w;
  const float* ln_b;
  long long z_copy_delta;  // byte distance from z to a tensor that receives a copy of it (0: none)
  __nv_bfloat16* a_out;    // [128][lines_alloc][pos_pitch]
  __nv_bfloat16* b_out;
  int n_lines, n_pos;
  int lines_alloc, pos_pitch;  // pos_pitch: multiple of 128 >= n_pos
  long long z_line_stride, z_pos_stride;
  long long m_line_stride, m_pos_stride;
  int half_tiles;          // a line's half tiles of 64 positions; a tile is two consecutive ones, of one line or of two
  int num_tiles;           // ceil(n_lines * half_tiles / 2)
  float eps;
};

namespace trimul_in {
constexpr uint32_t W_OFF = 0;                       // 4 M-tiles x 32 KB
constexpr uint32_t X_OFF = 4 * kOperandTile;        // 2 stages x 32 KB
constexpr uint32_t MASK_OFF = X_OFF + 2 * kOperandTile;  // 4 stages x 128 B
constexpr uint32_t BAR_OFF = MASK_OFF + 4 * 128;
constexpr uint32_t FLAG_OFF = BAR_OFF + 96;          // 4 stages x 4 "every pair of this quarter valid" bytes
constexpr uint32_t STAGE_OFF = MASK_OFF + 1024;      // per epilogue group a 16 KB tile [128 channels][64 pairs]
constexpr uint32_t SMEM_BYTES = STAGE_OFF + 2 * kOperandHalf + 1024;
constexpr int THREADS = 512;  // warps 0-3 epilogue of pairs 0-63, 4-7 of pairs 64-127, 8-15 producers (8 issues the MMAs)
}  // namespace trimul_in

// The LayerNorm output is halved (exactly) before the projections, so the accumulators hold p/2 and g/2
// and the gate is p * sigmoid(g) = p/2 + p/2 * tanh(g/2): one MUFU and one FMA per element.
// 512 threads, not 544: a 17th warp would round the register allocation up to 640 threads and cap every
// thread at 96 registers, which the LayerNorm producers spill at.  So there is no control warp: one of the producers issues.
// p and g of one half (a or b) are 256 TMEM columns, so the two halves of a tile double-buffer each other: both epilogue
// groups drain a half together, 64 pairs each, while the other half's products run (with a group per half, whose products
// had to wait for its own drain, a tile was a chain of products, drain and store: 78.5 us at N = 512).
// COPY: the producers also store the raw rows at z_copy_delta from their source.  The first op of a stack that leaves its
// input alone gets its working copy this way, for the write alone (N = 384: 26 us as a copy of its own before the stack).
template <bool F32, bool COPY, bool HALF>
__global__ void __launch_bounds__(512, 1)
trimul_in_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA,
                 const __grid_constant__ CUtensorMap tmB, TriMulInParams p) {
  using namespace trimul_in;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* x_full = w_full + 1;     // [2]
  uint64_t* x_empty = x_full + 2;    // [2]
  uint64_t* acc_full = x_empty + 2;  // [2]  a-half, b-half
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  uint8_t* mask_s = smem + MASK_OFF;
  uint8_t* flag_s = smem + FLAG_OFF;

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&x_full[i], 256);
      mbar_init(&x_empty[i], 1);
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 256);
    }
    fence_mbar_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp >= 8) {
    // ------------------------------------------------------------------ producers
    const int pt = threadIdx.x - 256;  // 0..255
    float gamma[8], beta[8];
    load_gamma_beta(p.ln_w, p.ln_b, pt, gamma, beta, 0.5f);
    const long long pos_stride = p.z_pos_stride, line_stride = p.z_line_stride;
    const long long mpos_stride = p.m_pos_stride, mline_stride = p.m_line_stride;
    // Warps 9-15 have nine pairs of rows each, warp 8 the last pair: it is the issuer (all its lanes wait on the barriers and
    // one elected lane issues -- a converged warp issues a tcgen05.mma several times faster than a lone thread of a diverged
    // one).  The tensor pipe takes only a few products ahead, so the issuing warp stands still for most of their time: as
    // one of the epilogue's warps it held up its whole group.
    const bool issuer = warp == 8;
    constexpr int G = 3;
    RowStream<F32, G, 3> rows;
    rows.c16 = lane & 15;
    rows.first = (issuer ? 126 : (warp - 9) * 2) + (lane >> 4);
    rows.step = 14;
    const int groups = issuer ? 1 : G;
    uint8_t mreg = 0;
    auto row_ptr = [&](int tile) { return TileRuns<HALF>(tile, p.half_tiles, p.n_lines).rows(p.z, p.n_pos, line_stride, pos_stride); };
    auto load_mask = [&](int tile) {
      if (pt < 128) {
        const TileRuns<HALF> t(tile, p.half_tiles, p.n_lines);
        const int k = pt >> 6, pos = t.pos_of(k) + (pt & 63);
        mreg = (k == 0 || t.there1) && pos < p.n_pos ? p.mask[t.line_of(k) * mline_stride + pos * mpos_stride] : 0;
      }
    };
    // Tile number `it` into its operand stage, and the loads of the block's next tile on their way.
    auto produce = [&](int tile, int it) {
      const int s = it & 1;
      const int next = tile + gridDim.x;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g >= groups) break;
        if (COPY) rows.copy(g, row_ptr(tile), p.z_copy_delta);
        rows.normalize(g, gamma, beta, p.eps);
        if (g == 0) mbar_wait(&x_empty[s], ((it >> 1) & 1) ^ 1, 13);
        rows.store(g, smem + X_OFF + s * kOperandTile);
        if (next < p.num_tiles) rows.load(g, row_ptr(next));
      }
      if (pt < 128) {
        mask_s[(it & 3) * 128 + pt] = mreg;
        const bool quarter_valid = __all_sync(0xffffffffu, mreg != 0);
        if (lane == 0) flag_s[(it & 3) * 4 + (pt >> 5)] = quarter_valid ? 1 : 0;
      }
      fence_proxy_async_smem();
      mbar_arrive(&x_full[s]);
      if (next < p.num_tiles) load_mask(next);
    };
    int tile = blockIdx.x;
    if (tile < p.num_tiles) {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (g < groups) rows.load(g, row_ptr(tile));
      load_mask(tile);
    }
    if (!issuer) {
      for (int it = 0; tile < p.num_tiles; tile += gridDim.x, ++it) produce(tile, it);
    } else if (tile < p.num_tiles) {
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(128, 128);
      const uint32_t w_s = smem_u32(smem + W_OFF);
      if (leader) {
        mbar_arrive_expect_tx(w_full, 4 * kOperandTile);
        for (int mt = 0; mt < 4; ++mt)
          for (int h = 0; h < 2; ++h)
            tma_load_2d(smem + W_OFF + mt * kOperandTile + h * kOperandHalf, &tmW, w_full, h * 64, mt * 128);
      }
      __syncwarp();
      produce(tile, 0);
      mbar_wait(w_full, 0, 10);
      for (int it = 0; tile < p.num_tiles; tile += gridDim.x, ++it) {
        const int s = it & 1;
        const uint32_t x_s = smem_u32(smem + X_OFF + s * kOperandTile);
        mbar_wait(&x_full[s], (it >> 1) & 1, 11);
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {  // p and g products of one half
          mbar_wait(&acc_empty[half], (it & 1) ^ 1, 12);  // both groups have drained this half of the previous tile
          tc_fence_after_sync();
          if (leader) {
            umma_k128(tmem_base + (half * 2) * 128, w_s + (half * 2) * kOperandTile, x_s, idesc, false);
            umma_k128(tmem_base + (half * 2 + 1) * 128, w_s + (half * 2 + 1) * kOperandTile, x_s, idesc, false);
            umma_commit(&acc_full[half]);
            if (half == 1) umma_commit(&x_empty[s]);
          }
          __syncwarp();
          // with products in the pipe, this warp's own rows of the next tile
          if (half == 0 && tile + int(gridDim.x) < p.num_tiles) produce(tile + gridDim.x, it + 1);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    // Lane = channel, columns = pairs; 16 columns at a time with the next chunk's TMEM loads in flight.  The gated
    // values go to the group's swizzled [128 channels][64 pairs] staging tile and leave by TMA store (a row
    // per channel of the channel-major plane).
    const int grp = warp >> 2;
    const int d = (warp & 3) * 32 + lane;  // channel inside the half == TMEM lane
    uint8_t* stage = smem + STAGE_OFF + grp * kOperandHalf;
    const uint32_t acc_addr = tmem_addr(tmem_base, (warp & 3) * 32, grp * 64);
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const TileRuns<HALF> t(tile, p.half_tiles, p.n_lines);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        mbar_wait(&acc_full[half], it & 1, 14);
        tc_fence_after_sync();
        const uint32_t* msk = reinterpret_cast<const uint32_t*>(mask_s + (it & 3) * 128 + grp * 64);
        // every pair of the tile unmasked?  (tiles away from the padding are, and then no select is needed)
        const bool all_valid = *reinterpret_cast<const uint32_t*>(flag_s + (it & 3) * 4) == 0x01010101u;
        const uint32_t p_addr = acc_addr + half * 256, g_addr = p_addr + 128;
        uint32_t pa[16], ga[16], pb[16], gb[16];
        tmem_ld_32x16(p_addr, pa);
        tmem_ld_32x16(g_addr, ga);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t(&pv)[16] = (c & 1) ? pb : pa;
          uint32_t(&gv)[16] = (c & 1) ? gb : ga;
          tmem_ld_wait();
          if (c < 3) {
            tmem_ld_32x16(p_addr + (c + 1) * 16, (c & 1) ? pa : pb);
            tmem_ld_32x16(g_addr + (c + 1) * 16, (c & 1) ? ga : gb);
          } else {
            tc_fence_before_sync();
            mbar_arrive(&acc_empty[half]);
          }
          uint32_t packed[8];
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float h0 = __uint_as_float(pv[j]), h1 = __uint_as_float(pv[j + 1]);
            float v0 = fmaf(h0, tanh_approx(__uint_as_float(gv[j])), h0);
            float v1 = fmaf(h1, tanh_approx(__uint_as_float(gv[j + 1])), h1);
            if (!all_valid) {
              const uint32_t m4 = msk[(c * 16 + j) >> 2];
              v0 = ((m4 >> ((j & 3) * 8)) & 0xff) ? v0 : 0.f;
              v1 = ((m4 >> (((j + 1) & 3) * 8)) & 0xff) ? v1 : 0.f;
            }
            packed[j >> 1] = pack_bf16x2(v0, v1);
          }
          if (c == 0) {  // the previous store has finished reading the staging tile (its wait hides behind the
            if (d == 0) tma_store_wait_read0();  // chunk's arithmetic above)
            named_bar_sync(1 + grp, 128);
          }
          *reinterpret_cast<uint4*>(stage + sw128_offset(d, c * 2)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          *reinterpret_cast<uint4*>(stage + sw128_offset(d, c * 2 + 1)) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        }
        fence_proxy_async_smem();
        named_bar_sync(1 + grp, 128);
        if (d == 0) {
          if (grp == 0 || t.there1) tma_store_3d(half ? &tmB : &tmA, stage, t.pos_of(grp), t.line_of(grp), 0);
          tma_store_commit();
        }
      }
    }
    if (d == 0) tma_store_wait0();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------

// Same lines x positions geometry as TriMulInParams; t is [128][lines_alloc][pos_pitch] (tensor map) and is
// indexed by (line, pos), so a transposed t goes with line = column, pos = row.
struct TriMulOutParams {
  const void* z;           // z stream: input of the op (gate and, optionally, residual)
  void* out;               // same dtype and strides as z, may alias it
  const float* ln_in_w;
  const float* ln_in_b;
  const float* ln_out_w;
  const float* ln_out_b;
  int n_lines, n_pos, pos_pitch;
  long long z_line_stride, z_pos_stride;
  int half_tiles, num_tiles;  // as in TriMulInParams
  int add_residual;
  int pos_is_dim1;         // the output tensor map is {channel, pos, line} (1) or {channel, line, pos} (0)
  float eps;
};

namespace trimul_out {
constexpr uint32_t W_OFF = 0;                          // p_out, g_out: 2 x 32 KB
constexpr uint32_t T_OFF = 2 * kOperandTile;           // raw t tiles [2 halves][128 d][64 j], 2 stages
constexpr uint32_t A1_OFF = T_OFF + 2 * kOperandTile;  // LN_out(t) operand
constexpr uint32_t A2_OFF = A1_OFF + kOperandTile;     // LN_in(z) operand
constexpr uint32_t LN_OFF = A2_OFF + kOperandTile;     // gamma_out[128], beta_out[128] fp32
constexpr uint32_t BAR_OFF = LN_OFF + 1024;
constexpr uint32_t STAGE_OFF = LN_OFF + 2048;          // 2 x 16 KB output tiles [128 pairs][128 B of channels]
constexpr uint32_t SMEM_BYTES = STAGE_OFF + 2 * kOperandHalf + 1024;
constexpr int THREADS = 512;  // warps 0-3 epilogue (thread 0 also issues the TMA loads and MMAs), 4-7 t transformers, 8-15 z producers
}  // namespace trimul_out

template <bool F32, bool HALF>
__global__ void __launch_bounds__(512, 1)
trimul_out_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmT,
                  const __grid_constant__ CUtensorMap tmO, TriMulOutParams p) {
  using namespace trimul_out;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* t_full = w_full + 1;     // [2] TMA landed a raw t tile
  uint64_t* t_empty = t_full + 2;    // [2] transformers are done with it
  uint64_t* a1_full = t_empty + 2;   // LN_out(t) operand written
  uint64_t* a2_full = a1_full + 1;   // LN_in(z) operand written
  uint64_t* a_empty = a2_full + 1;   // both operands consumed by the MMAs
  uint64_t* acc_full = a_empty + 1;  // [2]
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  float* ln_s = reinterpret_cast<float*>(smem + LN_OFF);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&t_full[i], 1);
      mbar_init(&t_empty[i], 128);
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 128);
    }
    mbar_init(a1_full, 128);
    mbar_init(a2_full, 256);
    mbar_init(a_empty, 1);
    fence_mbar_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmT);
    prefetch_tmap(&tmO);
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  if (threadIdx.x < 128) {
    ln_s[threadIdx.x] = p.ln_out_w[threadIdx.x];
    ln_s[128 + threadIdx.x] = p.ln_out_b[threadIdx.x];
  }
  __syncthreads();

  if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ t transformers
    // The raw tile is [d][j] (channel-major, as the contraction writes it); LayerNorm runs over d and the result is row j of A1.  A warp
    // has 32 pair columns: transposing matrix loads give a lane 4 columns x 32 channels (channels 8k + 2 (lane % 4) and the next,
    // columns 8m + lane / 4), which stay in its registers from the sums to the matrix stores of the operand's rows.  (Two passes of
    // 32-bit loads, two columns and 64 channels a lane, took the kernel 42.2 us instead of 39.8 at 384 tokens, 10.3 instead of 9.9 at
    // a tile a CTA.  On an unswizzled tile the eight rows of a matrix share their banks: 47.  These warps draining half of the channels
    // besides, through one staging tile a group: 41.)
    const int tw = warp - 4;
    const uint32_t src = smem_u32(smem + T_OFF) + (tw >> 1) * kOperandHalf + sw128_offset(lane & 7, (tw & 1) * 4 + (lane >> 3));
    const uint32_t dst = smem_u32(smem + A1_OFF);
    const uint32_t ln_addr = smem_u32(ln_s) + (lane & 3) * 8;
    const int jr = tw * 32 + lane;  // the operand row this lane addresses in the matrix stores
    int it = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++it) {
      const int s = it & 1;
      mbar_wait(&t_full[s], (it >> 1) & 1, 25);
      uint32_t v[16][4];
#pragma unroll
      for (int k = 0; k < 16; ++k)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[k][0]), "=r"(v[k][1]), "=r"(v[k][2]), "=r"(v[k][3])
                     : "r"(src + s * kOperandTile + k * 1024)
                     : "memory");
      mbar_arrive(&t_empty[s]);
      float mean[4], rstd[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          add_f32x2(a0, a1, bf16lo(v[k][m]), bf16hi(v[k][m]));
          add_f32x2(b0, b1, bf16lo(v[k + 1][m]), bf16hi(v[k + 1][m]));
        }
        mean[m] = (a0 + a1) + (b0 + b1);
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1)
#pragma unroll
        for (int m = 0; m < 4; ++m) mean[m] += __shfl_xor_sync(0xffffffffu, mean[m], o);
      // (the values are unpacked anew in each pass: kept unpacked they would not fit the registers)
#pragma unroll
      for (int k = 0; k < 16; ++k)
#pragma unroll
        for (int m = 0; m < 4; ++m) asm volatile("" : "+r"(v[k][m]));
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        mean[m] *= 1.0f / kD;
        float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          float x0 = bf16lo(v[k][m]), x1 = bf16hi(v[k][m]), y0 = bf16lo(v[k + 1][m]), y1 = bf16hi(v[k + 1][m]);
          add_f32x2(x0, x1, -mean[m], -mean[m]);
          add_f32x2(y0, y1, -mean[m], -mean[m]);
          fma_f32x2(a0, a1, x0, x1, x0, x1, a0, a1);
          fma_f32x2(b0, b1, y0, y1, y0, y1, b0, b1);
        }
        rstd[m] = (a0 + a1) + (b0 + b1);
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1)
#pragma unroll
        for (int m = 0; m < 4; ++m) rstd[m] += __shfl_xor_sync(0xffffffffu, rstd[m], o);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        rstd[m] = rsqrtf(rstd[m] * (1.0f / kD) + p.eps);
        mean[m] *= -rstd[m];
      }
#pragma unroll
      for (int k = 0; k < 16; ++k)
#pragma unroll
        for (int m = 0; m < 4; ++m) asm volatile("" : "+r"(v[k][m]));
      mbar_wait(a_empty, (it & 1) ^ 1, 26);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        float2 g, bb;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(g.x), "=f"(g.y) : "r"(ln_addr + k * 32) : "memory");
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(bb.x), "=f"(bb.y) : "r"(ln_addr + 512 + k * 32) : "memory");
        uint32_t o[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          float x0 = bf16lo(v[k][m]), x1 = bf16hi(v[k][m]);
          fma_f32x2(x0, x1, x0, x1, rstd[m], rstd[m], mean[m], mean[m]);
          fma_f32x2(x0, x1, x0, x1, g.x, g.y, bb.x, bb.y);
          o[m] = pack_bf16x2(x0, x1);
        }
        asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(
                         dst + (k >> 3) * kOperandHalf + sw128_offset(jr, k & 7)),
                     "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                     : "memory");
      }
      fence_proxy_async_smem();
      mbar_arrive(a1_full);
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ z producers: LN_in(z) -> A2
    const int pt = threadIdx.x - 256;  // 0..255
    float gamma[8], beta[8];
    load_gamma_beta(p.ln_in_w, p.ln_in_b, pt, gamma, beta);
    RowTile<256> regs;
    auto load_tile = [&](int tile) {
      regs.template load<F32, true, 8>(
          pt, TileRuns<HALF>(tile, p.half_tiles, p.n_lines).rows(p.z, p.n_pos, p.z_line_stride, p.z_pos_stride), gamma, beta, p.eps);
    };
    int it = 0;
    int tile = blockIdx.x;
    if (tile < p.num_tiles) load_tile(tile);
    for (; tile < p.num_tiles; tile += gridDim.x, ++it) {
      mbar_wait(a_empty, (it & 1) ^ 1, 27);
      regs.store_operand(pt, smem + A2_OFF);
      fence_proxy_async_smem();
      mbar_arrive(a2_full);
      const int next = tile + gridDim.x;
      if (next < p.num_tiles) load_tile(next);
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    // Lane = pair, columns = channels.  16 channels at a time with the next chunk's TMEM loads in flight; the
    // gated update goes to a swizzled [128 pairs][128 B] staging tile and leaves by TMA, two tiles in
    // rotation: added into z in place when the residual is wanted and out aliases z (a bulk reduce, so z is
    // not read here), stored otherwise (with the residual added here from global memory if it is wanted).
    constexpr int CPS = F32 ? 2 : 4;  // 16-channel chunks per staging tile (128 B of channels per pair)
    const int r = warp * 32 + lane;   // pair row of the tile == TMEM lane
    const bool reduce = p.add_residual && p.out == p.z;
    const bool read_res = p.add_residual && !reduce;
    // There is no control warp (a 17th warp would cap every thread at 96 registers): thread 0 issues the TMA
    // loads of the weights and the raw t tiles and, in step i, the two products of tile i; the four warps then
    // drain tile i - 1, whose products ran while tile i's operands were being written.
    constexpr uint32_t idesc = make_idesc_bf16(128, 128);
    const uint32_t w_s = smem_u32(smem + W_OFF);
    const uint32_t a1_s = smem_u32(smem + A1_OFF);
    const uint32_t a2_s = smem_u32(smem + A2_OFF);
    auto issue_t = [&](int tile, int s) {
      mbar_arrive_expect_tx(&t_full[s], kOperandTile);
      const TileRuns<HALF> t(tile, p.half_tiles, p.n_lines);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        tma_load_3d(smem + T_OFF + s * kOperandTile + k * kOperandHalf, &tmT, &t_full[s], t.pos_of(k), t.line_of(k), 0);
    };
    int my_tiles = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x) ++my_tiles;
    // Warp 0 as a whole waits on the barriers; one elected lane issues the loads and the products (a converged warp
    // issues a tcgen05.mma several times faster than a lone thread of a diverged one).
    const bool leader = warp == 0 && elect_one();
    if (warp == 0) {
      if (leader) {
        mbar_arrive_expect_tx(w_full, 2 * kOperandTile);
        for (int mt = 0; mt < 2; ++mt)
          for (int h = 0; h < 2; ++h)
            tma_load_2d(smem + W_OFF + mt * kOperandTile + h * kOperandHalf, &tmW, w_full, h * 64, mt * 128);
        if (my_tiles > 0) issue_t(blockIdx.x, 0);          // first two t tiles in flight
        if (my_tiles > 1) issue_t(blockIdx.x + gridDim.x, 1);
      }
      __syncwarp();
      mbar_wait(w_full, 0, 20);
    }
    __syncwarp();
    for (int step = 0; step <= my_tiles; ++step) {
      if (warp == 0 && step < my_tiles) {
        const int acc = step & 1;
        mbar_wait(&acc_empty[acc], ((step >> 1) & 1) ^ 1, 21);
        mbar_wait(a1_full, step & 1, 22);
        mbar_wait(a2_full, step & 1, 23);
        tc_fence_after_sync();
        if (leader) {
          umma_k128(tmem_base + acc * 256, a1_s, w_s, idesc, false);                       // p_out(LN_out(t))
          umma_k128(tmem_base + acc * 256 + 128, a2_s, w_s + kOperandTile, idesc, false);  // g_out(LN_in(z))
          umma_commit(a_empty);
          umma_commit(&acc_full[acc]);
        }
        __syncwarp();
        if (step + 2 < my_tiles) {  // refill the raw-t stage this tile used, once the transformers have released it
          mbar_wait(&t_empty[step & 1], (step >> 1) & 1, 24);
          if (leader) issue_t(blockIdx.x + (step + 2) * gridDim.x, step & 1);
        }
      }
      __syncwarp();
      if (step == 0) continue;
      const int it = step - 1;
      const int tile = blockIdx.x + it * gridDim.x;
      const TileRuns<HALF> t(tile, p.half_tiles, p.n_lines);
      const int run = HALF ? r >> 6 : 0;  // the lane's
      const int line = run ? t.line[1] : t.line[0], pos0 = run ? t.pos0[1] : t.pos0[0];
      const bool sender = (r & (HALF ? 63 : 127)) == 0;  // sends its run's rows off
      const int acc = it & 1;
      const int pos = HALF ? pos0 + (r & 63) : pos0 + r;
      const bool valid = (run == 0 || t.there1) && pos < p.n_pos;
      const uint8_t* zrow = static_cast<const uint8_t*>(p.z) + line * p.z_line_stride + pos * p.z_pos_stride;
      mbar_wait(&acc_full[acc], (it >> 1) & 1, 28);
      tc_fence_after_sync();
      const uint32_t p_addr = tmem_addr(tmem_base, warp * 32, acc * 256);
      const uint32_t g_addr = p_addr + 128;
      uint32_t pa[16], ga[16], pb[16], gb[16];
      tmem_ld_32x16(p_addr, pa);
      tmem_ld_32x16(g_addr, ga);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint8_t* stage = smem + STAGE_OFF + ((c / CPS) & 1) * kOperandHalf;
        if (c % CPS == 0) {  // the store that last used this staging tile has finished reading it
          if (sender) tma_store_wait_read1();
          named_bar_sync(1, 128);
        }
        uint32_t(&pv)[16] = (c & 1) ? pb : pa;
        uint32_t(&gv)[16] = (c & 1) ? gb : ga;
        tmem_ld_wait();
        if (c < 7) {
          tmem_ld_32x16(p_addr + (c + 1) * 16, (c & 1) ? pa : pb);
          tmem_ld_32x16(g_addr + (c + 1) * 16, (c & 1) ? ga : gb);
        } else {
          tc_fence_before_sync();
          mbar_arrive(&acc_empty[acc]);
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float x[8];
          if (read_res && valid) {
            load8<F32>(zrow, c * 16 + g * 8, x);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = 0.f;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e)
            x[e] = fmaf(__uint_as_float(pv[g * 8 + e]), sigmoid_fast(__uint_as_float(gv[g * 8 + e])), x[e]);
          if (F32) {
            const int k = (c % CPS) * 4 + g * 2;
            *reinterpret_cast<float4*>(stage + sw128_offset(r, k)) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4*>(stage + sw128_offset(r, k + 1)) = make_float4(x[4], x[5], x[6], x[7]);
          } else {
            *reinterpret_cast<uint4*>(stage + sw128_offset(r, (c % CPS) * 2 + g)) = make_uint4(
                pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
          }
        }
        if (c % CPS == CPS - 1) {
          fence_proxy_async_smem();
          named_bar_sync(1, 128);
          if (sender) {
            const int ch0 = (c / CPS) * (F32 ? 32 : 64);
            const int c1 = p.pos_is_dim1 ? pos0 : line, c2 = p.pos_is_dim1 ? line : pos0;
            const uint8_t* rows = stage + run * (kOperandHalf / 2);
            if (!valid) {  // (the run's first row is not there)
            } else if (reduce)
              tma_reduce_add_3d(&tmO, rows, ch0, c1, c2);
            else
              tma_store_3d(&tmO, rows, ch0, c1, c2);
            tma_store_commit();  // an empty group too: the waits count groups
          }
        }
      }
    }
    if ((r & (HALF ? 63 : 127)) == 0) tma_store_wait0();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200
