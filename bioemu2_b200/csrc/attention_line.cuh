// Triangle attention of short lines with the output projection: a CTA takes one line of up to 128 positions, all four heads of 32, and adds
// the projected update into the pair tensor.  Attention and gate as in flash_resident_kernel; a head's gated output goes to shared
// memory as the operand of  out += og W_o^T  instead of through global memory and a product of its own.  An fp32 pair tensor gets the
// sum from the memory (reduce-add); a bf16 one is read, added in fp32 and rounded once, which a reduction in bf16 would do twice.
//
//   warps 0-7    two groups of four softmax warps, heads g and g + 2 one after the other; then 64 output channels each
//   warps 8, 9   MMA issuers of the groups (8 also of the output projection)
//   warps 10, 11 loaders of the groups: a head's Q, K and bias tile as soon as the one before has been multiplied, V^T likewise
//
// One wave of lines, so the time is a line's chain: loads, two heads of a group, projection, output.  Attention and product were two
// launches of 10 and 6.4 us at 64 lines, of which a good half was launch, set-up and drain; this one takes 11.5.  Trunk of 4 blocks, us
// as two / as one: 24 tokens 445 / 433, 64 466 / 445, 110 528 / 482, 128 552 / 496 (a line a CTA beyond one wave would pay its chain
// twice: those lines, and longer ones, keep the two kernels).
#pragma once
#include "attention_resident.cuh"

namespace b200 {

namespace line_attention {
constexpr int NV = 48;                                 // rows of the V^T operand: 32 value rows, one row of ones, 15 of zeros
constexpr uint32_t Q_BYTES = 128 * 32 * 2, V_HALF = NV * 128;
constexpr uint32_t Q_OFF = 0;                          // [2 groups]
constexpr uint32_t K_OFF = Q_OFF + 2 * Q_BYTES;        // [2]
constexpr uint32_t V_OFF = K_OFF + 2 * Q_BYTES;        // [2][2 halves]
constexpr uint32_t BIAS_OFF = V_OFF + 4 * V_HALF;      // [2] x 32 KB; at last the output tiles
constexpr uint32_t A_OFF = BIAS_OFF + 2 * kOperandTile;  // gated outputs of all heads, 128 x 128 bf16
constexpr uint32_t W_OFF = A_OFF + kOperandTile;       // W_o
constexpr uint32_t IDENT_OFF = W_OFF + kOperandTile;   // 16 x 16 identity, see flash_resident_kernel
constexpr uint32_t BAR_OFF = IDENT_OFF + 512;
constexpr uint32_t SMEM_BYTES = BAR_OFF + 512 + 1024;
constexpr int THREADS = 384;
constexpr uint32_t TM_GROUP = 256, TM_S = 0, TM_P = 128, TM_O = 192;
}  // namespace line_attention

template <bool F32>
__global__ void __launch_bounds__(384, 1)
line_attention_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmBias,
                      const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmO, const __grid_constant__ FlashParams p) {
  using namespace line_attention;
  constexpr float kNegMasked = -1.0e6f * 1.4426950408889634f;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* w_full = bars;        // TMA
  uint64_t* a_full = bars + 1;    // count 256: every head's output is in A
  uint64_t* out_full = bars + 2;  // commit
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int g = warp < 8 ? warp >> 2 : warp & 1;
  uint64_t* gb = bars + 4 + g * 8;
  uint64_t* qkb_full = gb;        // TMA: Q, K, bias tile
  uint64_t* v_full = gb + 1;      // TMA
  uint64_t* s_full = gb + 2;      // commit: S, bias included; Q, K and the bias tile may be loaded again
  uint64_t* s_empty = gb + 3;     // count 128: the scores have been read
  uint64_t* p_full = gb + 4;      // count 128
  uint64_t* pv_done = gb + 5;     // commit: O; V^T may be loaded again
  uint64_t* z_full = gb + 6;      // TMA: the pair tensor's rows (bf16)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    mbar_init(a_full, 256);
    mbar_init(out_full, 1);
    for (int i = 0; i < 2; ++i) {
      uint64_t* x = bars + 4 + i * 8;
      for (int j = 0; j < 7; ++j) mbar_init(&x[j], (j == 3 || j == 4) ? 128 : 1);
    }
    fence_mbar_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmBias);
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmO);
  }
  if (threadIdx.x < 32) {  // identity: 16-byte unit u = (K chunk c, row i) holds K indices 8c .. 8c+7 of row i
    const int c = threadIdx.x >> 4, i = threadIdx.x & 15;
    uint32_t wds[4] = {0, 0, 0, 0};
    if ((i >> 3) == c) wds[(i & 7) >> 1] = (i & 1) ? 0x3F800000u : 0x00003F80u;
    *reinterpret_cast<uint4*>(smem + IDENT_OFF + c * 256 + i * 16) = make_uint4(wds[0], wds[1], wds[2], wds[3]);
  }
  for (int u = threadIdx.x; u < 4 * 128; u += THREADS) {  // the row of ones and the zeros below each V^T half tile
    const int half = u >> 7, unit = u & 127;
    const uint32_t one2 = unit < 8 ? 0x3F803F80u : 0u;
    *reinterpret_cast<uint4*>(smem + V_OFF + half * V_HALF + 32 * 128 + unit * 16) = make_uint4(one2, one2, one2, one2);
  }
  fence_proxy_async_smem();
  if (warp == 8) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  const int b = blockIdx.x;  // line

  if (warp >= 10) {
    if (lane == 0) {
      for (int it = 0; it < 2; ++it) {
        const int h = g + it * 2;
        if (it > 0) mbar_wait(s_full, 0, 170);
        uint8_t* bb = smem + BIAS_OFF + g * kOperandTile;
        mbar_arrive_expect_tx(qkb_full, 2 * Q_BYTES + kOperandTile);
        tma_load_3d(smem + Q_OFF + g * Q_BYTES, &tmQ, qkb_full, p.q_col0 + h * 32, 0, b);
        tma_load_3d(smem + K_OFF + g * Q_BYTES, &tmQ, qkb_full, p.k_col0 + h * 32, 0, b);
        tma_load_3d(bb, &tmBias, qkb_full, 0, 0, h);
        tma_load_3d(bb + kOperandHalf, &tmBias, qkb_full, 64, 0, h);
        if (it > 0) mbar_wait(pv_done, 0, 171);
        uint8_t* vb = smem + V_OFF + g * 2 * V_HALF;
        mbar_arrive_expect_tx(v_full, 2 * 32 * 128);
        tma_load_3d(vb, &tmV, v_full, 0, p.v_row0 + h * 32, b);
        tma_load_3d(vb + V_HALF, &tmV, v_full, 64, p.v_row0 + h * 32, b);
        if (it == 0 && g == 0) {
          mbar_arrive_expect_tx(w_full, kOperandTile);
          tma_load_2d(smem + W_OFF, &tmW, w_full, 0, 0);
          tma_load_2d(smem + W_OFF + kOperandHalf, &tmW, w_full, 64, 0);
        }
      }
      if (!F32) {
        mbar_wait(s_full, 1, 181);  // the second head's bias tile has been multiplied
        mbar_arrive_expect_tx(z_full, kOperandHalf);
        tma_load_3d(smem + BIAS_OFF + g * kOperandTile, &tmO, z_full, g * 64, 0, b);
      }
    }
  } else if (warp >= 8) {
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128), idesc_o = make_idesc_bf16(128, NV), idesc_b = make_idesc_bf16(128, 16);
    const uint32_t base = smem_u32(smem);
    const uint32_t z_lo = desc_lo(base + IDENT_OFF, 256);
    const uint32_t q_lo = desc_lo(base + Q_OFF + g * Q_BYTES), k_lo = desc_lo(base + K_OFF + g * Q_BYTES);
    const uint32_t b_lo = desc_lo(base + BIAS_OFF + g * kOperandTile), v_lo = desc_lo(base + V_OFF + g * 2 * V_HALF);
    const uint32_t tg = tmem_base + g * TM_GROUP;
    auto issue_s = [&](int it) {
      mbar_wait(qkb_full, it, 172);
      mbar_wait(s_empty, it ^ 1, 173);  // the first head's scores have been read
      tc_fence_after_sync();
      if (leader) {
#pragma unroll
        for (int k = 0; k < 2; ++k) umma_bf16_ss2(tg + TM_S, q_lo + 2 * k, kDescHiSw64, k_lo + 2 * k, kDescHiSw64, idesc_s, k > 0);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss2(tg + TM_S + 16 * k, b_lo + (k >> 2) * (kOperandHalf >> 4) + (k & 3) * 2, kDescHiSw128, z_lo, desc_hi_noswizzle(128),
                        idesc_b, true);
        umma_commit(s_full);
      }
      __syncwarp();
    };
    issue_s(0);
    for (int it = 0; it < 2; ++it) {
      if (it == 0) issue_s(1);
      mbar_wait(v_full, it, 174);
      mbar_wait(p_full, it, 175);
      tc_fence_after_sync();
      if (leader) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ts2(tg + TM_O, tg + TM_P + k * 8, v_lo + (k >> 2) * (V_HALF >> 4) + (k & 3) * 2, kDescHiSw128, idesc_o, k != 0);
        umma_commit(pv_done);
      }
      __syncwarp();
    }
    if (g == 0) {  // the output projection, over group 0's scores
      mbar_wait(w_full, 0, 176);
      mbar_wait(a_full, 0, 177);
      tc_fence_after_sync();
      if (leader) {
        umma_k128(tmem_base, base + A_OFF, base + W_OFF, idesc_s, false);
        umma_commit(out_full);
      }
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;  // query == TMEM lane
    const bool q_ok = r < p.N;
    const uint32_t tg = tmem_addr(tmem_base, quarter * 32, g * TM_GROUP);
    uint32_t okw[4];  // keys that exist and are unmasked
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int key = u * 32 + lane;
      okw[u] = __ballot_sync(0xffffffffu, key < p.N && p.mask[b * p.mask_row_stride + key * p.mask_key_stride] != 0);
    }
#pragma unroll 1
    for (int it = 0; it < 2; ++it) {
      const int h = g + it * 2;
      uint4 gate_v[4];
      if (q_ok) {
        const __nv_bfloat16* gsrc = p.gate + (long long)b * p.gate_b_stride + (long long)r * p.gate_pitch + p.gate_col0 + h * 32;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(gate_v[c].x), "=r"(gate_v[c].y), "=r"(gate_v[c].z), "=r"(gate_v[c].w)
                       : "l"(gsrc + c * 8));
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) gate_v[c] = make_uint4(0, 0, 0, 0);
      }
      // Softmax as in flash_resident_kernel, one tile of keys: the reference of a row is 0 until a maximum leaves the range.
      float m_ref = 0.f;
      bool shifted = false, only_masked = false;
      mbar_wait(s_full, it, 178);
      tc_fence_after_sync();
      uint32_t rare = (okw[0] & okw[1]) != 0xffffffffu ? 1u : 0u;
      if ((okw[2] & okw[3]) != 0xffffffffu) rare |= 2u;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        float v[64];
        tmem_ld_32x32_f(tg + TM_S + half * 64, v);
        tmem_ld_32x32_f(tg + TM_S + half * 64 + 32, v + 32);
        tmem_ld_wait();
        if (half == 1) {
          tc_fence_before_sync();
          mbar_arrive(s_empty);
        }
        bool redo = (rare >> half) & 1u;
        if (!redo) {
          uint32_t pk[32];
          const float mc = max64(v);
#pragma unroll
          for (int e = 0; e < 64; e += 2) pk[e >> 1] = pack_bf16x2(exp2_approx(v[e]), exp2_approx(v[e + 1]));
          tmem_st_32x32(tg + TM_P + half * 32, pk);  // (the first head's P.V has completed: its O has been read)
          redo = __any_sync(0xffffffffu, mc > kReferenceHigh || (half == 0 && mc < kReferenceLow));
        }
        if (redo) {
          const uint32_t wa = half ? okw[2] : okw[0], wb = half ? okw[3] : okw[1];
          const bool first = half == 0;
          if ((wa | wb) == 0 && (only_masked || first || !shifted)) {
            if (first) {
              only_masked = shifted = true;
              rare = 3u;
              m_ref = kNegMasked;
            }
            const int ones = only_masked ? p.N - half * 64 : 0;
            uint32_t pk[32];
#pragma unroll
            for (int e = 0; e < 64; e += 2) pk[e >> 1] = (e < ones ? 0x3F80u : 0u) | (e + 1 < ones ? 0x3F800000u : 0u);
            tmem_st_32x32(tg + TM_P + half * 32, pk);
            continue;
          }
          only_masked = false;
          const int left = p.N - half * 64;  // keys from here on exist while j < left
          float y[64];
#pragma unroll
          for (int j = 0; j < 64; ++j) y[j] = (((j < 32 ? wa : wb) >> (j & 31)) & 1u) ? v[j] : (j < left ? kNegMasked : -INFINITY);
          const float mc = max64(y);
          const bool move = mc - m_ref > kReferenceHigh || (first && mc < kReferenceLow);
          if (__any_sync(0xffffffffu, move)) {
            const float scale = move ? exp2_approx(m_ref - mc) : 1.0f;
            tmem_st_wait();
#pragma unroll 1
            for (int c = 0; c < 2 * half; ++c) {
              uint32_t w[16];
              tmem_ld_32x16(tg + TM_P + c * 16, w);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2(bf16lo(w[j]) * scale, bf16hi(w[j]) * scale);
              tmem_st_32x16(tg + TM_P + c * 16, w);
            }
            tmem_st_wait();
            if (move) m_ref = mc;
            shifted = true;
            rare = 3u;
          }
          uint32_t pk[32];
#pragma unroll
          for (int e = 0; e < 64; e += 2) pk[e >> 1] = pack_bf16x2(exp2_approx(y[e] - m_ref), exp2_approx(y[e + 1] - m_ref));
          tmem_st_32x32(tg + TM_P + half * 32, pk);
        }
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(p_full);
      mbar_wait(pv_done, it, 179);
      tc_fence_after_sync();
      float o[32];
      tmem_ld_32x32_f(tg + TM_O, o);
      const float l_row = tmem_ld_32x1_f(tg + TM_O + 32);
      tmem_ld_wait();
      tc_fence_before_sync();
      const float inv_l = __fdividef(1.0f, l_row);
      uint8_t* a_row = smem + A_OFF + (h >> 1) * kOperandHalf;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t gw[4] = {gate_v[c].x, gate_v[c].y, gate_v[c].z, gate_v[c].w};
        uint32_t y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          y[e] = pack_bf16x2(o[c * 8 + 2 * e] * inv_l * bf16lo(gw[e]), o[c * 8 + 2 * e + 1] * inv_l * bf16hi(gw[e]));
        *reinterpret_cast<uint4*>(a_row + sw128_offset(r, (h & 1) * 4 + c)) = make_uint4(y[0], y[1], y[2], y[3]);
      }
    }
    fence_proxy_async_smem();
    mbar_arrive(a_full);
    // ---- output: 64 channels of the projection a group, added into the pair tensor
    mbar_wait(out_full, 0, 180);
    tc_fence_after_sync();
    float v[64];
    const uint32_t o_addr = tmem_addr(tmem_base, quarter * 32, g * 64);
    tmem_ld_32x32_f(o_addr, v);
    tmem_ld_32x32_f(o_addr + 32, v + 32);
    tmem_ld_wait();
    tc_fence_before_sync();
    uint8_t* stage = smem + BIAS_OFF + g * kOperandTile;  // the group's bias tile has been multiplied
    if (F32) {
#pragma unroll
      for (int q = 0; q < 16; ++q)
        *reinterpret_cast<float4*>(stage + (q >> 3) * kOperandHalf + sw128_offset(r, q & 7)) =
            make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
    } else {
      mbar_wait(z_full, 0, 182);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint4* unit = reinterpret_cast<uint4*>(stage + sw128_offset(r, q));
        uint32_t w[4] = {unit->x, unit->y, unit->z, unit->w};
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = pack_bf16x2(v[q * 8 + 2 * e] + bf16lo(w[e]), v[q * 8 + 2 * e + 1] + bf16hi(w[e]));
        *unit = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    fence_proxy_async_smem();
    named_bar_sync(1 + g, 128);
    if ((threadIdx.x & 127) == 0) {
      if (F32) {
        tma_reduce_add_3d(&tmO, stage, g * 64, 0, b);
        tma_reduce_add_3d(&tmO, stage + kOperandHalf, g * 64 + 32, 0, b);
      } else {
        tma_store_3d(&tmO, stage, g * 64, 0, b);
      }
      tma_store_commit();
      tma_store_wait0();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200
