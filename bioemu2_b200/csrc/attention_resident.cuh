// Attention with an additive pair bias for short rows: the same function as flash_core_kernel (attention.cuh), for key rows
// whose whole bias row block fits in shared memory (at most NB tiles of 128 keys).
//
// A CTA has G softmax groups of four warps.  A work item is a "pass": one head, one tile of 128 queries and G consecutive
// batch items ("lines") that share the bias; group g takes line g.  The bias row block of a (head, query tile) stays in
// shared memory for all lines, so per line only Q, K and V^T are read; flash_core_kernel loads it again for every line, and
// its groups are two query tiles of one line, so rows of up to 128 tokens leave the second group idle.  The groups run
// through their tile streams independently (each has its own loader and MMA warp): while one is between two items the
// other computes.
//
// Tensor memory per group: S (128 fp32 columns), P (64 columns of packed bf16, the A operand of P.V) and the output
// accumulator O (NV columns), which stays there for the whole item.  V^T carries a row of ones below its VR rows, so
// column VR of O is the row sum of P -- the softmax denominator comes out of the same product, from the same rounded P.
//   softmax warps  one thread per query row.  A score tile (bias already added by the tensor core) is read in two halves
//                  and leaves as P = 2^(score - reference), packed bf16.  The reference of a row is 0 until its maximum
//                  leaves a range in which fp32 and bf16 exponents carry everything: so no exponential waits for a maximum,
//                  and the maximum only decides, afterwards, whether a half tile has to be done again.
//   loader warps   one per group: Q once per item, K and V^T through two-stage rings, the key mask of the tile as bits;
//                  group 0's also brings the bias row blocks
//   MMA warps      one per group: S = Q.K^T + bias tile as soon as the softmax threads have read the previous S (the bias
//                  is added by the tensor core: eight 128 x 16 x 16 products of the bias tile's 16-column blocks, as
//                  the A operand, with a 16 x 16 identity, each onto its own 16 accumulator columns); O (+)= P.V as
//                  soon as P is written.  The tile stream runs on across items.
//
// What bounds it: the chain  S full -> read, exponentials, P written -> next S full  of a group, 2,780 clocks a tile of which
// 2,050 would be the special-function pipe's share for both groups, and about 2,500 clocks more at an item's ends (from the
// launches at 256, 384 and 512 keys: 64.8, 193.6 and 407.4 thousand clocks for 6.9, 15.6 and 27.7 items a group).  Against N^3 * 4
// exponentials at 16 per clock and SM that is 0.44 of the floor at 256 keys, 0.49 at 384 and 0.56 at 512.  K and V^T come once
// per query tile: at 512 keys 672 MB are read from DRAM where every operand once would be 270 MB, 0.5 of the copy bandwidth.
// One launch of triangle attention, 4 heads of 32 (ms, flash_core_kernel before -> here): N = 64 0.0143 -> 0.0082,
// 128 0.0184 -> 0.0105, 203 0.0410 -> 0.0323, 256 0.0454 -> 0.0339, 512 0.263 -> 0.208.  For longer rows (a ring of bias tiles
// shared by the groups) this form drew enough power to pull the SM clock from 1.95 to 1.59 GHz and was slower (N = 1536: 6.1
// against 5.3 ms), so those keep flash_core_kernel.  Tried without gain: part of the exponentials as a polynomial on the FMA
// pipe, two threads per row, alternating the groups' exponential phases.
#pragma once
#include "attention.cuh"

namespace b200 {

// VR: value rows loaded per head (VR >= dh_out); VR < DH leaves the row of ones inside the padded head.
template <int DH, int VR, int G>
struct FlashResidentCfg {
  static constexpr int NB = DH == 64 ? 2 : 4;              // bias tiles that stay resident
  static constexpr int NV = VR + 16;                     // rows of the V^T operand: VR value rows, one row of ones, 15 of zeros
  static constexpr uint32_t Q_BYTES = 128 * DH * 2;      // per group
  static constexpr uint32_t K_BYTES = 128 * DH * 2;      // per stage
  static constexpr uint32_t V_HALF = NV * 128;           // NV rows x 64 keys x 2 B
  static constexpr uint32_t V_BYTES = 2 * V_HALF;
  static constexpr uint32_t V_TMA_BYTES = 2 * VR * 128;  // what TMA writes per stage (the value rows of both halves)
  static constexpr uint32_t Q_OFF = 0;                   // [G]
  static constexpr uint32_t K_OFF = G * Q_BYTES;         // [G][2]
  static constexpr uint32_t V_OFF = K_OFF + G * 2 * K_BYTES;         // [G][2]
  static constexpr uint32_t BIAS_OFF = V_OFF + G * 2 * V_BYTES;      // [NB] tiles x 32 KB
  static constexpr uint32_t MASK_OFF = BIAS_OFF + NB * kOperandTile; // [G][4] x 4 words
  // 16 x 16 identity (bf16) as an unswizzled K-major operand: two 16-byte K chunks of 16 rows each.
  static constexpr uint32_t IDENT_OFF = MASK_OFF + 256;
  static constexpr uint32_t BAR_OFF = IDENT_OFF + 512;
  static constexpr uint32_t SMEM_BYTES = BAR_OFF + 512 + 1024;
  static constexpr int THREADS = 192 * G;                // per group four softmax warps, an MMA warp and a loader warp
  // tensor-memory columns of one group
  static constexpr uint32_t TM_GROUP = 256;              // column stride between groups
  static constexpr uint32_t TM_S = 0, TM_P = 128, TM_O = 192;   // O: VR value columns, then the row sum
  static_assert(VR % 8 == 0 && VR <= DH && NV % 16 == 0, "V operand");
  static_assert(G == 1 || TM_O + NV <= TM_GROUP, "two groups do not fit the tensor memory");
  static_assert(TM_O + NV <= 512, "tensor memory");
  static_assert(SMEM_BYTES <= 232448, "shared memory");
};

// A row's reference is 0 until a maximum leaves this range (base-2 logits): then P and the sums stay within 2^-30 .. 2^60 per
// key, which fp32 and bf16 carry without loss, and most rows never subtract anything.
constexpr float kReferenceLow = -30.0f, kReferenceHigh = 60.0f;

__device__ __forceinline__ float max64(const float* v) {
  float m[8];
#pragma unroll
  for (int k = 0; k < 8; ++k)
    m[k] = max3(max3(v[k * 8], v[k * 8 + 1], v[k * 8 + 2]), max3(v[k * 8 + 3], v[k * 8 + 4], v[k * 8 + 5]),
                fmaxf(v[k * 8 + 6], v[k * 8 + 7]));
  return max3(max3(m[0], m[1], m[2]), max3(m[3], m[4], m[5]), fmaxf(m[6], m[7]));
}

// The pass a work index stands for (lines of a row block first); step() moves on to the next index without divisions.
struct FlashPass {
  int bg, h, qt, pr;
  __device__ __forceinline__ FlashPass(const FlashParams& p, int work) {
    pr = work % p.npairs;
    work /= p.npairs;
    qt = work % p.nqt;
    work /= p.nqt;
    h = work % p.H;
    bg = work / p.H;
  }
  __device__ __forceinline__ void step(const FlashParams& p) {
    if (++pr < p.npairs) return;
    pr = 0;
    if (++qt < p.nqt) return;
    qt = 0;
    if (++h < p.H) return;
    h = 0;
    ++bg;
  }
};

template <int DH, int VR, int G>
__global__ void __launch_bounds__(192 * G, 1)
flash_resident_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmV,
                  const __grid_constant__ CUtensorMap tmBias, const __grid_constant__ FlashParams p) {
  using Cfg = FlashResidentCfg<DH, VR, G>;
  constexpr bool SW64 = (DH == 32);
  constexpr int NB = Cfg::NB;
  constexpr float kNegMasked = -1.0e6f * 1.4426950408889634f;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* bias_full = bars;         // [NB] TMA
  uint64_t* bias_empty = bars + 4;    // [NB] one arrival per group
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  constexpr int kMmaWarp = 4 * G;         // + g
  constexpr int kLoaderWarp = 5 * G;      // + g
  const int g = warp < kMmaWarp ? warp >> 2 : warp < kLoaderWarp ? warp - kMmaWarp : warp - kLoaderWarp;
  uint64_t* gb = bars + 8 + g * 20;
  uint64_t* q_full = gb;              // TMA
  uint64_t* q_empty = gb + 1;         // commit: every S product of the item has been issued and has completed
  uint64_t* k_full = gb + 2;          // [2] TMA
  uint64_t* k_empty = gb + 4;         // [2] commit
  uint64_t* v_full = gb + 6;          // [2] TMA
  uint64_t* v_empty = gb + 8;         // [2] commit
  uint64_t* s_full = gb + 10;         // commit: S of the current key tile (bias included) is in tensor memory
  uint64_t* s_empty = gb + 11;        // count 128: every softmax thread of the group has read its scores
  uint64_t* p_full = gb + 12;         // count 128: P is written (and O rescaled if it had to be)
  uint64_t* pv_done = gb + 13;        // commit: O += P.V of the current key tile has completed
  uint64_t* mask_full = gb + 14;      // [4] count 1 (loader)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8 + G * 20);
  // Validity bits of a tile's keys, 4 words per slot: bit j of word w <=> key 32*w + j of the tile exists and is unmasked.
  // Slot n & 3 for tile n: it is written again for tile n + 4, whose K stage is free only after S(n + 2), which waited for
  // every softmax thread to have read S(n + 1) -- after it had read these bits.
  uint4* mask_bits = reinterpret_cast<uint4*>(smem + Cfg::MASK_OFF) + g * 4;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NB; ++i) {
      mbar_init(&bias_full[i], 1);
      mbar_init(&bias_empty[i], G);
    }
    for (int gg = 0; gg < G; ++gg) {
      uint64_t* x = bars + 8 + gg * 20;
      for (int i = 0; i < 18; ++i) mbar_init(&x[i], (i == 11 || i == 12) ? 128 : 1);
    }
    fence_mbar_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmBias);
  }
  if (threadIdx.x < 32) {  // identity: 16-byte unit u = (K chunk c, row i) holds K indices 8c .. 8c+7 of row i
    const int c = threadIdx.x >> 4, i = threadIdx.x & 15;
    uint32_t wds[4] = {0, 0, 0, 0};
    if ((i >> 3) == c) wds[(i & 7) >> 1] = (i & 1) ? 0x3F800000u : 0x00003F80u;
    *reinterpret_cast<uint4*>(smem + Cfg::IDENT_OFF + c * 256 + i * 16) = make_uint4(wds[0], wds[1], wds[2], wds[3]);
  }
  // Below the VR value rows of every V^T half tile: a row of ones (bf16 1.0) and 15 rows of zeros, written once --
  // TMA only ever writes the value rows.  16 rows x 128 B = 128 16-byte units per half tile.
  for (int u = threadIdx.x; u < G * 2 * 2 * 128; u += blockDim.x) {
    const int half = u >> 7, unit = u & 127;
    const uint32_t one2 = unit < 8 ? 0x3F803F80u : 0u;  // units 0..7 are row 0 of the block
    *reinterpret_cast<uint4*>(smem + Cfg::V_OFF + half * Cfg::V_HALF + VR * 128 + unit * 16) = make_uint4(one2, one2, one2, one2);
  }
  fence_proxy_async_smem();
  if (warp == kMmaWarp) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  const int T = p.nkt;
  // Contiguous ranges of passes per CTA.
  const int w0 = int((long long)p.total_work * blockIdx.x / gridDim.x);
  const int w1 = int((long long)p.total_work * (blockIdx.x + 1) / gridDim.x);
  auto line_of = [&](const FlashPass& x) { return x.bg * p.bias_div + x.pr * G + g; };
  auto line_ok = [&](const FlashPass& x) { return x.pr * G + g < p.bias_div && line_of(x) < p.Bt; };
  // n counts the key tiles of a group over all its items: every per-tile barrier completes one phase per n (parity n & 1), the
  // K and V stages alternate with n; w counts the group's items.

  if (warp >= kLoaderWarp) {
    // ------------------------------------------------------------------------------ loader of a group (group 0: bias too)
    int n = 0, w = 0, blocks = 0;  // blocks: bias row blocks so far
    FlashPass x(p, w0);
    for (int work = w0; work < w1; ++work, x.step(p)) {
      if (g == 0 && (work == w0 || x.pr == 0)) {
        for (int t = 0; t < T; ++t) {
          mbar_wait(&bias_empty[t], (blocks & 1) ^ 1, 78);
          if (lane == 0) {
            uint8_t* bb = smem + Cfg::BIAS_OFF + t * kOperandTile;
            mbar_arrive_expect_tx(&bias_full[t], kOperandTile);
            tma_load_3d(bb, &tmBias, &bias_full[t], t * 128, x.qt * 128, x.bg * p.H + x.h);
            tma_load_3d(bb + kOperandHalf, &tmBias, &bias_full[t], t * 128 + 64, x.qt * 128, x.bg * p.H + x.h);
          }
          __syncwarp();
        }
        ++blocks;
      }
      if (!line_ok(x)) continue;
      const int b = line_of(x);
      const uint8_t* mrow = p.mask + (long long)(b / p.mask_div) * p.mask_row_stride;
      mbar_wait(q_empty, (w & 1) ^ 1, 60);
      if (lane == 0) {
        mbar_arrive_expect_tx(q_full, Cfg::Q_BYTES);
        tma_load_3d(smem + Cfg::Q_OFF + g * Cfg::Q_BYTES, &tmQ, q_full, p.q_col0 + x.h * DH, x.qt * 128, b);
      }
      __syncwarp();
      for (int t = 0; t < T; ++t, ++n) {
        const int st = n & 1;
        uint8_t mv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int key = t * 128 + u * 32 + lane;
          mv[u] = key < p.N ? mrow[key * p.mask_key_stride] : 0;
        }
        mbar_wait(&k_empty[st], ((n >> 1) & 1) ^ 1, 61);
        if (lane == 0) {
          mbar_arrive_expect_tx(&k_full[st], Cfg::K_BYTES);
          tma_load_3d(smem + Cfg::K_OFF + (g * 2 + st) * Cfg::K_BYTES, &tmQ, &k_full[st], p.k_col0 + x.h * DH, t * 128, b);
        }
        __syncwarp();
        uint4 bits;
        bits.x = __ballot_sync(0xffffffffu, mv[0] != 0);
        bits.y = __ballot_sync(0xffffffffu, mv[1] != 0);
        bits.z = __ballot_sync(0xffffffffu, mv[2] != 0);
        bits.w = __ballot_sync(0xffffffffu, mv[3] != 0);
        if (lane == 0) {
          mask_bits[n & 3] = bits;
          mbar_arrive(&mask_full[n & 3]);
        }
        __syncwarp();
        mbar_wait(&v_empty[st], ((n >> 1) & 1) ^ 1, 75);
        if (lane == 0) {
          uint8_t* vb = smem + Cfg::V_OFF + (g * 2 + st) * Cfg::V_BYTES;
          mbar_arrive_expect_tx(&v_full[st], Cfg::V_TMA_BYTES);
          tma_load_3d(vb, &tmV, &v_full[st], t * 128, p.v_row0 + x.h * DH, b);
          tma_load_3d(vb + Cfg::V_HALF, &tmV, &v_full[st], t * 128 + 64, p.v_row0 + x.h * DH, b);
        }
        __syncwarp();
      }
      ++w;
    }
  } else if (warp >= kMmaWarp) {
    // ------------------------------------------------------------------------------ MMA issuer of a group
    // The whole warp walks the group's tile stream and waits on the barriers; one elected lane issues the products
    // and the commits (a converged warp issues a tcgen05.mma several times faster than a lone thread of a diverged one).
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128);
    constexpr uint32_t idesc_o = make_idesc_bf16(128, Cfg::NV);
    constexpr uint32_t idesc_b = make_idesc_bf16(128, 16);
    constexpr uint32_t qk_hi = SW64 ? kDescHiSw64 : kDescHiSw128;
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t z_lo = desc_lo(smem_base + Cfg::IDENT_OFF, 256);
    const uint32_t q_lo = desc_lo(smem_base + Cfg::Q_OFF + g * Cfg::Q_BYTES);
    const uint32_t tg = tmem_base + g * Cfg::TM_GROUP;
    FlashPass x(p, w0);
    int work = w0, t = 0, n = 0, w = 0;      // next S product
    int blocks = 0;                          // bias row blocks before this one
    // Issues the group's next S product, if there is one; gives back the bias tiles of blocks whose last pass has no line for it.
    auto issue_s = [&]() -> bool {
      while (work < w1) {
        const bool last = work + 1 == w1 || x.pr + 1 == p.npairs;  // the row block's last pass in this CTA
        if (!line_ok(x)) {
          if (last) {
            for (int tt = 0; tt < T; ++tt) {
              mbar_wait(&bias_full[tt], blocks & 1, 69);
              if (leader) mbar_arrive(&bias_empty[tt]);
            }
            ++blocks;
          }
          ++work;
          x.step(p);
          continue;
        }
        const int st = n & 1;
        if (t == 0) mbar_wait(q_full, w & 1, 64);
        const uint32_t k_lo = desc_lo(smem_base + Cfg::K_OFF + (g * 2 + st) * Cfg::K_BYTES);
        const uint32_t b_lo = desc_lo(smem_base + Cfg::BIAS_OFF + t * kOperandTile);
        mbar_wait(&mask_full[n & 3], (n >> 2) & 1, 73);  // so that S being full tells the softmax threads that the bits are there
        mbar_wait(&k_full[st], (n >> 1) & 1, 62);
        mbar_wait(&bias_full[t], blocks & 1, 68);
        mbar_wait(s_empty, (n & 1) ^ 1, 63);   // the scores of tile n - 1 have been read
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
          for (int k = 0; k < DH / 16; ++k)
            umma_bf16_ss2(tg + Cfg::TM_S, q_lo + 2 * k, qk_hi, k_lo + 2 * k, qk_hi, idesc_s, k > 0);
          umma_commit(&k_empty[st]);
          if (t + 1 == T) umma_commit(q_empty);
          // + bias tile: step k adds bias[:, 16k .. 16k+15] onto the same columns of the accumulator
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_bf16_ss2(tg + Cfg::TM_S + 16 * k, b_lo + (k >> 2) * (kOperandHalf >> 4) + (k & 3) * 2, kDescHiSw128, z_lo,
                          desc_hi_noswizzle(128), idesc_b, true);
          umma_commit(s_full);
          if (last) umma_commit(&bias_empty[t]);
        }
        __syncwarp();
        ++n;
        if (++t == T) {
          t = 0;
          ++w;
          if (last) ++blocks;
          ++work;
          x.step(p);
        }
        return true;
      }
      return false;
    };
    int m = 0, tp = 0;  // next P.V product
    bool have = issue_s();
    while (have) {
      have = issue_s();  // the next score tile: of this item, or the first one of the next item
      const int st = m & 1;
      const uint32_t v_lo = desc_lo(smem_base + Cfg::V_OFF + (g * 2 + st) * Cfg::V_BYTES);
      mbar_wait(&v_full[st], (m >> 1) & 1, 66);
      mbar_wait(p_full, m & 1, 65);
      tc_fence_after_sync();
      if (leader) {
#pragma unroll
        for (int k = 0; k < 8; ++k)  // A = P from tensor memory: 16 keys = 8 packed columns per K step
          umma_bf16_ts2(tg + Cfg::TM_O, tg + Cfg::TM_P + k * 8, v_lo + (k >> 2) * (Cfg::V_HALF >> 4) + (k & 3) * 2,
                        kDescHiSw128, idesc_o, (tp | k) != 0);  // the item's first product overwrites O
        umma_commit(pv_done);
        umma_commit(&v_empty[st]);
      }
      __syncwarp();
      ++m;
      if (++tp == T) tp = 0;
    }
  } else {
    // ------------------------------------------------------------------------------ softmax threads: one per query row
    const int quarter = warp & 3;          // TMEM lane quarter of this warp
    const int r = quarter * 32 + lane;     // query row of the tile == TMEM lane
    const uint32_t tg = tmem_addr(tmem_base, quarter * 32, g * Cfg::TM_GROUP);
    int n = 0;
    FlashPass x(p, w0);
    for (int work = w0; work < w1; ++work, x.step(p)) {
      if (!line_ok(x)) continue;
      const int b = line_of(x);
      const int q = x.qt * 128 + r;
      const bool q_ok = q < p.N;
      float m_ref = 0.f;         // what P and O (and the row sum in O) are expressed against
      bool shifted = false;      // some row of the warp has a reference other than 0
      bool only_masked = false;  // no valid key in the half tiles so far: every row's reference is the masked score
      uint4 gate_v[VR / 8];

      for (int t = 0; t < T; ++t, ++n) {
        if (t + 1 == T && p.gate && q_ok) {  // the gate of the item's output, a tile ahead of its use
          const __nv_bfloat16* gsrc = p.gate + (long long)b * p.gate_b_stride + (long long)q * p.gate_pitch + p.gate_col0 + x.h * p.dh_out;
#pragma unroll
          for (int c = 0; c < VR / 8; ++c)
            if (c * 8 < p.dh_out)
              asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(gate_v[c].x), "=r"(gate_v[c].y), "=r"(gate_v[c].z), "=r"(gate_v[c].w)
                           : "l"(gsrc + c * 8));
        }
        mbar_wait(s_full, n & 1, 67);
        tc_fence_after_sync();
        const uint4 okw = mask_bits[n & 3];
        // bit h: half tile h is not the common one (a test of the words inside the loop takes 217 instead of 208 us at 512 keys)
        uint32_t rare = (okw.x & okw.y) != 0xffffffffu ? 1u : 0u;
        if ((okw.z & okw.w) != 0xffffffffu) rare |= 2u;
        if (shifted) rare = 3u;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          float v[64];
          tmem_ld_32x32_f(tg + Cfg::TM_S + h * 64, v);
          tmem_ld_32x32_f(tg + Cfg::TM_S + h * 64 + 32, v + 32);
          tmem_ld_wait();
          if (h == 1) {
            tc_fence_before_sync();
            mbar_arrive(s_empty);  // the next tile's Q.K^T may overwrite S
          }
          // The common half tile: no key masked, every reference of the warp 0.  The exponentials do not wait for the maximum;
          // it only decides afterwards whether the half tile has to be done again.
          bool redo = (rare >> h) & 1u;
          if (!redo) {
            uint32_t pk[32];
            const float mc = max64(v);
#pragma unroll
            for (int e = 0; e < 64; e += 2) pk[e >> 1] = pack_bf16x2(exp2_approx(v[e]), exp2_approx(v[e + 1]));
            if (h == 0) {  // the previous tile's P.V has completed: P may be overwritten
              mbar_wait(pv_done, (n & 1) ^ 1, 70);
              tc_fence_after_sync();
            }
            tmem_st_32x32(tg + Cfg::TM_P + h * 32, pk);
            redo = __any_sync(0xffffffffu, mc > kReferenceHigh || (t == 0 && h == 0 && mc < kReferenceLow));
          }
          if (redo) {
            const uint32_t wa = h ? okw.z : okw.x, wb = h ? okw.w : okw.y;
            const bool first = t == 0 && h == 0;
            // No valid key: against a reference of 0 the weights are 0; while nothing but masked keys has been seen the
            // reference is their score, and the weight of each that exists is 1.  Padded lines are consecutive, so one CTA
            // has nearly all of a query tile's: by way of the half tiles below they set the launch's time (512 tokens, 37 of
            // them padded: 283 us; a full mask takes 208, this 211).
            if ((wa | wb) == 0 && (only_masked || first || !shifted)) {
              if (first) {
                only_masked = shifted = true;
                rare = 3u;
                m_ref = kNegMasked;
              }
              const int ones = only_masked ? p.N - (t * 128 + h * 64) : 0;
              uint32_t pk[32];
#pragma unroll
              for (int e = 0; e < 64; e += 2) pk[e >> 1] = (e < ones ? 0x3F80u : 0u) | (e + 1 < ones ? 0x3F800000u : 0u);
              mbar_wait(pv_done, (n & 1) ^ 1, 79);
              tc_fence_after_sync();
              tmem_st_32x32(tg + Cfg::TM_P + h * 32, pk);
              continue;
            }
            only_masked = false;
            const int left = p.N - (t * 128 + h * 64);  // keys from here on exist while j < left
            float y[64];
#pragma unroll
            for (int j = 0; j < 64; ++j)
              y[j] = (((j < 32 ? wa : wb) >> (j & 31)) & 1u) ? v[j] : (j < left ? kNegMasked : -INFINITY);
            const float mc = max64(y);
            const bool move = mc - m_ref > kReferenceHigh || (first && mc < kReferenceLow);
            mbar_wait(pv_done, (n & 1) ^ 1, 76);
            tc_fence_after_sync();
            if (__any_sync(0xffffffffu, move)) {
              // rare: a row leaves the range of its reference.  The maximum just seen becomes the reference; O and what this
              // tile has written of P are put on it.
              const float scale = move ? exp2_approx(m_ref - mc) : 1.0f;
              tmem_st_wait();
              if (t > 0) {
#pragma unroll 1
                for (int c = 0; c < Cfg::NV / 16; ++c) {
                  float o[16];
                  tmem_ld_32x16_f(tg + Cfg::TM_O + c * 16, o);
                  tmem_ld_wait();
#pragma unroll
                  for (int j = 0; j < 16; ++j) o[j] *= scale;
                  tmem_st_32x16_f(tg + Cfg::TM_O + c * 16, o);
                }
              }
#pragma unroll 1
              for (int c = 0; c < 2 * h; ++c) {
                uint32_t w[16];
                tmem_ld_32x16(tg + Cfg::TM_P + c * 16, w);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2(bf16lo(w[j]) * scale, bf16hi(w[j]) * scale);
                tmem_st_32x16(tg + Cfg::TM_P + c * 16, w);
              }
              tmem_st_wait();
              if (move) m_ref = mc;
              shifted = true;
              rare = 3u;
            }
            uint32_t pk[32];
#pragma unroll
            for (int e = 0; e < 64; e += 2) pk[e >> 1] = pack_bf16x2(exp2_approx(y[e] - m_ref), exp2_approx(y[e + 1] - m_ref));
            tmem_st_32x32(tg + Cfg::TM_P + h * 32, pk);
          }
        }
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(p_full);
      }
      // ---- the item's output: O and the row sum, once the last P.V has completed
      mbar_wait(pv_done, (n & 1) ^ 1, 71);
      tc_fence_after_sync();
      float o[VR];
#pragma unroll
      for (int c = 0; c < VR / 16; ++c) tmem_ld_32x16_f(tg + Cfg::TM_O + c * 16, o + c * 16);
      const float l_row = tmem_ld_32x1_f(tg + Cfg::TM_O + VR);
      tmem_ld_wait();
      tc_fence_before_sync();  // the next item's first P.V overwrites O; it is issued after this thread's next p_full arrival
      if (q_ok) {
        const float inv_l = __fdividef(1.0f, l_row);
        __nv_bfloat16* dst = p.out + (long long)b * p.out_b_stride + (long long)q * p.out_pitch + p.out_col0 + x.h * p.dh_out;
#pragma unroll
        for (int c = 0; c < VR / 8; ++c) {
          if (c * 8 < p.dh_out) {
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = o[c * 8 + e] * inv_l;
            if (p.gate) {
              const uint32_t gw[4] = {gate_v[c].x, gate_v[c].y, gate_v[c].z, gate_v[c].w};
              if (p.gate_activated) {
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] *= (e & 1) ? bf16hi(gw[e >> 1]) : bf16lo(gw[e >> 1]);
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  y[e] *= sigmoid_fast((e & 1) ? bf16hi(gw[e >> 1]) : bf16lo(gw[e >> 1]));
              }
            }
            *reinterpret_cast<uint4*>(dst + c * 8) = make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]),
                                                                pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200
