// Sliding-window attention with pair bias for the atom transformer: a query window of W atoms attends to the Hk keys
// centred on it (context = (Hk - W) / 2 atoms on either side, zero rows beyond the ends of the sequence).
//
// The work is small and oddly shaped (32 x 128 scores per window and head, head dim 32): for ~4,000 atoms it is a fraction of
// a GFLOP per sample, while the pair features that feed the bias are tens of MB.
//
//   window_bias16_kernel     bias[b][w][h][i][j] = proj_z(LayerNorm(z[b][w][i][j][:]))[h] for c_z = 16: one thread per pair
//   window_bias_kernel       any c_z: c_z / 4 lanes per pair
//   window_mma_kernel        windows of 16-query tiles and 128 keys: one CTA per (sample, window), a warp per head and 16
//                            queries, scores and weighted sum by mma.sync (a tcgen05 tile of 128 rows would be three
//                            quarters padding here).  fp32 softmax; the weights enter the second product as the sum of two
//                            bf16 values, so they keep 16 bits: against fp64 the kernel's error is that of the CUDA-core
//                            one, whose weights are fp32 (1.658e-3 for both at head dims 32 and 64, 1.661e-3 at 16: it
//                            is the rounding of the bf16 result)
//   window_pair_kernel       the bias (c_z = 16) and window_mma_kernel's attention of all samples of a window in one CTA
//   window_attention_kernel  other shapes: fp32 CUDA cores, one thread per (head, query)
// 4,096 atoms x 8 samples: window attention 115 us on CUDA cores (instruction-bound) -> 43 here, bias 36 us (shuffles) -> 10.
#pragma once
#include "elementwise.cuh"

namespace b200 {

struct WindowBiasParams {
  const void* z;       // [pairs][c_z], fp32 or bf16
  const float* ln_w;   // [c_z]
  const float* ln_b;   // [c_z] or nullptr
  const float* w_z;    // [heads][c_z]
  float* bias;         // [pairs / (W*Hk)][heads][W*Hk]
  long long pairs;     // B * NW * W * Hk
  int window_pairs;    // W * Hk
  int c_z, heads;
  float eps;
};

constexpr int kWindowMaxHeads = 16;

// A group of LPR lanes (a power of two >= c_z / 4) shares one pair: each lane holds four channels, the LayerNorm
// statistics and the per-head dot products are reduced across the group with shuffles, so a warp's loads cover
// 32 / LPR consecutive rows (contiguous memory) instead of 32 rows a stride apart.
template <bool F32>
__global__ void __launch_bounds__(256)
window_bias_kernel(WindowBiasParams p, int lpr) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int sub = lane / lpr, l = lane % lpr;
  const int rpw = 32 / lpr;
  const bool has = l * 4 < p.c_z;
  const long long warp_global = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long warp_stride = (long long)gridDim.x * (blockDim.x >> 5);
  float g[4] = {0.f, 0.f, 0.f, 0.f}, bt[4] = {0.f, 0.f, 0.f, 0.f};
  if (has) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      g[e] = p.ln_w[l * 4 + e];
      bt[e] = p.ln_b ? p.ln_b[l * 4 + e] : 0.f;
    }
  }
  const float inv = 1.0f / float(p.c_z);
  // every lane runs the same number of iterations: the shuffles are warp-wide
  for (long long rb = warp_global * rpw; rb < p.pairs; rb += warp_stride * rpw) {
    const long long t = rb + sub;
    const bool act = has && t < p.pairs;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    if (act) {
      if (F32) {
        const float4 v = *reinterpret_cast<const float4*>(static_cast<const float*>(p.z) + t * p.c_z + l * 4);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
      } else {
        const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p.z) + t * p.c_z + l * 4);
        x[0] = bf16lo(v.x); x[1] = bf16hi(v.x); x[2] = bf16lo(v.y); x[3] = bf16hi(v.y);
      }
    }
    float s = (x[0] + x[1]) + (x[2] + x[3]);
    for (int o = lpr >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = s * inv;
    float ss = 0.f;
    if (has) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] -= mean;
        ss = fmaf(x[e], x[e], ss);
      }
    }
    for (int o = lpr >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rstd = rsqrtf(ss * inv + p.eps);
    float y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = has ? fmaf(x[e] * rstd, g[e], bt[e]) : 0.f;
    const long long win = t / p.window_pairs;
    const int ij = int(t - win * p.window_pairs);
    float* dst = p.bias + win * p.heads * p.window_pairs + ij;
    for (int h = 0; h < p.heads; ++h) {
      float acc = 0.f;
      if (has) {
        const float* wr = p.w_z + h * p.c_z + l * 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc = fmaf(y[e], __ldg(wr + e), acc);
      }
      for (int o = lpr >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (l == (h % lpr) && t < p.pairs) dst[(long long)h * p.window_pairs] = acc;
    }
  }
}

// c_z = 16: the 16 channels of a pair in one thread, no shuffles; a warp's stores are contiguous for every head.
template <bool F32>
__global__ void __launch_bounds__(256)
window_bias16_kernel(WindowBiasParams p) {
  pdl_wait();
  __shared__ float ws[kWindowMaxHeads * 16 + 32];  // projection rows, LayerNorm weight, bias
  for (int i = threadIdx.x; i < p.heads * 16; i += blockDim.x) ws[i] = p.w_z[i];
  if (threadIdx.x < 16) {
    ws[kWindowMaxHeads * 16 + threadIdx.x] = p.ln_w[threadIdx.x];
    ws[kWindowMaxHeads * 16 + 16 + threadIdx.x] = p.ln_b ? p.ln_b[threadIdx.x] : 0.f;
  }
  __syncthreads();
  const float* lnw = ws + kWindowMaxHeads * 16;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < p.pairs; t += (long long)gridDim.x * blockDim.x) {
    float x[16];
    const uint8_t* row = static_cast<const uint8_t*>(p.z) + t * 16 * (long long)zbytes<F32>();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      float v[8];
      load8<F32>(row, k * 8, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[k * 8 + e] = v[e];
    }
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int e = 0; e < 16; ++e) s += x[e];
    const float mean = s * (1.0f / 16);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      x[e] -= mean;
      ss = fmaf(x[e], x[e], ss);
    }
    const float rstd = rsqrtf(ss * (1.0f / 16) + p.eps);
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = fmaf(x[e] * rstd, lnw[e], lnw[16 + e]);
    const long long win = t / p.window_pairs;
    float* dst = p.bias + win * p.heads * p.window_pairs + (t - win * p.window_pairs);
    for (int h = 0; h < p.heads; ++h) {
      float acc = 0.f;
#pragma unroll
      for (int e = 0; e < 16; ++e) acc = fmaf(x[e], ws[h * 16 + e], acc);
      dst[(long long)h * p.window_pairs] = acc;
    }
  }
}

struct WindowAttnParams {
  const __nv_bfloat16* qkv;   // [BM][L] rows of qkv_pitch: q (bias added) | k | v, L = NW * W atoms
  const __nv_bfloat16* gate;  // [BM][L] rows of gate_pitch: gate logits
  int qkv_pitch, gate_pitch;
  const float* bias;          // [B][NW][heads][W][Hk]
  const uint8_t* mask;        // [B][L], non-zero = valid atom
  __nv_bfloat16* out;         // [BM][L][c_s] = sigmoid(gate) * attention output
  int NW, W, Hk, heads, M;
  float scale;                // 1 / sqrt(head dim)
};

constexpr float kWindowMasked = -1e6f;  // the reference REPLACES masked logits by -inf = -1e6 (masked_fill_)

template <int DH>
__global__ void __launch_bounds__(256)
window_attention_kernel(WindowAttnParams p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int c_s = p.heads * DH;
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* Vs = Ks + (size_t)p.Hk * c_s;
  uint8_t* kvalid = reinterpret_cast<uint8_t*>(Vs + (size_t)p.Hk * c_s);

  const int f = blockIdx.x;
  const int bm = f / p.NW, w = f - bm * p.NW, b = bm / p.M;
  const int L = p.NW * p.W;
  const int a0 = w * p.W - (p.Hk - p.W) / 2;  // atom index of key 0 (may be negative)
  const long long item = (long long)bm * L;

  // stage the window's K and V rows (zero rows outside the sequence, as the zero-padded unfold gives)
  const int vec_per_row = c_s >> 3;
  for (int idx = threadIdx.x; idx < p.Hk * vec_per_row; idx += blockDim.x) {
    const int j = idx / vec_per_row, v = idx - j * vec_per_row;
    const int a = a0 + j;
    uint4 kk = make_uint4(0, 0, 0, 0), vv = make_uint4(0, 0, 0, 0);
    if (a >= 0 && a < L) {
      const __nv_bfloat16* src = p.qkv + (item + a) * p.qkv_pitch + c_s + v * 8;
      kk = *reinterpret_cast<const uint4*>(src);
      vv = *reinterpret_cast<const uint4*>(src + c_s);
    }
    reinterpret_cast<uint4*>(Ks)[idx] = kk;
    reinterpret_cast<uint4*>(Vs)[idx] = vv;
  }
  for (int j = threadIdx.x; j < p.Hk; j += blockDim.x) {
    const int a = a0 + j;
    kvalid[j] = (a >= 0 && a < L && p.mask[(long long)b * L + a]) ? 1 : 0;
  }
  __syncthreads();

  const int h = threadIdx.x / p.W, i = threadIdx.x - h * p.W;
  if (h >= p.heads) return;
  const long long atom = item + w * p.W + i;
  float q[DH], o[DH];
  {
    const __nv_bfloat16* qs = p.qkv + atom * p.qkv_pitch + h * DH;
#pragma unroll
    for (int d = 0; d < DH; d += 8) {
      float x[8];
      load8<false>(qs, d, x);
#pragma unroll
      for (int e = 0; e < 8; ++e) q[d + e] = x[e] * p.scale;
    }
  }
#pragma unroll
  for (int d = 0; d < DH; ++d) o[d] = 0.f;
  const float* brow = p.bias + ((((long long)b * p.NW + w) * p.heads + h) * p.W + i) * p.Hk;
  float m = -INFINITY, l = 0.f;
  for (int j0 = 0; j0 < p.Hk; j0 += 8) {
    float s[8];
    const float4 b0 = *reinterpret_cast<const float4*>(brow + j0), b1 = *reinterpret_cast<const float4*>(brow + j0 + 4);
    const float bj[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    float cmax = -INFINITY;
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
      const __nv_bfloat16* kr = Ks + (size_t)(j0 + jj) * c_s + h * DH;
      float acc = 0.f;
#pragma unroll
      for (int d = 0; d < DH; d += 8) {
        float x[8];
        load8<false>(kr, d, x);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc = fmaf(q[d + e], x[e], acc);
      }
      s[jj] = kvalid[j0 + jj] ? acc + bj[jj] : kWindowMasked;
      cmax = fmaxf(cmax, s[jj]);
    }
    const float m_new = fmaxf(m, cmax);
    const float corr = __expf(m - m_new);  // 0 on the first chunk (m = -inf)
    l *= corr;
#pragma unroll
    for (int d = 0; d < DH; ++d) o[d] *= corr;
    m = m_new;
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
      const float pj = __expf(s[jj] - m);
      l += pj;
      const __nv_bfloat16* vr = Vs + (size_t)(j0 + jj) * c_s + h * DH;
#pragma unroll
      for (int d = 0; d < DH; d += 8) {
        float x[8];
        load8<false>(vr, d, x);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[d + e] = fmaf(pj, x[e], o[d + e]);
      }
    }
  }
  const float inv_l = 1.0f / l;
  const __nv_bfloat16* gs = p.gate + atom * p.gate_pitch + h * DH;
  __nv_bfloat16* dst = p.out + atom * c_s + h * DH;
#pragma unroll
  for (int d = 0; d < DH; d += 8) {
    float g[8], y[8];
    load8<false>(gs, d, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = o[d + e] * inv_l / (1.0f + __expf(-g[e]));
    store8<false>(dst, d, y);
  }
}

// ---- mma.sync m16n8k16 (bf16, fp32 accumulation) and its operand loads
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(smem))
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(smem))
               : "memory");
}

constexpr int kWindowMmaKeys = 128;

// Shared memory: K and V rows of the window, pitch c_s * 2 + 16 bytes (eight consecutive rows of an 8 x 8 matrix fall on
// different banks), then the keys' validity bytes.  Warp = (head, 16-query tile); blockDim = heads * W / 16 warps.
template <int DH>
__global__ void __launch_bounds__(512)
window_mma_kernel(WindowAttnParams p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  constexpr int HK = kWindowMmaKeys;
  const int c_s = p.heads * DH;
  const int pitch = c_s * 2 + 16;
  uint8_t* Ks = smem_raw;
  uint8_t* Vs = Ks + HK * pitch;
  uint8_t* kvalid = Vs + HK * pitch;
  const int f = blockIdx.x;
  const int bm = f / p.NW, w = f - bm * p.NW, b = bm / p.M;
  const int L = p.NW * p.W;
  const int a0 = w * p.W - (HK - p.W) / 2;  // atom index of key 0 (may be negative)
  const long long item = (long long)bm * L;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int vec_per_row = c_s >> 3;  // zero rows outside the sequence, as the zero-padded unfold gives
  for (int idx = threadIdx.x; idx < HK * vec_per_row; idx += blockDim.x) {
    const int j = idx / vec_per_row, v = idx - j * vec_per_row;
    const int a = a0 + j;
    const bool in = a >= 0 && a < L;
    const __nv_bfloat16* src = p.qkv + (item + (in ? a : 0)) * p.qkv_pitch + c_s + v * 8;
    const uint32_t n = in ? 16u : 0u;  // source bytes; the rest of the 16 is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(Ks + j * pitch + v * 16)), "l"(src), "r"(n) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(Vs + j * pitch + v * 16)), "l"(src + c_s), "r"(n) : "memory");
  }
  for (int j = threadIdx.x; j < HK; j += blockDim.x) {
    const int a = a0 + j;
    kvalid[j] = (a >= 0 && a < L && p.mask[(long long)b * L + a]) ? 1 : 0;
  }
  const int tiles = p.W >> 4;
  const int h = warp / tiles, q0 = (warp - h * tiles) * 16;
  const int gr = lane >> 2, gc = (lane & 3) * 2;  // this lane's accumulator rows gr, gr + 8 and columns gc, gc + 1
  // Q fragments straight from global memory: rows gr / gr + 8, 16 dims per step
  uint32_t qf[DH / 16][4];
  {
    const __nv_bfloat16* r0 = p.qkv + (item + w * p.W + q0 + gr) * p.qkv_pitch + h * DH + gc;
    const __nv_bfloat16* r1 = r0 + 8ll * p.qkv_pitch;
#pragma unroll
    for (int k = 0; k < DH / 16; ++k) {
      qf[k][0] = *reinterpret_cast<const uint32_t*>(r0 + k * 16);
      qf[k][1] = *reinterpret_cast<const uint32_t*>(r1 + k * 16);
      qf[k][2] = *reinterpret_cast<const uint32_t*>(r0 + k * 16 + 8);
      qf[k][3] = *reinterpret_cast<const uint32_t*>(r1 + k * 16 + 8);
    }
  }
  // The bias, divided by the score scale, is where the score accumulators start: its loads are in flight with K and V.
  float s[HK / 8][4];
  {
    const float* brow = p.bias + ((((long long)b * p.NW + w) * p.heads + h) * p.W + q0 + gr) * HK + gc;
    const float unscale = 1.0f / p.scale;
#pragma unroll
    for (int n = 0; n < HK / 8; ++n) {
      const float2 b0 = *reinterpret_cast<const float2*>(brow + n * 8), b1 = *reinterpret_cast<const float2*>(brow + 8 * HK + n * 8);
      s[n][0] = b0.x * unscale, s[n][1] = b0.y * unscale, s[n][2] = b1.x * unscale, s[n][3] = b1.y * unscale;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  // scores: 16 queries x 128 keys
#pragma unroll
  for (int k = 0; k < DH / 16; ++k) {
#pragma unroll
    for (int n = 0; n < HK / 8; n += 2) {  // two 8-key tiles x 16 dims per load
      uint32_t kf[4];
      ldmatrix_x4(kf, Ks + (n * 8 + (lane & 7) + ((lane >> 4) << 3)) * pitch + (h * DH + k * 16 + ((lane >> 3) & 1) * 8) * 2);
      mma_bf16(s[n], qf[k], kf[0], kf[1]);
      mma_bf16(s[n + 1], qf[k], kf[2], kf[3]);
    }
  }
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int n = 0; n < HK / 8; ++n) {
    const bool ok0 = kvalid[n * 8 + gc], ok1 = kvalid[n * 8 + gc + 1];
    s[n][0] = ok0 ? s[n][0] * p.scale : kWindowMasked;
    s[n][1] = ok1 ? s[n][1] * p.scale : kWindowMasked;
    s[n][2] = ok0 ? s[n][2] * p.scale : kWindowMasked;
    s[n][3] = ok1 ? s[n][3] * p.scale : kWindowMasked;
    m0 = max3(m0, s[n][0], s[n][1]);
    m1 = max3(m1, s[n][2], s[n][3]);
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  float l0 = 0.f, l1 = 0.f;
  float o[DH / 8][4];
#pragma unroll
  for (int d = 0; d < DH / 8; ++d)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[d][e] = 0.f;
#pragma unroll
  for (int k = 0; k < HK / 16; ++k) {  // 16 keys per step: the weights of two score tiles are the A operand
    float e[8];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      e[u * 4 + 0] = __expf(s[2 * k + u][0] - m0);
      e[u * 4 + 1] = __expf(s[2 * k + u][1] - m0);
      e[u * 4 + 2] = __expf(s[2 * k + u][2] - m1);
      e[u * 4 + 3] = __expf(s[2 * k + u][3] - m1);
      l0 += e[u * 4 + 0] + e[u * 4 + 1];
      l1 += e[u * 4 + 2] + e[u * 4 + 3];
    }
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // register u: (row gr | gr + 8) of the first, then of the second tile
      const float x0 = e[u * 2], x1 = e[u * 2 + 1];
      hi[u] = pack_bf16x2(x0, x1);
      lo[u] = pack_bf16x2(x0 - bf16lo(hi[u]), x1 - bf16hi(hi[u]));
    }
#pragma unroll
    for (int d = 0; d < DH / 8; d += 2) {  // 16 keys x two 8-dim tiles per load
      uint32_t vf[4];
      ldmatrix_x4_trans(vf, Vs + (k * 16 + (lane & 15)) * pitch + (h * DH + d * 8 + (lane >> 4) * 8) * 2);
      mma_bf16(o[d], hi, vf[0], vf[1]);
      mma_bf16(o[d + 1], hi, vf[2], vf[3]);
      mma_bf16(o[d], lo, vf[0], vf[1]);
      mma_bf16(o[d + 1], lo, vf[2], vf[3]);
    }
  }
#pragma unroll
  for (int x = 1; x < 4; x <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, x);
    l1 += __shfl_xor_sync(0xffffffffu, l1, x);
  }
  const float i0 = 1.0f / l0, i1 = 1.0f / l1;
  const long long atom = item + w * p.W + q0 + gr;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const __nv_bfloat16* gs = p.gate + (atom + half * 8) * p.gate_pitch + h * DH + gc;
    __nv_bfloat16* dst = p.out + (atom + half * 8) * c_s + h * DH + gc;
    const float inv = half ? i1 : i0;
#pragma unroll
    for (int d = 0; d < DH / 8; ++d) {
      const uint32_t gv = *reinterpret_cast<const uint32_t*>(gs + d * 8);
      const float y0 = o[d][half * 2] * inv / (1.0f + __expf(-bf16lo(gv)));
      const float y1 = o[d][half * 2 + 1] * inv / (1.0f + __expf(-bf16hi(gv)));
      *reinterpret_cast<uint32_t*>(dst + d * 8) = pack_bf16x2(y0, y1);
    }
  }
}


// ---- the pair bias and all samples of a window in one kernel
struct WindowPairParams {
  WindowAttnParams a;  // a.bias unused
  const void* z;       // [B][NW][W][128][16]
  const float* ln_w;   // [16]
  const float* ln_b;   // [16] or nullptr
  const float* w_z;    // [heads][16]
  float eps;
  int chunks;          // CTAs of a window: each takes every chunks-th share of the samples
};

template <int DH>
struct WindowPairCfg {
  static constexpr int HK = kWindowMmaKeys;
  static constexpr int BIAS_PITCH = HK + 8;  // floats: four rows of a fragment's 8-byte loads fall on different banks
  // K or V of a window: boxes of 64 columns, [128 keys][128 B] each, swizzled as TMA writes them
  __host__ __device__ static constexpr uint32_t kv_bytes(int heads) { return uint32_t(heads * DH / 64) * kOperandHalf; }
  __host__ __device__ static constexpr uint32_t bias_bytes(int heads, int W) { return uint32_t(heads) * W * BIAS_PITCH * 4; }
  __host__ __device__ static constexpr uint32_t smem_bytes(int heads, int W) {
    return 4 * kv_bytes(heads) + bias_bytes(heads, W) + uint32_t(heads) * 17 * 4 + 64 + 1024;
  }
};

// window_mma_kernel for pair tensors of 16 channels, with the bias projected here: a CTA owns a window, computes its bias once
// into shared memory (fp32) and walks its samples.  Two teams of warps (a warp per head and 16 queries in each) take the samples
// in turn, so that one team's loads run under the other's products; inside a team the next sample's K, queries and gate are
// asked for as soon as the scores are done, its V^T after the weighted sum.
// 4,096 atoms x 8 samples, 128 windows: 33 us, 11 of them the bias (its pair rows from DRAM, beside the write-back of what the
// layer wrote before), 5 a pair of samples, the chain of the teams' steps: over the launch issue slots are 38 % used, the threads' data
// pipe 43 %, the tensor pipe 19 %.  As two kernels the bias went through global
// memory and came back once per sample (64 KB a window, as much as K and V), and nothing covered a CTA's loads: 11.4 + 43 us.
// At 128 registers a thread it spills 36 bytes with heads of 32, 8 with 16.
template <bool F32, int DH>
__global__ void __launch_bounds__(512, 1)
window_pair_kernel(const __grid_constant__ CUtensorMap tmKV, const __grid_constant__ WindowPairParams pp) {
  using Cfg = WindowPairCfg<DH>;
  constexpr int HK = Cfg::HK, BP = Cfg::BIAS_PITCH;
  const WindowAttnParams& p = pp.a;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int c_s = p.heads * DH;
  const uint32_t kv = Cfg::kv_bytes(p.heads);
  float* bias = reinterpret_cast<float*>(smem + 4 * kv);
  float* wz = bias + p.heads * p.W * BP;   // [heads][16] projection rows times the LayerNorm weight / score scale
  float* wz0 = wz + p.heads * 16;          // [heads] what the LayerNorm bias adds
  uint64_t* bars = reinterpret_cast<uint64_t*>((reinterpret_cast<uintptr_t>(wz0 + p.heads) + 7) & ~uintptr_t(7));
  const int chunk = blockIdx.x % pp.chunks, bw = blockIdx.x / pp.chunks;
  const int b = bw / p.NW, w = bw - b * p.NW;
  const int L = p.NW * p.W;
  const int a0 = w * p.W - (HK - p.W) / 2;  // atom index of key 0 (may be negative)
  const int team_threads = blockDim.x >> 1;
  const int team = threadIdx.x >= team_threads ? 1 : 0;
  const int warp = (threadIdx.x - team * team_threads) >> 5, lane = threadIdx.x & 31;
  uint8_t* Ks = smem + team * 2 * kv;
  uint8_t* Vs = Ks + kv;
  uint64_t* k_full = bars + team * 2;
  uint64_t* v_full = k_full + 1;
  const int step = 2 * pp.chunks;
  const int m_first = chunk * 2 + team;
  const bool loader = threadIdx.x == team * team_threads;  // the team's thread that issues its loads
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(&bars[i], 1);
    fence_mbar_init();
    prefetch_tmap(&tmKV);
  }
  __syncthreads();
  pdl_wait();

  auto load_rows = [&](uint8_t* dst, uint64_t* bar, int m, int col) {  // zero rows outside the sequence, as the zero-padded unfold gives
    mbar_arrive_expect_tx(bar, kv);
    for (int c = 0; c < c_s / 64; ++c) tma_load_3d(dst + c * kOperandHalf, &tmKV, bar, col + c * 64, a0, b * p.M + m);
  };
  const int tiles = p.W >> 4;
  const int h = warp / tiles, q0 = (warp - h * tiles) * 16;
  const int gr = lane >> 2, gc = (lane & 3) * 2;  // this lane's accumulator rows gr, gr + 8 and columns gc, gc + 1
  uint32_t qf[DH / 16][4];
  auto load_q = [&](int m) {  // fragments straight from global memory: rows gr / gr + 8, 16 dims per step
    const __nv_bfloat16* r0 = p.qkv + ((long long)(b * p.M + m) * L + w * p.W + q0 + gr) * p.qkv_pitch + h * DH + gc;
    const __nv_bfloat16* r1 = r0 + 8ll * p.qkv_pitch;
#pragma unroll
    for (int k = 0; k < DH / 16; ++k) {
      qf[k][0] = *reinterpret_cast<const uint32_t*>(r0 + k * 16);
      qf[k][1] = *reinterpret_cast<const uint32_t*>(r1 + k * 16);
      qf[k][2] = *reinterpret_cast<const uint32_t*>(r0 + k * 16 + 8);
      qf[k][3] = *reinterpret_cast<const uint32_t*>(r1 + k * 16 + 8);
    }
  };
  if (loader && m_first < p.M) {  // the first sample's rows come while the bias is computed
    load_rows(Ks, k_full, m_first, c_s);
    load_rows(Vs, v_full, m_first, 2 * c_s);
  }

  // ---- bias, divided by the score scale: it is where the score accumulators start
  if (threadIdx.x < p.heads * 16) {  // whole warps: the number of heads is even
    const float wv = pp.w_z[threadIdx.x];
    wz[threadIdx.x] = wv * pp.ln_w[lane & 15] / p.scale;
    float t = pp.ln_b ? pp.ln_b[lane & 15] * wv : 0.f;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 15) == 0) wz0[threadIdx.x >> 4] = t / p.scale;
  }
  __syncthreads();
  {
    // Two pairs of a thread at a time, the next two on their way.
    const int pairs = p.W * HK, stride = blockDim.x;
    const uint8_t* zrow = static_cast<const uint8_t*>(pp.z) + (long long)bw * pairs * 16 * zbytes<F32>();
    auto load = [&](int base, uint64_t (&x)[2][8]) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int ij = base + u * stride;
        const uint8_t* row = zrow + (long long)(ij < pairs ? ij : 0) * 16 * zbytes<F32>();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          float v[8];
          load8<F32>(row, k * 8, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) x[u][k * 4 + e] = pack_f32x2(v[2 * e], v[2 * e + 1]);
        }
      }
    };
    auto project = [&](int base, uint64_t (&x)[2][8]) {
      float rstd[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint64_t s[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = add2(x[u][e], x[u][e + 4]);
        float s0, s1;
        unpack_f32x2(add2(add2(s[0], s[1]), add2(s[2], s[3])), s0, s1);
        const float mean = (s0 + s1) * (-1.0f / 16);
        const uint64_t mean2 = pack_f32x2(mean, mean);
        uint64_t q[2] = {0, 0};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          x[u][e] = add2(x[u][e], mean2);
          q[e & 1] = fma2(x[u][e], x[u][e], q[e & 1]);
        }
        unpack_f32x2(add2(q[0], q[1]), s0, s1);
        rstd[u] = rsqrtf((s0 + s1) * (1.0f / 16) + pp.eps);
      }
      for (int hh = 0; hh < p.heads; hh += 2) {  // an even number: heads fill boxes of 64 columns
        uint64_t acc[2][2] = {{0, 0}, {0, 0}};
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(wz + (hh + k) * 16 + e * 2);
#pragma unroll
            for (int u = 0; u < 2; ++u) acc[k][u] = fma2(x[u][e + 1], wv.y, fma2(x[u][e], wv.x, acc[k][u]));
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int ij = base + u * stride;
          float* dst = bias + (hh * p.W + ij / HK) * BP + ij % HK;
          if (ij < pairs) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              float s0, s1;
              unpack_f32x2(acc[k][u], s0, s1);
              dst[k * p.W * BP] = fmaf(s0 + s1, rstd[u], wz0[hh + k]);
            }
          }
        }
      }
    };
    uint64_t xa[2][8], xb[2][8];
    int base = threadIdx.x;
    load(base, xa);
    while (base < pairs) {
      load(base + 2 * stride, xb);
      project(base, xa);
      base += 2 * stride;
      if (base >= pairs) break;
      load(base + 2 * stride, xa);
      project(base, xb);
      base += 2 * stride;
    }
  }
  // validity of this lane's keys n * 8 + gc, n * 8 + gc + 1: bits 2n, 2n + 1
  uint32_t ok = 0;
#pragma unroll
  for (int u = 0; u < HK / 32; ++u) {
    const int a = a0 + u * 32 + lane;
    const uint32_t word = __ballot_sync(0xffffffffu, a >= 0 && a < L && p.mask[(long long)b * L + a] != 0);
#pragma unroll
    for (int n = 0; n < 4; ++n) ok |= ((word >> (n * 8 + gc)) & 3u) << (2 * (u * 4 + n));
  }
  const bool all_ok = __all_sync(0xffffffffu, ok == 0xffffffffu);
  if (m_first < p.M) load_q(m_first);
  __syncthreads();

  const float c2 = p.scale * 1.4426950408889634f;  // to base-2 logits, in the exponent's multiply-add
  const float masked = kWindowMasked / p.scale;
  const int head_box = h * DH / 64, head_unit = (h * DH % 64) / 8;  // the head's 64-column box, its first 16-byte unit there
  uint32_t phase = 0;
  for (int m = m_first; m < p.M; m += step, phase ^= 1) {
    const bool more = m + step < p.M;
    float s[HK / 8][4];
    const float* brow = bias + (h * p.W + q0 + gr) * BP + gc;
#pragma unroll
    for (int n = 0; n < HK / 8; ++n) {
      const float2 b0 = *reinterpret_cast<const float2*>(brow + n * 8), b1 = *reinterpret_cast<const float2*>(brow + 8 * BP + n * 8);
      s[n][0] = b0.x, s[n][1] = b0.y, s[n][2] = b1.x, s[n][3] = b1.y;
    }
    mbar_wait(k_full, phase, 82);
    // scores: 16 queries x 128 keys
#pragma unroll
    for (int k = 0; k < DH / 16; ++k) {
#pragma unroll
      for (int n = 0; n < HK / 8; n += 2) {  // two 8-key tiles x 16 dims per load
        uint32_t kf[4];
        ldmatrix_x4(kf, Ks + head_box * kOperandHalf + sw128_offset(n * 8 + (lane & 7) + ((lane >> 4) << 3), head_unit + k * 2 + ((lane >> 3) & 1)));
        mma_bf16(s[n], qf[k], kf[0], kf[1]);
        mma_bf16(s[n + 1], qf[k], kf[2], kf[3]);
      }
    }
    named_bar_sync(1 + team, team_threads);  // the team has read K
    if (more) {
      if (loader) load_rows(Ks, k_full, m + step, c_s);
      load_q(m + step);
    }
    const long long atom = (long long)(b * p.M + m) * L + w * p.W + q0 + gr;
    const __nv_bfloat16* gs = p.gate + atom * p.gate_pitch + h * DH + gc;
    uint32_t gv[2][DH / 8];
#pragma unroll
    for (int d = 0; d < DH / 8; ++d) {
      gv[0][d] = *reinterpret_cast<const uint32_t*>(gs + d * 8);
      gv[1][d] = *reinterpret_cast<const uint32_t*>(gs + 8ll * p.gate_pitch + d * 8);
    }
    float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < HK / 8; ++n) {
      if (!all_ok) {
        const bool ok0 = (ok >> (2 * n)) & 1u, ok1 = (ok >> (2 * n + 1)) & 1u;
        s[n][0] = ok0 ? s[n][0] : masked;
        s[n][1] = ok1 ? s[n][1] : masked;
        s[n][2] = ok0 ? s[n][2] : masked;
        s[n][3] = ok1 ? s[n][3] : masked;
      }
      m0 = max3(m0, s[n][0], s[n][1]);
      m1 = max3(m1, s[n][2], s[n][3]);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    }
    mbar_wait(v_full, phase, 83);
    const float n0 = -m0 * c2, n1 = -m1 * c2;
    float l0 = 0.f, l1 = 0.f;
    float o[DH / 8][4];
#pragma unroll
    for (int d = 0; d < DH / 8; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[d][e] = 0.f;
#pragma unroll
    for (int k = 0; k < HK / 16; ++k) {  // 16 keys per step: the weights of two score tiles are the A operand
      float e[8];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        e[u * 4 + 0] = exp2_approx(fmaf(s[2 * k + u][0], c2, n0));
        e[u * 4 + 1] = exp2_approx(fmaf(s[2 * k + u][1], c2, n0));
        e[u * 4 + 2] = exp2_approx(fmaf(s[2 * k + u][2], c2, n1));
        e[u * 4 + 3] = exp2_approx(fmaf(s[2 * k + u][3], c2, n1));
        l0 += e[u * 4 + 0] + e[u * 4 + 1];
        l1 += e[u * 4 + 2] + e[u * 4 + 3];
      }
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // register u: (row gr | gr + 8) of the first, then of the second tile
        const float x0 = e[u * 2], x1 = e[u * 2 + 1];
        hi[u] = pack_bf16x2(x0, x1);
        lo[u] = pack_bf16x2(x0 - bf16lo(hi[u]), x1 - bf16hi(hi[u]));
      }
#pragma unroll
      for (int d = 0; d < DH / 8; d += 2) {  // 16 keys x two 8-dim tiles per load
        uint32_t vf[4];
        ldmatrix_x4_trans(vf, Vs + head_box * kOperandHalf + sw128_offset(k * 16 + (lane & 15), head_unit + d + (lane >> 4)));
        mma_bf16(o[d], hi, vf[0], vf[1]);
        mma_bf16(o[d + 1], hi, vf[2], vf[3]);
        mma_bf16(o[d], lo, vf[0], vf[1]);
        mma_bf16(o[d + 1], lo, vf[2], vf[3]);
      }
    }
    named_bar_sync(1 + team, team_threads);  // the team has read V
    if (more && loader) load_rows(Vs, v_full, m + step, 2 * c_s);
#pragma unroll
    for (int x = 1; x < 4; x <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, x);
      l1 += __shfl_xor_sync(0xffffffffu, l1, x);
    }
    const float i0 = 1.0f / l0, i1 = 1.0f / l1;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      __nv_bfloat16* dst = p.out + (atom + half * 8) * c_s + h * DH + gc;
      const float inv = half ? i1 : i0;
#pragma unroll
      for (int d = 0; d < DH / 8; ++d) {
        const float y0 = quotient(o[d][half * 2] * inv, 1.0f + __expf(-bf16lo(gv[half][d])));
        const float y1 = quotient(o[d][half * 2 + 1] * inv, 1.0f + __expf(-bf16hi(gv[half][d])));
        *reinterpret_cast<uint32_t*>(dst + d * 8) = pack_bf16x2(y0, y1);
      }
    }
  }
}

}  // namespace b200
