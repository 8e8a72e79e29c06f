// Row kernels of the fp32-accurate pair ops, between tcgen05 products of split operands.
//
// An fp32 value travels as hi = bf16(x), lo = bf16(x - hi).  A product of split operands is three ordinary products
// (hi.hi + hi.lo + lo.hi) laid end to end along K: one operand reads hi | hi | lo, the other hi | lo | hi.  Activations whose
// hi part is whole K blocks of 64 are stored once as (hi | lo) and the operands of the triangle contraction, whose K is the
// token count, as hi and lo planes; the product's loads read hi twice.  All arithmetic here is fp32 with expf and exact
// division.  Every kernel is bound by memory: each reads its input once, 16 bytes a lane, and writes its output once.
#pragma once
#include "elementwise.cuh"

namespace b200 {

// LayerNorm (when normalize) and split of 128-channel rows: x fp32 [.][128] -> y bf16 [n_lines * pitch][hi 128 | lo 128].
// Row (line, pos) reads x row line * line_stride + pos * pos_stride, zeros for pos >= n_pos (the padding that makes a line a
// whole number of 16-byte units).  A warp keeps four rows in registers: one read, two-pass statistics (the row kernel that
// reads each row three times: 20.2 us for 40 000 rows).
__global__ void __launch_bounds__(256)
ln_split128_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, const float* __restrict__ w,
                   const float* __restrict__ b, long long rows, int n_pos, int pitch, long long line_stride,
                   long long pos_stride, int normalize) {
  constexpr int R = 4;
  pdl_wait();
  const int lane = threadIdx.x & 31;
  float wv[4], bv[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    wv[e] = normalize && w ? w[lane * 4 + e] : 1.f;
    bv[e] = normalize && b ? b[lane * 4 + e] : 0.f;
  }
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R; r0 < rows; r0 += warps * R) {
    float4 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const long long r = r0 + i, line = r / pitch;
      const int pos = int(r - line * pitch);
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && pos < n_pos)
        v[i] = *reinterpret_cast<const float4*>(x + (line * line_stride + pos * pos_stride) * 128 + lane * 4);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const long long r = r0 + i;
      if (r >= rows) break;
      float f[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      if (normalize) {
        const float mean = warp_sum((f[0] + f[1]) + (f[2] + f[3])) * (1.f / 128.f);
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          f[e] -= mean;
          ss = fmaf(f[e], f[e], ss);
        }
        const float rstd = rsqrtf(warp_sum(ss) * (1.f / 128.f) + 1e-5f);
        const bool pad = r % pitch >= n_pos;
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = pad ? 0.f : f[e] * rstd * wv[e] + bv[e];
      }
      uint2 hi, lo;
      split_pair(f[0], f[1], hi.x, lo.x);
      split_pair(f[2], f[3], hi.y, lo.y);
      __nv_bfloat16* yr = y + r * 256 + lane * 4;
      *reinterpret_cast<uint2*>(yr) = hi;
      *reinterpret_cast<uint2*>(yr + 128) = lo;
    }
  }
}

// LayerNorm over the channels of t fp32 [128][n_rows][pitch] and split: y bf16 [n_rows * n_cols][hi 128 | lo 128].  A block
// turns 128 channels x 32 pairs over in shared memory (permute and split in passes of their own: 44 us at 200 tokens).
__global__ void __launch_bounds__(256)
ln_split_channels_kernel(const float* __restrict__ t, __nv_bfloat16* __restrict__ y, const float* __restrict__ w,
                         const float* __restrict__ b, int n_rows, int n_cols, int pitch) {
  __shared__ float tile[32][129];
  pdl_wait();
  const int row = blockIdx.y, j0 = blockIdx.x * 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    const int q = (threadIdx.x & 7) * 4, d0 = threadIdx.x >> 3;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = d0 + i * 32;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j0 + q < pitch) v[i] = *reinterpret_cast<const float4*>(t + ((long long)d * n_rows + row) * pitch + j0 + q);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = d0 + i * 32;
      tile[q][d] = v[i].x, tile[q + 1][d] = v[i].y, tile[q + 2][d] = v[i].z, tile[q + 3][d] = v[i].w;
    }
  }
  __syncthreads();
  const int c = lane * 2;  // channels c, c + 1, c + 64, c + 65
  const float wv[4] = {w[c], w[c + 1], w[c + 64], w[c + 65]}, bv[4] = {b[c], b[c + 1], b[c + 64], b[c + 65]};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = warp * 4 + i;
    if (j0 + j >= n_cols) break;
    float f[4] = {tile[j][c], tile[j][c + 1], tile[j][c + 64], tile[j][c + 65]};
    const float mean = warp_sum((f[0] + f[1]) + (f[2] + f[3])) * (1.f / 128.f);
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f[e] -= mean;
      ss = fmaf(f[e], f[e], ss);
    }
    const float rstd = rsqrtf(warp_sum(ss) * (1.f / 128.f) + 1e-5f);
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = f[e] * rstd * wv[e] + bv[e];
    uint32_t hi[2], lo[2];
    split_pair(f[0], f[1], hi[0], lo[0]);
    split_pair(f[2], f[3], hi[1], lo[1]);
    uint32_t* yr = reinterpret_cast<uint32_t*>(y + ((long long)row * n_cols + j0 + j) * 256);
    yr[lane] = hi[0], yr[lane + 32] = hi[1], yr[lane + 64] = lo[0], yr[lane + 96] = lo[1];
  }
}

// out[row][col] = [x +] p * sigmoid(g) over 128 channels: p in pair order, g in (line, pos) order of the projection.
__global__ void __launch_bounds__(256)
gate_pairs_kernel(const float* __restrict__ p, const float* __restrict__ g, const float* x, float* out,
                  int n, int pitch, int incoming) {
  pdl_wait();
  const long long total = (long long)n * n * 32;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long pair = i >> 5;
    const int v = int(i & 31) * 4;
    const int r = int(pair / n), c = int(pair - (long long)r * n);
    const long long gr = incoming ? (long long)c * pitch + r : (long long)r * pitch + c;
    const float4 pv = *reinterpret_cast<const float4*>(p + pair * 128 + v);
    const float4 gv = *reinterpret_cast<const float4*>(g + gr * 128 + v);
    float4 o = x ? *reinterpret_cast<const float4*>(x + pair * 128 + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    o.x += pv.x / (1.f + expf(-gv.x));
    o.y += pv.y / (1.f + expf(-gv.y));
    o.z += pv.z / (1.f + expf(-gv.z));
    o.w += pv.w / (1.f + expf(-gv.w));
    *reinterpret_cast<float4*>(out + pair * 128 + v) = o;
  }
}

}  // namespace b200
