// C ABI of the library (declared in include/b200pair.h): argument checks, tensor-map
// construction and kernel launches.  The kernels live in the .cuh files beside this one and are
// compiled into this single translation unit.
#include <cstdarg>
#include <type_traits>

#include "host_util.cuh"
#include "umma.cuh"
#include "row_tile.cuh"
#include "bmm_nt.cuh"
#include "trimul.cuh"
#include "transition.cuh"
#include "ln_linear.cuh"
#include "pair_cond.cuh"
#include "cond_block.cuh"
#include "elementwise.cuh"
#include "accurate.cuh"
#include "opm.cuh"
#include "attention.cuh"
#include "attention_resident.cuh"
#include "attention_line.cuh"
#include "pair_bias.cuh"
#include "triatt.cuh"
#include "window_attention.cuh"

namespace b200 {

template <int DH>
static int launch_window_attention(const WindowAttnParams& p, int BM, cudaStream_t st) {
  // whole 16-query tiles, the 128 keys whose scores a warp holds in registers, and at most 16 warps: the mma.sync kernel
  if (p.W % 16 == 0 && p.Hk == kWindowMmaKeys && p.heads * (p.W / 16) <= 16 && p.qkv_pitch % 8 == 0 && p.gate_pitch % 2 == 0) {
    const uint32_t smem = uint32_t(2 * kWindowMmaKeys * (p.heads * DH * 2 + 16) + kWindowMmaKeys);
    if (smem <= 227 * 1024) {
      B200_LAUNCH(window_mma_kernel<DH>, BM * p.NW, p.heads * (p.W / 16) * 32, smem, st, p);
      return B200_OK;
    }
  }
  const uint32_t smem = uint32_t(2u * p.Hk * p.heads * DH * 2u + p.Hk + 16);
  B200_LAUNCH(window_attention_kernel<DH>, BM * p.NW, p.heads * p.W, smem, st, p);
  return B200_OK;
}

// Whether window_pair_kernel takes these shapes: whole 16-query tiles, 128 keys, 16 pair channels, heads of 16 or 32 (with 64 it
// spills 190 bytes, with 32 36) in boxes of 64 columns, two teams of warps within 512 threads and their K and V in shared memory; and the
// windows in one wave of CTAs that have samples enough to pay for a bias phase of their own.  Three layers, heads 4 x 32, us as two
// kernels / as one (windows x samples): 16 x 8 118 / 131, 32 x 4 121 / 131, 64 x 2 126 / 132, 32 x 6 131 / 132, 64 x 3 136 / 132, 64 x 8
// 173 / 154, 95 x 3 147 / 142, 96 x 1 132 / 125, 128 x 2 151 / 134, 128 x 8 317 / 274, 148 x 1 141 / 125, 148 x 8 343 / 281; beyond a
// wave 149 x 1 149 / 160, 149 x 8 402 / 419, 160 x 4 277 / 285.  Of 72 pairs of 16 to 192 windows and 1 to 8 samples it takes the slower
// of the two by more than 1 % in these: 80 x 3 139 / 142 as one; as two 80 x 1 128 / 124, 80 x 2 138 / 132, 95 x 1 132 / 125, 95 x 2 143
// / 132, 176 x 2 194 / 185, 192 x 1 166 / 164, 192 x 2 199 / 188, 192 x 6 348 / 344, 192 x 8 457 / 436 (149 x 3 within the spread).
static bool window_pair_fits(const WindowAttnParams& p, int B, int head_dim, int c_z, const void* z) {
  if ((head_dim != 16 && head_dim != 32) || p.W % 16 || p.W > p.Hk || p.Hk != kWindowMmaKeys || c_z != 16 || p.heads * (p.W / 16) > 8 ||
      p.qkv_pitch % 8 || p.gate_pitch % 2 || p.heads * head_dim % 64 || !aligned(z, 32))
    return false;
  const int64_t windows = int64_t(B) * p.NW;
  if (windows > sm_count() || (p.M == 1 ? windows < 96 : windows * p.M < 192)) return false;
  const uint32_t smem = head_dim == 16 ? WindowPairCfg<16>::smem_bytes(p.heads, p.W) : WindowPairCfg<32>::smem_bytes(p.heads, p.W);
  return smem <= 227 * 1024;
}

template <int DH>
static int launch_window_pair(WindowPairParams p, int B, bool f32, cudaStream_t st) {
  // A window's samples go to `chunks` CTAs, each of which computes the bias: as many as make the estimated time shortest (a wave's
  // bias takes about as long as one and a half samples of a team).
  const int windows = B * p.a.NW, most = (p.a.M + 1) / 2, sms = sm_count();
  int64_t best = INT64_MAX;
  p.chunks = 1;
  for (int c = 1; c <= most; ++c) {
    const int64_t waves = (int64_t(windows) * c + sms - 1) / sms, rounds = (p.a.M + 2 * c - 1) / (2 * c);
    const int64_t cost = waves * (3 + 2 * rounds);
    if (cost < best) best = cost, p.chunks = c;
  }
  CUtensorMap tmKV;
  {
    const uint64_t dims[3] = {uint64_t(3 * p.a.heads * DH), uint64_t(p.a.NW) * p.a.W, uint64_t(B) * p.a.M};
    const uint64_t str[2] = {uint64_t(p.a.qkv_pitch) * 2, uint64_t(p.a.NW) * p.a.W * p.a.qkv_pitch * 2};
    const uint32_t box[3] = {64, kWindowMmaKeys, 1};
    if (int e = make_tmap_bf16(&tmKV, p.a.qkv, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const int threads = 2 * p.a.heads * (p.a.W / 16) * 32;
  const uint32_t smem = WindowPairCfg<DH>::smem_bytes(p.a.heads, p.a.W);
  if (f32) B200_LAUNCH((window_pair_kernel<true, DH>), windows * p.chunks, threads, smem, st, tmKV, p);
  else B200_LAUNCH((window_pair_kernel<false, DH>), windows * p.chunks, threads, smem, st, tmKV, p);
  return B200_OK;
}

static int grid_for(int64_t work_items, int per_block) {
  int64_t blocks = (work_items + per_block - 1) / per_block;
  const int64_t cap = int64_t(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return int(blocks);
}

struct BmmLaunch {
  const void* A;
  const void* B;
  void* C;
  int batch, M, N, K;
  int64_t lda, ldb, ldc, sa, sb, sc;  // elements
  float scale = 1.0f;
  const float* scale_ptr = nullptr;
  const float* bias = nullptr;
  int out_f32 = 0;
  int opm_ntok = 0;
  const void* residual = nullptr;
  bool round_once = false;  // bf16 residual in C itself: read, added in fp32 and rounded once, not reduced into memory in bf16
  bool b_shared = false;  // one B for every batch item
  const float* mul = nullptr;  // bulk output: per-element fp32 factor, row pitch mul_pitch
  int mul_pitch = 0;
  bool swiglu = false;  // bulk bf16 output: N columns are 64-wide (a | b) block pairs, C has N / 2 columns of silu(a) * b
  int row_groups = 0;          // bulk bf16 output, M = 32 * row_groups: group g of batch item b is C + g * group_stride + b * sc
  int64_t group_stride = 0;
  int b_rows = 0;              // rows of B that exist, if fewer than N (the rest count as zeros)
  bool split = false;   // with swiglu: C has N columns, (hi | lo) of the fp32 values
  bool parts = false;   // A and B are hi and lo planes, `batch` slices each, K is one part's width
  const uint8_t* gate_mask = nullptr;  // gated split operands (kEpiGateSplit): C [N / 256][2 * 128][M], M contiguous
  int mask_pitch = 0, mask_n = 0;
  int64_t mask_line = 0, mask_pos = 0;
  int a_fold = 0, b_fold = 0;  // operand stored as (hi | lo), each part this many K blocks of 64, read as hi | hi | lo
};

// Tile width by the estimated time of the busiest CTA.  A K block of 64 takes a 256-wide tile about 1.5 times as long as a
// 128-wide one (48 against 32 KB through L2 for twice the product), the last tile's epilogue is exposed; in units of a
// thousandth of a 128-wide block: 256 columns where they fill the waves, 128 where the narrow tile leaves fewer CTAs idle.
// Against the better of the two widths, over 60 products of the trunk, the token and atom blocks, the contractions and the
// outer product mean: within 2 % of it, once 5 % (rows x columns x K, us, 128 / 256 wide: 256 x 768 x 3072 12.2 / 18.8,
// 2048 x 2816 x 768 12.2 / 13.5, 2048 x 6144 x 768 20.7 / 18.9, 3584 x 2816 x 768 17.9 / 18.6 where the estimate takes 256;
// 128 batches of 384^3 21.8 / 25.7, of 512^3 42.5 / 38.7).
// 64 columns where even the narrow tiles are few: a K block of 64 is then bound by shared memory (24 KB written and 24 read, against
// 32 and 32), and twice the SMs share the epilogues.  Token layers x 4 (rows, us with 128-wide tiles at the least / with 64): 32 280 /
// 263, 256 289 / 268, 512 297 / 286, 800 354 / 341, 1600 434 / 433, 2048 the same tiles.  Of 261 products (24 to 20000 rows,
// widths of the trunk, the token and atom blocks, contractions; one after the other in a graph) it is taken for 186: 185 are 6 to 20 %
// shorter than with the 128-wide tiles' best (1024 x 384 x 384 5.3 / 4.3), short K among them although wider tiles then have eight
// epilogue warps; 128 batches of 128 x 128 x 64 take 3.69 us instead of 3.59.
// Products that run on a side stream underneath another's kernels go by the same estimate: wide tiles for those, since they
// take less SM time, moved a trunk's time both ways (4 blocks, us, without / with: 144 tokens 890 / 902, 160 1024 / 1006,
// 203 1144 / 1154, 256 1292 / 1322, 320 and more the same).
static int bmm_tile_n(int M, int N, int K, int batch, int narrowest, int widest) {
  const int64_t tm = (M + 127) / 128, kb = (K + 63) / 64, sms = sm_count();
  auto cost = [&](int bn, int64_t per_block, int64_t tail) {
    const int64_t tiles = tm * ((N + bn - 1) / bn) * batch;
    return (tiles + sms - 1) / sms * (kb * per_block + 700) + tail;
  };
  int bn = 128;
  int64_t best = cost(128, 1000, 2500);
  if (widest > 128 && cost(256, 1500, 5000) <= best) bn = 256, best = cost(256, 1500, 5000);
  if (narrowest < 128 && cost(64, 760, 1250) < best) bn = 64;
  return bn;
}

static int launch_bmm(const BmmLaunch& a, cudaStream_t stream) {
  const int64_t c_batch = a.sc > 0 ? a.sc : a.ldc * int64_t(a.M);
  const int c_esz = a.out_f32 ? 4 : 2;
  // Bulk output through the C tensor map where the layout allows it (the map clips the last column group): the
  // residual (if any) being C itself.
  const bool bulk_c = a.opm_ntok == 0 && (a.ldc * c_esz) % 16 == 0 && (c_batch * c_esz) % 16 == 0 && aligned(a.C, 16);
  // An fp32 residual elsewhere comes by TMA tiles, as a gate's factors do (read by the lanes from their rows: 11 us against 7
  // for 65536 x 128 x 128), and so does a bf16 one that is rounded once.
  const bool add = bulk_c && a.residual && !a.mul && !a.swiglu &&
                   (a.out_f32 ? a.residual != a.C && a.batch == 1 && aligned(a.residual, 16) : a.residual == a.C && a.round_once);
  // 64-wide tiles: bulk output of whole rows
  const bool narrow = bulk_c && (add || a.residual == nullptr || a.residual == a.C) && (a.bias == nullptr || aligned(a.bias, 16)) &&
                      !a.swiglu && a.opm_ntok == 0 && a.row_groups == 0;
  const int BN = a.split || a.gate_mask ? 256
                                        : bmm_tile_n(a.M, a.N, a.parts ? 3 * a.K : a.K, a.batch, narrow ? 64 : 128, a.mul || add ? 128 : 256);
  CUtensorMap tmA, tmB;
  const bool a_shared = a.batch > 1 && a.sa == 0;  // one A for every batch item
  {
    const uint64_t dims[3] = {uint64_t(a.a_fold ? a.a_fold * 128 : a.K), uint64_t(a.M), uint64_t(a_shared ? 1 : a.parts ? 2 * a.batch : a.batch)};
    const uint64_t str[2] = {uint64_t(a.lda) * 2, uint64_t(a.sa > 0 ? a.sa : a.lda * a.M) * 2};
    const uint32_t box[3] = {64, 128, 1};
    if (int e = make_tmap_bf16(&tmA, a.A, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t dims[3] = {uint64_t(a.b_fold ? a.b_fold * 128 : a.K), uint64_t(a.b_rows ? a.b_rows : a.N), uint64_t(a.b_shared ? 1 : a.parts ? 2 * a.batch : a.batch)};
    const uint64_t str[2] = {uint64_t(a.ldb) * 2, uint64_t(a.sb > 0 ? a.sb : a.ldb * (a.b_rows ? a.b_rows : a.N)) * 2};
    const uint32_t box[3] = {64, uint32_t(BN), 1};
    if (int e = make_tmap_bf16(&tmB, a.B, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  BmmParams p;
  p.C = a.C;
  p.c_batch_stride = a.sc;
  p.ldc = int(a.ldc);
  p.m_valid = a.M;
  p.n_valid = a.N;
  p.tiles_m = (a.M + 127) / 128;
  p.tiles_n = (a.N + BN - 1) / BN;
  p.batch = a.batch;
  p.k_blocks = (a.K + 63) / 64 * (a.parts ? 3 : 1);
  p.part_blocks = a.parts ? (a.K + 63) / 64 : 0;
  p.part_batch = a.batch;
  p.mask = a.gate_mask;
  p.mask_pitch = a.mask_pitch;
  p.mask_n = a.mask_n;
  p.mask_line = a.mask_line;
  p.mask_pos = a.mask_pos;
  p.scale = a.scale;
  p.scale_ptr = a.scale_ptr;
  p.bias = a.bias;
  p.out_f32 = a.out_f32;
  p.opm_ntok = a.opm_ntok;
  p.residual = a.residual;
  p.a_shared = a_shared ? 1 : 0;
  p.b_shared = a.b_shared ? 1 : 0;
  p.a_fold = a.a_fold ? a.a_fold : INT_MAX;
  p.b_fold = a.b_fold ? a.b_fold : INT_MAX;
  p.tma_c = 0;
  CUtensorMap tmC = tmA;
  const int c_cols = 128 / c_esz;  // columns of one staging tile
  if (a.gate_mask) {
    const uint64_t dims[3] = {uint64_t(a.M), 256, uint64_t(a.N / 256)};
    const uint64_t str[2] = {uint64_t(a.M) * 2, uint64_t(a.sc) * 2};
    const uint32_t box[3] = {64, 128, 1};
    if (int e = make_tmap_bf16(&tmC, a.C, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
    p.tma_c = 1;
  } else if (a.row_groups > 0) {
    if (!bulk_c || a.out_f32 || a.residual || a.M != 32 * a.row_groups || a.group_stride % 8)
      return fail(B200_ERR_INVALID_ARGUMENT, "grouped rows need aligned bf16 bulk output");
    const uint64_t dims[4] = {uint64_t(a.N), 32, uint64_t(a.row_groups), uint64_t(a.batch)};
    const uint64_t str[3] = {uint64_t(a.ldc) * 2, uint64_t(a.group_stride) * 2, uint64_t(a.sc) * 2};
    const uint32_t box[4] = {64, 32, 4, 1};
    if (int e = make_tmap_bf16(&tmC, a.C, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
    p.tma_c = 3;
  } else if (bulk_c && (add || a.residual == nullptr || a.residual == a.C) && (a.bias == nullptr || aligned(a.bias, 16))) {
    uint64_t dims[3], str[2];
    uint32_t box[3];
    dims[0] = uint64_t(a.swiglu && !a.split ? a.N / 2 : a.N);
    box[0] = uint32_t(c_cols);
    dims[1] = uint64_t(a.M), dims[2] = uint64_t(a.batch);
    str[0] = uint64_t(a.ldc) * c_esz, str[1] = uint64_t(c_batch) * c_esz;
    box[1] = 128, box[2] = 1;
    if (int e = make_tmap(&tmC, a.out_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.C, 3, dims,
                          str, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return e;
    p.tma_c = a.residual && !add ? 2 : 1;
  }
  if ((a.mul || a.swiglu) && (!p.tma_c || (a.mul && (!aligned(a.mul, 16) || a.mul_pitch % 4 || a.batch != 1))))
    return fail(B200_ERR_INVALID_ARGUMENT, "a gated product needs bulk output and 16-byte aligned factors");
  CUtensorMap tmM = tmC;
  if (a.mul || (add && a.out_f32)) {
    const uint64_t dims[2] = {uint64_t(a.N), uint64_t(a.M)};
    const uint64_t str[1] = {uint64_t(add ? a.ldc : a.mul_pitch) * 4};
    const uint32_t box[2] = {32, 128};
    if (int e = make_tmap(&tmM, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, add ? a.residual : a.mul, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const int total = p.tiles_m * p.tiles_n * a.batch;
  const int grid = total < sm_count() ? total : sm_count();
  auto go = [&](auto bn, auto epi) -> int {
    B200_LAUNCH((bmm_nt_kernel<bn.value, epi.value>), grid, (BmmCfg<bn.value, epi.value>::THREADS), (BmmCfg<bn.value, epi.value>::SMEM_BYTES), stream, tmA, tmB, tmC,
                tmM, p);
    return 0;
  };
  auto pick = [&](auto bn) -> int {
    if (a.opm_ntok > 0) return go(bn, std::integral_constant<int, kEpiOuter>());
    if (a.swiglu) return go(bn, std::integral_constant<int, kEpiSwiglu>());
    if (!p.tma_c) return go(bn, std::integral_constant<int, kEpiDirect>());
    // Up to four K blocks the epilogue is the longer part of a tile; beyond, its warps are covered and the K stages that
    // the second pair of staging tiles takes the place of count (us, four warps against eight: 32768 x 768 x 128 29.1 / 21.7,
    // 128 x 256^3 10.0 / 8.5, 128 x 384^3 21.5 / 23.9, 512 x 40000 x 384 26.5 / 30.1).
    return p.k_blocks <= 4 ? go(bn, std::integral_constant<int, kEpiBulkWide>()) : go(bn, std::integral_constant<int, kEpiBulk>());
  };
  if (a.gate_mask) return go(std::integral_constant<int, 256>(), std::integral_constant<int, kEpiGateSplit>());
  if (a.split) return go(std::integral_constant<int, 256>(), std::integral_constant<int, kEpiSwigluSplit>());
  const auto bn64 = std::integral_constant<int, 64>();
  const auto bn128 = std::integral_constant<int, 128>();
  if (add && p.tma_c) return BN == 64 ? go(bn64, std::integral_constant<int, kEpiAdd>()) : go(bn128, std::integral_constant<int, kEpiAdd>());
  if (a.mul) return BN == 64 ? go(bn64, std::integral_constant<int, kEpiMul>()) : go(bn128, std::integral_constant<int, kEpiMul>());
  if (BN == 64) return go(bn64, std::integral_constant<int, kEpiBulk>());
  return BN == 256 ? pick(std::integral_constant<int, 256>()) : pick(std::integral_constant<int, 128>());
}

static int launch_rows_to_bf16(const void* x, bool f32, __nv_bfloat16* y, const float* w, const float* b,
                               int64_t rows, int cols, bool normalize, cudaStream_t stream, bool silu = false,
                               const void* x2 = nullptr, int cols1 = 0) {
  const int warps = 8;
  int64_t blocks = (rows + warps - 1) / warps;
  const int64_t cap = int64_t(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  if (!x2 && cols <= 128) {  // narrow rows: several rows per warp
    const int nn = normalize, ss = silu;
    if (cols <= 64) {
      if (f32) B200_LAUNCH(layernorm_rows_narrow_kernel<true, 8>, int(blocks), warps * 32, 0, stream, x, y, w, b, rows,
                           cols, 1e-5f, nn, ss);
      else B200_LAUNCH(layernorm_rows_narrow_kernel<false, 8>, int(blocks), warps * 32, 0, stream, x, y, w, b, rows, cols,
                       1e-5f, nn, ss);
    } else {
      if (f32) B200_LAUNCH(layernorm_rows_narrow_kernel<true, 16>, int(blocks), warps * 32, 0, stream, x, y, w, b, rows,
                           cols, 1e-5f, nn, ss);
      else B200_LAUNCH(layernorm_rows_narrow_kernel<false, 16>, int(blocks), warps * 32, 0, stream, x, y, w, b, rows,
                       cols, 1e-5f, nn, ss);
    }
    return 0;
  }
  if (f32)
    B200_LAUNCH(layernorm_rows_kernel<true>, int(blocks), warps * 32, 0, stream, x, y, w, b, rows, cols, 1e-5f, normalize,
                silu, x2, cols1);
  else
    B200_LAUNCH(layernorm_rows_kernel<false>, int(blocks), warps * 32, 0, stream, x, y, w, b, rows, cols, 1e-5f,
                normalize, silu, x2, cols1);
  return 0;
}

static int launch_adaln(const void* x, bool f32, const float* cond, int cw, int alpha_col, int beta_col, float lns,
                        __nv_bfloat16* y, void* x_copy, int64_t rows, int cols, cudaStream_t stream) {
  if (cols <= 128) {
    const int grid = grid_for(rows, 16);
    if (f32) B200_LAUNCH(adaln_rows_narrow_kernel<true>, grid, 256, 0, stream, x, cond, cw, alpha_col, beta_col, lns, y, x_copy, rows, cols, 1e-5f);
    else B200_LAUNCH(adaln_rows_narrow_kernel<false>, grid, 256, 0, stream, x, cond, cw, alpha_col, beta_col, lns, y, x_copy, rows, cols, 1e-5f);
    return 0;
  }
  const int grid = grid_for(rows, 8);
  if (f32) B200_LAUNCH(adaln_rows_kernel<true>, grid, 256, 0, stream, x, cond, cw, alpha_col, beta_col, lns, y, x_copy, rows, cols, 1e-5f);
  else B200_LAUNCH(adaln_rows_kernel<false>, grid, 256, 0, stream, x, cond, cw, alpha_col, beta_col, lns, y, x_copy, rows, cols, 1e-5f);
  return 0;
}

// Describes where the attention core finds its operands (all bf16, device memory).
struct FlashLaunch {
  const void* qk;        // rows of `qk_width` columns; Q heads at q_col0 + h*DH, K heads at k_col0 + h*DH
  int64_t qk_width;      // elements per row
  int64_t qk_b_stride;   // elements between batch items
  const void* vT;        // [Bt][H*DH][v_pitch]
  int64_t v_pitch;
  const void* bias;      // [groups*H][N][bias_pitch]
  int64_t bias_pitch;
  int bias_groups;
  FlashParams p;
};

// Tensor maps of the attention operands: Q / K tiles of DH columns, V^T tiles of v_rows rows, bias tiles.
static int flash_maps(const FlashLaunch& a, int DH, int v_rows, CUtensorMap* tmQ, CUtensorMap* tmV, CUtensorMap* tmB) {
  const FlashParams& p = a.p;
  {
    const uint64_t dims[3] = {uint64_t(a.qk_width), uint64_t(p.N), uint64_t(p.Bt)};
    const uint64_t str[2] = {uint64_t(a.qk_width) * 2, uint64_t(a.qk_b_stride) * 2};
    const uint32_t box[3] = {uint32_t(DH), 128, 1};
    if (int e = make_tmap_bf16(tmQ, a.qk, 3, dims, str, box, DH == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B))
      return e;
  }
  {
    const uint64_t dims[3] = {uint64_t(p.N), uint64_t(p.H) * DH, uint64_t(p.Bt)};
    const uint64_t str[2] = {uint64_t(a.v_pitch) * 2, uint64_t(a.v_pitch) * p.H * DH * 2};
    const uint32_t box[3] = {64, uint32_t(v_rows), 1};
    if (int e = make_tmap_bf16(tmV, a.vT, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t dims[3] = {uint64_t(p.N), uint64_t(p.N), uint64_t(a.bias_groups) * p.H};
    const uint64_t str[2] = {uint64_t(a.bias_pitch) * 2, uint64_t(a.bias_pitch) * p.N * 2};
    const uint32_t box[3] = {64, 128, 1};
    if (int e = make_tmap_bf16(tmB, a.bias, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  return 0;
}

template <int DH, int G>
static int launch_flash_core(const FlashLaunch& a, cudaStream_t stream) {
  using Cfg = FlashCfg<DH, G>;
  CUtensorMap tmQ, tmV, tmB;
  if (int e = flash_maps(a, DH, DH, &tmQ, &tmV, &tmB)) return e;
  FlashParams p = a.p;
  p.nqt = (p.N + 127) / 128;
  p.nkt = (p.N + 127) / 128;
  if (p.nkt > Cfg::MAX_T)
    return fail(B200_ERR_INVALID_ARGUMENT, "attention supports at most %d tokens (got %d)", Cfg::MAX_T * 128, p.N);
  p.nqg = (p.nqt + G - 1) / G;
  p.total_work = p.Bt * p.H * p.nqg;
  const int grid = p.total_work < sm_count() ? p.total_work : sm_count();
  B200_LAUNCH(flash_core_kernel<DH, G>, grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream, tmQ, tmQ, tmV, tmB, p);
  return 0;
}

template <int DH, int VR, int G>
static int launch_flash_resident(const FlashLaunch& a, cudaStream_t stream) {
  using Cfg = FlashResidentCfg<DH, VR, G>;
  CUtensorMap tmQ, tmV, tmB;
  if (int e = flash_maps(a, DH, VR, &tmQ, &tmV, &tmB)) return e;
  FlashParams p = a.p;
  p.nqt = (p.N + 127) / 128;
  p.nkt = (p.N + 127) / 128;
  p.npairs = (p.bias_div + G - 1) / G;
  p.total_work = (p.Bt + p.bias_div - 1) / p.bias_div * p.H * p.nqt * p.npairs;
  const int grid = p.total_work < sm_count() ? p.total_work : sm_count();
  B200_LAUNCH((flash_resident_kernel<DH, VR, G>), grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream, tmQ, tmV, tmB, p);
  return 0;
}

// Rows whose bias row block stays in shared memory go to flash_resident_kernel, longer ones to flash_core_kernel (why the
// line lies there: attention_resident.cuh).  A head of 64 columns with more than 48 of them in use does not leave room for
// two groups in tensor memory, nor, with the bias block, in shared memory.
static int launch_flash(const FlashLaunch& a, int DH, cudaStream_t stream) {
  const int tiles = (a.p.N + 127) / 128;
  if (DH == 32)
    return tiles <= FlashResidentCfg<32, 32, 2>::NB ? launch_flash_resident<32, 32, 2>(a, stream) : launch_flash_core<32, 2>(a, stream);
  if (a.p.dh_out <= 48 && tiles <= FlashResidentCfg<64, 48, 2>::NB) return launch_flash_resident<64, 48, 2>(a, stream);
  return launch_flash_core<64, 1>(a, stream);
}

// Lines that line_attention_kernel takes: one tile of queries and keys, four heads of 32, one wave of CTAs (a line each), the update
// added in place.
static bool line_attention_fits(const FlashLaunch& a) { return a.p.N <= 128 && a.p.H == 4 && a.p.dh_out == 32 && a.p.Bt <= sm_count(); }

// out: pair (line, pos) at out + line * line_stride + pos * pos_stride elements.
static int launch_line_attention(const FlashLaunch& a, const void* w_o, void* out, bool f32, int64_t line_stride, int64_t pos_stride,
                                 cudaStream_t stream) {
  CUtensorMap tmQ, tmV, tmB, tmW, tmO;
  if (int e = flash_maps(a, 32, 32, &tmQ, &tmV, &tmB)) return e;
  {
    const uint64_t dims[2] = {128, 128};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&tmW, w_o, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t esz = f32 ? 4 : 2;
    const uint64_t dims[3] = {uint64_t(kD), uint64_t(a.p.N), uint64_t(a.p.Bt)};
    const uint64_t str[2] = {uint64_t(pos_stride) * esz, uint64_t(line_stride) * esz};
    const uint32_t box[3] = {f32 ? 32u : 64u, 128, 1};
    if (int e = make_tmap(&tmO, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, out, 3, dims, str, box,
                          CU_TENSOR_MAP_SWIZZLE_128B))
      return e;
  }
  if (f32) B200_LAUNCH(line_attention_kernel<true>, a.p.Bt, line_attention::THREADS, line_attention::SMEM_BYTES, stream, tmQ, tmV, tmB, tmW, tmO, a.p);
  else B200_LAUNCH(line_attention_kernel<false>, a.p.Bt, line_attention::THREADS, line_attention::SMEM_BYTES, stream, tmQ, tmV, tmB, tmW, tmO, a.p);
  return 0;
}

static int launch_pair_bias(const void* z, bool f32, const float* ln_w, const float* ln_b, const void* w_z,
                            __nv_bfloat16* zb, int n_lines, int n_pos, long long z_line_stride, long long z_pos_stride,
                            long long out_plane, long long out_pitch, int H, cudaStream_t stream) {
  CUtensorMap tmW;
  const uint64_t dims[2] = {128, 16};
  const uint64_t str[1] = {256};
  const uint32_t box[2] = {64, 16};
  if (int e = make_tmap_bf16(&tmW, w_z, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  PairBiasParams p;
  p.z = z;
  p.ln_w = ln_w;
  p.ln_b = ln_b;
  p.zb = zb;
  p.n_lines = n_lines;
  p.n_pos = n_pos;
  p.z_line_stride = z_line_stride;
  p.z_pos_stride = z_pos_stride;
  p.out_plane = out_plane;
  p.out_pitch = out_pitch;
  p.H = H;
  p.num_tiles = n_lines * ((n_pos + 127) / 128);
  p.scale = 1.4426950408889634f;
  p.eps = 1e-5f;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  if (f32)
    B200_LAUNCH(pair_bias_kernel<true>, grid, pair_bias::THREADS, pair_bias::SMEM_BYTES, stream, tmW, p);
  else
    B200_LAUNCH(pair_bias_kernel<false>, grid, pair_bias::THREADS, pair_bias::SMEM_BYTES, stream, tmW, p);
  return 0;
}

template <bool F32, int SRC>
static int launch_ln_linear(const LnLinearParams& p, const void* w, float* out, cudaStream_t stream) {
  using Cfg = LnLinearCfg<SRC>;
  CUtensorMap tmW, tmO;
  {
    const uint64_t dims[2] = {128 * SRC, 128};
    const uint64_t str[1] = {256 * SRC};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&tmW, w, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t dims[2] = {128, uint64_t(p.rows)};
    const uint64_t str[1] = {512};
    const uint32_t box[2] = {32, 128};
    if (int e = make_tmap(&tmO, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  B200_LAUNCH((ln_linear_kernel<F32, SRC>), grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream, tmW, tmO, p);
  return 0;
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_version(void) { return 100; }

const char* b200_last_error(void) { return g_last_error; }

// Compute capability check only (cached per thread); *dev_out receives the current device ordinal.
static int check_arch(int* dev_out) {
  static thread_local int cached_dev = -1;
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  if (dev_out) *dev_out = dev;
  if (dev == cached_dev) return B200_OK;
  int major = 0;
  B200_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  if (major != 10)
    return fail(B200_ERR_UNSUPPORTED_DEVICE, "device %d has compute capability %d.x; this library is sm_100a only",
                dev, major);
  cached_dev = dev;
  return B200_OK;
}

// Host-visible copy of the device status word, one per device ordinal: 64 bytes of pinned, mapped host memory
// that a kernel writes when one of its bounded waits runs out (or it cannot run at all).  Set up by the first ordinary call on a device.
static int* g_host_status[64] = {nullptr};

static int ensure_host_status(int dev) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (g_host_status[dev]) return B200_OK;
  int* hp = nullptr;
  B200_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&hp), 64, cudaHostAllocMapped | cudaHostAllocPortable));
  *hp = 0;
  int* dp = nullptr;
  B200_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&dp), hp, 0));
  B200_CUDA(cudaMemcpyToSymbol(g_host_status_ptr, &dp, sizeof(dp)));
  g_host_status[dev] = hp;
  return B200_OK;
}

int b200_check_device(void) {
  int dev = 0;
  if (int e = check_arch(&dev)) return e;
  if (dev < 0 || dev >= 64) return B200_OK;
  if (!g_host_status[dev])
    if (int e = ensure_host_status(dev)) return e;
  const int st = *reinterpret_cast<volatile int*>(g_host_status[dev]);
  if (st != 0)
    return fail(B200_ERR_DEVICE_WAIT,
                "an earlier kernel on device %d %s (status %#x, site %d): its results and "
                "those of the kernels after it are invalid; b200_device_status() reads and clears the status",
                dev, (st & 0xff) == kDevMisaligned ? "found its shared memory misaligned" : "gave up a bounded wait", st, st >> 8);
  return B200_OK;
}

int b200_peek_status(int* status) {
  B200_CHECK_ARG(status != nullptr, "status is NULL");
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  *status = (dev >= 0 && dev < 64 && g_host_status[dev]) ? *reinterpret_cast<volatile int*>(g_host_status[dev]) : 0;
  return B200_OK;
}

unsigned long long b200_launch_count(void) { return g_launch_count.load(std::memory_order_relaxed); }

int b200_device_status(int* status) {
  B200_CHECK_ARG(status != nullptr, "status is NULL");
  B200_CUDA(cudaDeviceSynchronize());
  int v = 0;
  B200_CUDA(cudaMemcpyFromSymbol(&v, g_dev_status, sizeof(int)));
  if (v != 0) {
    const int zero = 0;
    B200_CUDA(cudaMemcpyToSymbol(g_dev_status, &zero, sizeof(int)));
  }
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && g_host_status[dev]) *reinterpret_cast<volatile int*>(g_host_status[dev]) = 0;
  *status = v;
  return B200_OK;
}

int b200_layernorm_fwd(const void* x, void* y, const float* w, const float* b, int64_t rows, int cols, float eps,
                       b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && y, "x/y is NULL");
  B200_CHECK_ARG(rows >= 0, "rows < 0");
  B200_CHECK_ARG(cols > 0 && cols % 8 == 0 && cols <= 1024, "cols=%d must be a multiple of 8 and <= 1024", cols);
  B200_CHECK_ARG(aligned(x, 16) && aligned(y, 16), "x/y must be 16-byte aligned");
  if (rows == 0) return B200_OK;
  const int warps = 8;
  int64_t blocks = (rows + warps - 1) / warps;
  const int64_t cap = int64_t(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  B200_LAUNCH(layernorm_rows_kernel<false>, int(blocks), warps * 32, 0, static_cast<cudaStream_t>(stream), x,
              static_cast<__nv_bfloat16*>(y), w, b, rows, cols, eps, 1, 0, nullptr, 0);
  return B200_OK;
}

int b200_bmm_nt_bf16(const void* A, const void* B, void* C, int batch, int M, int N, int K, int64_t lda,
                     int64_t ldb, int64_t ldc, int64_t sa, int64_t sb, int64_t sc, float scale,
                     b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(A && B && C, "A/B/C is NULL");
  B200_CHECK_ARG(batch > 0 && M > 0 && N > 0 && K > 0, "batch/M/N/K must be positive");
  B200_CHECK_ARG(N % 8 == 0, "N=%d must be a multiple of 8", N);
  B200_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0, "row pitches must be multiples of 8 elements");
  B200_CHECK_ARG(sa % 8 == 0 && sb % 8 == 0 && sc % 8 == 0, "batch strides must be multiples of 8 elements");
  B200_CHECK_ARG(batch == 1 || (sa > 0 && sb > 0), "batch strides must be positive");
  B200_CHECK_ARG(lda >= K && ldb >= K && ldc >= N, "row pitch smaller than the row");
  B200_CHECK_ARG(aligned(A, 16) && aligned(B, 16) && aligned(C, 16), "A/B/C must be 16-byte aligned");
  BmmLaunch a{A, B, C, batch, M, N, K, lda, ldb, ldc, sa, sb, sc};
  a.scale = scale;
  return launch_bmm(a, static_cast<cudaStream_t>(stream));
}

static inline int padded_n(int N) { return (N + 127) / 128 * 128; }

size_t b200_trimul_workspace_bytes(int N) {
  if (N <= 0) return 0;
  const size_t Np = size_t(padded_n(N));
  return 3 * size_t(kD) * Np * Np * sizeof(__nv_bfloat16);  // a, b, t
}

// Slab geometry of the two pair-walking kernels of triangle multiplication.
struct TriMulGeom {
  int n_lines, n_pos, lines_alloc, pos_pitch;
  long long z_line_stride, z_pos_stride;  // bytes
  long long m_line_stride, m_pos_stride;  // bytes
  int half_tiles;  // of 64 positions a line: those that hold one, or the whole pitch where a caller's product reads it
};

// Half tiles of a line of the two kernels: an odd number has them cut tiles across lines.  In one wave a tile a line takes no longer,
// and is spared the second division and store (PairMixer of 4 blocks, 48 tokens: 219 us, cut 223).
static int line_half_tiles(int n_lines, int n_pos, int pos_pitch) {
  return n_lines * (pos_pitch / 128) <= sm_count() ? pos_pitch / 64 : (n_pos + 63) / 64;
}

static int launch_trimul_project(const void* z, const uint8_t* mask, __nv_bfloat16* a_buf, __nv_bfloat16* b_buf,
                                 const b200_trimul_weights* w, const TriMulGeom& g, bool f32, cudaStream_t stream,
                                 long long z_copy_delta = 0) {
  CUtensorMap tmWin;
  const uint64_t dims[2] = {128, 512};
  const uint64_t str[1] = {256};
  const uint32_t box[2] = {64, 128};
  if (int e = make_tmap_bf16(&tmWin, w->w_in, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  CUtensorMap tmA, tmB;  // channel-major a/b planes, stored as [128 channels][64 pairs] boxes of one line
  {
    const uint64_t dims[3] = {uint64_t(g.pos_pitch), uint64_t(g.lines_alloc), uint64_t(kD)};
    const uint64_t str[2] = {uint64_t(g.pos_pitch) * 2, uint64_t(g.pos_pitch) * g.lines_alloc * 2};
    const uint32_t box[3] = {64, 1, 128};
    if (int e = make_tmap_bf16(&tmA, a_buf, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
    if (int e = make_tmap_bf16(&tmB, b_buf, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  TriMulInParams pi;
  pi.z = z;
  pi.mask = mask;
  pi.z_copy_delta = z_copy_delta;
  pi.ln_w = w->ln_in_w;
  pi.ln_b = w->ln_in_b;
  pi.a_out = a_buf;
  pi.b_out = b_buf;
  pi.n_lines = g.n_lines;
  pi.n_pos = g.n_pos;
  pi.lines_alloc = g.lines_alloc;
  pi.pos_pitch = g.pos_pitch;
  pi.z_line_stride = g.z_line_stride;
  pi.z_pos_stride = g.z_pos_stride;
  pi.m_line_stride = g.m_line_stride;
  pi.m_pos_stride = g.m_pos_stride;
  pi.half_tiles = g.half_tiles;
  pi.num_tiles = (g.n_lines * g.half_tiles + 1) / 2;
  pi.eps = 1e-5f;
  const int grid = pi.num_tiles < sm_count() ? pi.num_tiles : sm_count();
  auto go = [&](auto copy, auto half) -> int {
    if (f32) B200_LAUNCH((trimul_in_kernel<true, copy.value, half.value>), grid, trimul_in::THREADS, trimul_in::SMEM_BYTES, stream, tmWin, tmA, tmB, pi);
    else B200_LAUNCH((trimul_in_kernel<false, copy.value, half.value>), grid, trimul_in::THREADS, trimul_in::SMEM_BYTES, stream, tmWin, tmA, tmB, pi);
    return 0;
  };
  if (g.half_tiles & 1) return z_copy_delta ? go(std::true_type(), std::true_type()) : go(std::false_type(), std::true_type());
  return z_copy_delta ? go(std::true_type(), std::false_type()) : go(std::false_type(), std::false_type());
}

static int launch_trimul_output(const void* z, void* out, const __nv_bfloat16* t_buf, const b200_trimul_weights* w,
                                const TriMulGeom& g, bool add_residual, bool f32, cudaStream_t stream) {
  CUtensorMap tmWout, tmT;
  {
    const uint64_t dims[2] = {128, 256};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&tmWout, w->w_out, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t dims[3] = {uint64_t(g.pos_pitch), uint64_t(g.lines_alloc), uint64_t(kD)};
    const uint64_t str[2] = {uint64_t(g.pos_pitch) * 2, uint64_t(g.pos_pitch) * g.lines_alloc * 2};
    const uint32_t box[3] = {64, 1, 128};
    if (int e = make_tmap_bf16(&tmT, t_buf, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  // Output tiles [128 pairs][128 B of channels]; the dimension with the smaller stride comes first.
  CUtensorMap tmO;
  const bool pos_first = g.z_pos_stride <= g.z_line_stride;
  {
    const uint64_t np = uint64_t(g.n_pos), nl = uint64_t(g.n_lines);
    const uint64_t dims[3] = {uint64_t(kD), pos_first ? np : nl, pos_first ? nl : np};
    const uint64_t str[2] = {uint64_t(pos_first ? g.z_pos_stride : g.z_line_stride),
                             uint64_t(pos_first ? g.z_line_stride : g.z_pos_stride)};
    const uint32_t run = g.half_tiles & 1 ? 64 : 128;
    const uint32_t box[3] = {f32 ? 32u : 64u, pos_first ? run : 1u, pos_first ? 1u : run};
    if (int e = make_tmap(&tmO, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, out, 3, dims,
                          str, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return e;
  }
  TriMulOutParams po;
  po.z = z;
  po.out = out;
  po.ln_in_w = w->ln_in_w;
  po.ln_in_b = w->ln_in_b;
  po.ln_out_w = w->ln_out_w;
  po.ln_out_b = w->ln_out_b;
  po.n_lines = g.n_lines;
  po.n_pos = g.n_pos;
  po.pos_pitch = g.pos_pitch;
  po.z_line_stride = g.z_line_stride;
  po.z_pos_stride = g.z_pos_stride;
  po.pos_is_dim1 = pos_first ? 1 : 0;
  po.half_tiles = g.half_tiles;
  po.num_tiles = (g.n_lines * g.half_tiles + 1) / 2;
  po.add_residual = add_residual ? 1 : 0;
  po.eps = 1e-5f;
  const int grid = po.num_tiles < sm_count() ? po.num_tiles : sm_count();
  auto go = [&](auto half) -> int {
    if (f32) B200_LAUNCH((trimul_out_kernel<true, half.value>), grid, trimul_out::THREADS, trimul_out::SMEM_BYTES, stream, tmWout, tmT, tmO, po);
    else B200_LAUNCH((trimul_out_kernel<false, half.value>), grid, trimul_out::THREADS, trimul_out::SMEM_BYTES, stream, tmWout, tmT, tmO, po);
    return 0;
  };
  return g.half_tiles & 1 ? go(std::true_type()) : go(std::false_type());
}

static bool trimul_weights_ok(const b200_trimul_weights* w) {
  return w && w->w_in && w->w_out && w->ln_in_w && w->ln_in_b && w->ln_out_w && w->ln_out_b && aligned(w->w_in, 16) &&
         aligned(w->w_out, 16);
}

// Argument checks and the three launches of triangle multiplication; the callers have checked the device.  z_read: an event on another
// stream after which out may be written.
static int trimul_fwd_impl(const void* z, const uint8_t* mask, void* out, const b200_trimul_weights* w, int B, int N,
                           int incoming, int add_residual, int z_dtype, void* workspace, size_t workspace_bytes,
                           b200_stream_t stream_,
                           cudaEvent_t z_read = nullptr) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  B200_CHECK_ARG(z && mask && out && w, "z/mask/out/w is NULL");
  B200_CHECK_ARG(trimul_weights_ok(w), "a weight pointer is NULL or not 16-byte aligned");
  B200_CHECK_ARG(B > 0 && N > 0, "B=%d, N=%d must be positive", B, N);
  B200_CHECK_ARG(z_dtype == B200_DTYPE_BF16 || z_dtype == B200_DTYPE_F32, "unknown z_dtype %d", z_dtype);
  B200_CHECK_ARG(aligned(z, 32) && aligned(out, 32), "z/out must be 32-byte aligned");
  const bool f32 = z_dtype == B200_DTYPE_F32;
  const size_t esz = f32 ? 4 : 2;
  const size_t need = b200_trimul_workspace_bytes(N);
  if (!workspace || workspace_bytes < need || !aligned(workspace, 1024))
    return fail(B200_ERR_WORKSPACE, "workspace must be 1024-byte aligned and hold %zu bytes (got %zu)", need,
                workspace_bytes);
  const int Np = padded_n(N);
  const size_t plane = size_t(kD) * Np * Np;
  __nv_bfloat16* a_buf = static_cast<__nv_bfloat16*>(workspace);
  __nv_bfloat16* b_buf = a_buf + plane;
  __nv_bfloat16* t_buf = b_buf + plane;
  const long long row_b = (long long)N * kD * esz, col_b = (long long)kD * esz;
  // projection walks rows (outgoing) or columns (incoming); the output stage always walks rows
  const int halves = line_half_tiles(N, N, Np);
  TriMulGeom gin{N, N, Np, Np, incoming ? col_b : row_b, incoming ? row_b : col_b, incoming ? 1 : N, incoming ? N : 1, halves};
  TriMulGeom gout{N, N, Np, Np, row_b, col_b, 0, 0, halves};
  for (int bi = 0; bi < B; ++bi) {
    const uint8_t* zb = static_cast<const uint8_t*>(z) + size_t(bi) * N * N * kD * esz;
    uint8_t* ob = static_cast<uint8_t*>(out) + size_t(bi) * N * N * kD * esz;
    // z + update into another tensor: the projection stage copies z there, the output stage then adds in place (reading
    // the residual row by row in its epilogue took 84 us against 46 at N = 384)
    const bool copy = add_residual && ob != zb;
    if (int e = launch_trimul_project(zb, mask + size_t(bi) * N * N, a_buf, b_buf, w, gin, f32, stream, copy ? ob - zb : 0)) return e;
    {
      const int64_t plane_el = int64_t(Np) * Np;
      const int K = (N + 63) / 64 * 64;  // whole K blocks: the positions beyond N are zero
      BmmLaunch a{a_buf, b_buf, t_buf, kD, Np, Np, K, Np, Np, Np, plane_el, plane_el, plane_el};
      if (int e = launch_bmm(a, stream)) return e;
    }
    if (z_read && bi == 0) B200_CUDA(cudaStreamWaitEvent(stream, z_read, 0));
    if (int e = launch_trimul_output(copy ? ob : zb, ob, t_buf, w, gout, add_residual != 0, f32, stream)) return e;
  }
  return B200_OK;
}

int b200_trimul_fwd(const void* z, const uint8_t* mask, void* out, const b200_trimul_weights* w, int B, int N,
                    int incoming, int add_residual, int z_dtype, void* workspace, size_t workspace_bytes,
                    b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  return trimul_fwd_impl(z, mask, out, w, B, N, incoming, add_residual, z_dtype, workspace, workspace_bytes, stream);
}

// Staged form for sharded callers: the projection and output stages on a rectangular slab, the contraction
// (b200_bmm_nt) and whatever exchange the caller needs in between.
int b200_trimul_project(const void* z, const uint8_t* mask, void* a_out, void* b_out, const b200_trimul_weights* w,
                        int n_rows, int n_cols, int64_t z_row_stride, int64_t mask_row_stride, int incoming,
                        int pos_pitch, int z_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(z && mask && a_out && b_out, "z/mask/a_out/b_out is NULL");
  B200_CHECK_ARG(trimul_weights_ok(w), "a weight pointer is NULL or not 16-byte aligned");
  B200_CHECK_ARG(n_rows > 0 && n_cols > 0, "n_rows=%d, n_cols=%d must be positive", n_rows, n_cols);
  B200_CHECK_ARG((z_dtype | 1) == 1, "unknown z_dtype %d", z_dtype);
  const int n_pos = incoming ? n_rows : n_cols, n_lines = incoming ? n_cols : n_rows;
  B200_CHECK_ARG(pos_pitch % 128 == 0 && pos_pitch >= n_pos, "pos_pitch=%d must be a multiple of 128 and >= %d", pos_pitch,
                 n_pos);
  B200_CHECK_ARG(z_row_stride >= int64_t(n_cols) * kD && z_row_stride % 8 == 0 && mask_row_stride >= n_cols,
                 "row strides smaller than a row");
  B200_CHECK_ARG(aligned(z, 32) && aligned(a_out, 16) && aligned(b_out, 16), "z must be 32-byte aligned, a/b 16-byte");
  const bool f32 = z_dtype == B200_DTYPE_F32;
  const long long esz = f32 ? 4 : 2;
  const long long row_b = z_row_stride * esz, col_b = kD * esz;
  TriMulGeom g{n_lines, n_pos, n_lines, pos_pitch, incoming ? col_b : row_b, incoming ? row_b : col_b,
               incoming ? 1 : mask_row_stride, incoming ? mask_row_stride : 1, pos_pitch / 64};
  return launch_trimul_project(z, mask, static_cast<__nv_bfloat16*>(a_out), static_cast<__nv_bfloat16*>(b_out), w, g, f32,
                               static_cast<cudaStream_t>(stream));
}

int b200_trimul_output(const void* t, const void* z, void* out, const b200_trimul_weights* w, int n_rows, int n_cols,
                       int64_t z_row_stride, int transposed_t, int pos_pitch, int add_residual, int z_dtype,
                       b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(t && z && out, "t/z/out is NULL");
  B200_CHECK_ARG(trimul_weights_ok(w), "a weight pointer is NULL or not 16-byte aligned");
  B200_CHECK_ARG(n_rows > 0 && n_cols > 0, "n_rows=%d, n_cols=%d must be positive", n_rows, n_cols);
  B200_CHECK_ARG((z_dtype | 1) == 1, "unknown z_dtype %d", z_dtype);
  const int n_pos = transposed_t ? n_rows : n_cols, n_lines = transposed_t ? n_cols : n_rows;
  B200_CHECK_ARG(pos_pitch % 128 == 0 && pos_pitch >= n_pos, "pos_pitch=%d must be a multiple of 128 and >= %d", pos_pitch,
                 n_pos);
  B200_CHECK_ARG(z_row_stride >= int64_t(n_cols) * kD && z_row_stride % 8 == 0, "row stride smaller than a row");
  B200_CHECK_ARG(aligned(z, 32) && aligned(out, 32) && aligned(t, 16), "z/out must be 32-byte aligned, t 16-byte");
  const bool f32 = z_dtype == B200_DTYPE_F32;
  const long long esz = f32 ? 4 : 2;
  const long long row_b = z_row_stride * esz, col_b = kD * esz;
  TriMulGeom g{n_lines, n_pos, n_lines, pos_pitch, transposed_t ? col_b : row_b, transposed_t ? row_b : col_b, 0, 0,
               line_half_tiles(n_lines, n_pos, pos_pitch)};
  return launch_trimul_output(z, out, static_cast<const __nv_bfloat16*>(t), w, g, add_residual != 0, f32,
                              static_cast<cudaStream_t>(stream));
}

int b200_bmm_nt(const void* A, const void* B, void* C, int batch, int M, int N, int K, int64_t lda, int64_t ldb,
                int64_t ldc, int64_t a_batch_stride, int64_t b_batch_stride, int64_t c_batch_stride, float scale,
                int out_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(A && B && C, "A/B/C is NULL");
  B200_CHECK_ARG(batch > 0 && M > 0 && N > 0 && K > 0, "batch/M/N/K must be positive");
  B200_CHECK_ARG(N % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0, "N and the row pitches must be multiples of 8");
  B200_CHECK_ARG(a_batch_stride % 8 == 0 && b_batch_stride % 8 == 0 && c_batch_stride % 8 == 0,
                 "batch strides must be multiples of 8 elements");
  B200_CHECK_ARG(batch == 1 || (a_batch_stride >= 0 && b_batch_stride > 0),
                 "batch strides must be positive (a_batch_stride may be 0: one A shared by every batch item)");
  B200_CHECK_ARG(lda >= K && ldb >= K && ldc >= N, "row pitch smaller than the row");
  B200_CHECK_ARG((out_dtype | 1) == 1, "unknown out_dtype %d", out_dtype);
  B200_CHECK_ARG(aligned(A, 16) && aligned(B, 16) && aligned(C, 32), "A/B must be 16-byte aligned, C 32-byte aligned");
  BmmLaunch a{A, B, C, batch, M, N, K, lda, ldb, ldc, a_batch_stride, b_batch_stride, c_batch_stride};
  a.scale = scale;
  a.out_f32 = out_dtype == B200_DTYPE_F32;
  return launch_bmm(a, static_cast<cudaStream_t>(stream));
}

int b200_transition_hidden_fwd(const void* x, void* out, const void* w13, const void* w3, const float* ln_w, const float* ln_b,
                               int64_t rows, int hidden, int use_norm, int add_residual, int x_dtype, b200_stream_t stream_) {
  if (int e = b200_check_device()) return e;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  B200_CHECK_ARG(x && out && w13 && w3, "x/out/w13/w3 is NULL");
  B200_CHECK_ARG(hidden == 512 || hidden == 256, "hidden=%d must be 256 or 512", hidden);
  B200_CHECK_ARG(!use_norm || (ln_w && ln_b), "use_norm needs ln_w and ln_b");
  B200_CHECK_ARG(rows >= 0 && rows < (int64_t(1) << 31), "rows out of range");
  B200_CHECK_ARG(x_dtype == B200_DTYPE_BF16 || x_dtype == B200_DTYPE_F32, "unknown x_dtype %d", x_dtype);
  B200_CHECK_ARG(aligned(x, 32) && aligned(out, 32) && aligned(w13, 16) && aligned(w3, 16),
                 "x/out must be 32-byte aligned, weights 16-byte aligned");
  if (rows == 0) return B200_OK;
  CUtensorMap tmW1, tmW3;
  {
    const uint64_t dims[2] = {128, uint64_t(2 * hidden)};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&tmW1, w13, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t dims[2] = {uint64_t(hidden), 128};
    const uint64_t str[1] = {uint64_t(hidden) * 2};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&tmW3, w3, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const bool f32 = x_dtype == B200_DTYPE_F32;
  CUtensorMap tmO;  // output rows, [128 rows][64 B] boxes
  {
    const uint64_t dims[2] = {uint64_t(kD), uint64_t(rows)};
    const uint64_t str[1] = {uint64_t(kD) * (f32 ? 4 : 2)};
    const uint32_t box[2] = {f32 ? 16u : 32u, 128};
    if (int e = make_tmap(&tmO, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, out, 2, dims, str, box,
                          CU_TENSOR_MAP_SWIZZLE_64B))
      return e;
  }
  TransitionParams p;
  p.x = x;
  p.out = out;
  p.ln_w = use_norm ? ln_w : nullptr;
  p.ln_b = use_norm ? ln_b : nullptr;
  p.rows = rows;
  p.num_tiles = int((rows + 127) / 128);
  p.use_norm = use_norm ? 1 : 0;
  p.add_residual = add_residual ? 1 : 0;
  p.eps = 1e-5f;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  if (hidden == 512) {
    if (f32) B200_LAUNCH((transition_kernel<true, 8>), grid, transition::THREADS, transition::SMEM_BYTES, stream, tmW1, tmW3, tmO, p);
    else B200_LAUNCH((transition_kernel<false, 8>), grid, transition::THREADS, transition::SMEM_BYTES, stream, tmW1, tmW3, tmO, p);
  } else {
    if (f32) B200_LAUNCH((transition_kernel<true, 4>), grid, transition::THREADS, transition::SMEM_BYTES, stream, tmW1, tmW3, tmO, p);
    else B200_LAUNCH((transition_kernel<false, 4>), grid, transition::THREADS, transition::SMEM_BYTES, stream, tmW1, tmW3, tmO, p);
  }
  return B200_OK;
}

int b200_transition_fwd(const void* x, void* out, const void* w13, const void* w3, const float* ln_w, const float* ln_b,
                        int64_t rows, int use_norm, int add_residual, int x_dtype, b200_stream_t stream) {
  return b200_transition_hidden_fwd(x, out, w13, w3, ln_w, ln_b, rows, 512, use_norm, add_residual, x_dtype, stream);
}

int b200_ln_linear_fwd(const void* x1, const void* x2, const float* ln_w, const float* ln_b, const void* w,
                       const float* residual, float* out, int64_t rows, int x_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x1 && w && out, "x1/w/out is NULL");
  B200_CHECK_ARG(rows >= 0 && rows < (int64_t(1) << 31), "rows out of range");
  B200_CHECK_ARG((x_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x1, 32) && aligned(x2, 32) && aligned(w, 16) && aligned(out, 32) && aligned(residual, 32),
                 "x1/x2/out/residual must be 32-byte aligned, w 16-byte aligned");
  if (rows == 0) return B200_OK;
  LnLinearParams p{x1, x2, ln_w, ln_b, residual, rows, int((rows + 127) / 128), 1e-5f};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool f32 = x_dtype == B200_DTYPE_F32;
  if (x2) return f32 ? launch_ln_linear<true, 2>(p, w, out, st) : launch_ln_linear<false, 2>(p, w, out, st);
  return f32 ? launch_ln_linear<true, 1>(p, w, out, st) : launch_ln_linear<false, 1>(p, w, out, st);
}

int b200_pair_cond_fwd(const void* x1, const void* x2, const float* ln_w, const float* ln_b, const void* w,
                       const b200_transition_weights* transitions, int n_transitions, float* out, int64_t rows, int x_dtype,
                       b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x1 && x2 && w && transitions && out, "x1/x2/w/transitions/out is NULL");
  B200_CHECK_ARG(n_transitions > 0 && n_transitions <= kPairCondMaxTransitions, "n_transitions=%d must be 1..%d", n_transitions,
                 kPairCondMaxTransitions);
  B200_CHECK_ARG(rows >= 0 && rows < (int64_t(1) << 31), "rows out of range");
  B200_CHECK_ARG((x_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x1, 32) && aligned(x2, 32) && aligned(w, 16) && aligned(out, 32),
                 "x1/x2/out must be 32-byte aligned, w 16-byte aligned");
  for (int t = 0; t < n_transitions; ++t) {
    const b200_transition_weights& tw = transitions[t];
    B200_CHECK_ARG(tw.hidden == 256 && tw.w13 && tw.w3 && aligned(tw.w13, 16) && aligned(tw.w3, 16), "transition %d: bad weights", t);
    B200_CHECK_ARG(tw.ln_w && tw.ln_b, "transition %d: bad LayerNorm", t);
  }
  if (rows == 0) return B200_OK;
  PairCondMaps maps;
  memset(&maps, 0, sizeof(maps));
  PairCondParams p{x1, x2, ln_w, ln_b, {}, {}, rows, int((rows + 127) / 128), n_transitions, 1e-5f};
  {
    const uint64_t dims[2] = {256, 128};
    const uint64_t str[1] = {512};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&maps.w0, w, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  for (int t = 0; t < n_transitions; ++t) {
    const uint64_t dims13[2] = {128, 512}, dims3[2] = {256, 128};
    const uint64_t str13[1] = {256}, str3[1] = {512};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&maps.w13[t], transitions[t].w13, 2, dims13, str13, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
    if (int e = make_tmap_bf16(&maps.w3[t], transitions[t].w3, 2, dims3, str3, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
    p.t_ln_w[t] = transitions[t].ln_w;
    p.t_ln_b[t] = transitions[t].ln_b;
  }
  {
    const uint64_t dims[2] = {uint64_t(kD), uint64_t(rows)};
    const uint64_t str[1] = {uint64_t(kD) * 4};
    const uint32_t box[2] = {32, 128};
    if (int e = make_tmap(&maps.out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (x_dtype == B200_DTYPE_F32) B200_LAUNCH(pair_cond_kernel<true>, grid, pair_cond::THREADS, pair_cond::SMEM_BYTES, st, maps, p);
  else B200_LAUNCH(pair_cond_kernel<false>, grid, pair_cond::THREADS, pair_cond::SMEM_BYTES, st, maps, p);
  return B200_OK;
}

// ------------------------------------------------------------------------------------------------ no-allocation variant
// Scratch for b200_trimul_fwd_static: the three channel-major planes a, b, t for N <= 256 (padded to 256),
// plus slack so the base can be rounded up to the 1024-byte alignment the kernels' launcher asks for.
// It lives in the library image: every GPU that loads the library holds these 48 MiB until the process exits.
#define B200_STATIC_TRIMUL_MAX_N 256
static __device__ __align__(256) unsigned char g_trimul_static_scratch[size_t(3) * 128 * 256 * 256 * 2 + 1024];

// Device address of the scratch per device ordinal, resolved on first use with that device current.
// (In host code the array's name is only a handle for the runtime, never a pointer a kernel may be given.)
static void* g_trimul_static_ptr[64] = {nullptr};

int b200_trimul_fwd_static(const void* z, const uint8_t* mask, void* out, const b200_trimul_weights* w, int B, int N,
                           int incoming, int add_residual, int z_dtype, b200_stream_t stream) {
  // Only the compute-capability check: the ordinary entry points also set up a pinned status word on their first
  // call, which is an allocation this entry point promises not to make.
  if (int e = check_arch(nullptr)) return e;
  B200_CHECK_ARG(N > 0 && N <= B200_STATIC_TRIMUL_MAX_N,
                 "b200_trimul_fwd_static handles N <= %d (got %d); use b200_trimul_fwd with a caller workspace",
                 B200_STATIC_TRIMUL_MAX_N, N);
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  B200_CHECK_ARG(dev >= 0 && dev < 64, "device ordinal %d out of range", dev);
  if (!g_trimul_static_ptr[dev]) {
    void* ptr = nullptr;
    B200_CUDA(cudaGetSymbolAddress(&ptr, g_trimul_static_scratch));
    g_trimul_static_ptr[dev] = ptr;
  }
  uintptr_t base = (reinterpret_cast<uintptr_t>(g_trimul_static_ptr[dev]) + 1023) & ~uintptr_t(1023);
  return trimul_fwd_impl(z, mask, out, w, B, N, incoming, add_residual, z_dtype, reinterpret_cast<void*>(base),
                         b200_trimul_workspace_bytes(N), stream);
}

// ------------------------------------------------------------------------------------------------ OPM
static void opm_plan(int S, int N, int* Sp, int* CI, size_t* ab_bytes, size_t* outer_bytes) {
  *Sp = (S + 7) / 8 * 8;
  const size_t per_tok = size_t(N) * 1024 * 2;               // bytes of outer products for one token row
  // Chunks near 1 GiB: an L2-sized chunk (48 MB) was measured slower, 0.58 ms against 0.42 ms for a 1024 x 384 MSA
  // (five times the launches, each with a tail).
  size_t ci = (size_t(1) << 30) / per_tok;
  ci = ci / 4 * 4;
  if (ci < 4) ci = 4;
  const size_t n4 = size_t(N + 3) / 4 * 4;
  if (ci > n4) ci = n4;
  *CI = int(ci);
  *ab_bytes = (size_t(N) * 32 * size_t(*Sp) * 2 + 1023) / 1024 * 1024;
  *outer_bytes = (ci * per_tok + 1023) / 1024 * 1024;
}

size_t b200_opm_workspace_bytes(int S, int N) {
  if (S <= 0 || N <= 0) return 0;
  int Sp, CI;
  size_t ab, outer;
  opm_plan(S, N, &Sp, &CI, &ab, &outer);
  return 2 * ab + outer + 1024;
}

// j0, nj: the token columns of the output to compute (all N rows always); ext_scale: device scalar replacing
// 1 / (number of valid MSA rows) -- for a caller that holds only part of the MSA depth; add_bias: whether proj_o's bias
// is added (exactly one of the partial results that are later summed should carry it).
static int opm_run(const void* m, const uint8_t* mask, int mask_ndim, void* out, const b200_opm_weights* w, int B,
                   int S, int N, int j0, int nj, const float* ext_scale, bool add_bias, int m_dtype, int out_dtype,
                   void* workspace, size_t workspace_bytes, b200_stream_t stream_, const float* residual = nullptr) {
  if (int e = b200_check_device()) return e;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  B200_CHECK_ARG(m && mask && out && w, "m/mask/out/w is NULL");
  B200_CHECK_ARG(w->w_ab && w->w_o && w->ln_w && w->ln_b && w->bias_o, "a weight pointer is NULL");
  B200_CHECK_ARG(B > 0 && S > 0 && N > 0, "B=%d, S=%d, N=%d must be positive", B, S, N);
  B200_CHECK_ARG(mask_ndim == 3 || (mask_ndim == 2 && B == 1), "mask must be [B,S,N], or [B,N] with B == 1");
  B200_CHECK_ARG((m_dtype | 1) == 1 && (out_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(m, 32) && aligned(out, 32) && aligned(w->w_ab, 16) && aligned(w->w_o, 16),
                 "m/out must be 32-byte aligned, weights 16-byte aligned");
  const size_t need = b200_opm_workspace_bytes(S, N);
  if (!workspace || workspace_bytes < need || !aligned(workspace, 1024))
    return fail(B200_ERR_WORKSPACE, "workspace must be 1024-byte aligned and hold %zu bytes (got %zu)", need,
                workspace_bytes);
  int Sp, CI;
  size_t ab_bytes, outer_bytes;
  opm_plan(S, N, &Sp, &CI, &ab_bytes, &outer_bytes);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __nv_bfloat16* aT = reinterpret_cast<__nv_bfloat16*>(ws);
  __nv_bfloat16* bT = reinterpret_cast<__nv_bfloat16*>(ws + ab_bytes);
  __nv_bfloat16* outer = reinterpret_cast<__nv_bfloat16*>(ws + 2 * ab_bytes);
  float* inv = reinterpret_cast<float*>(ws + 2 * ab_bytes + outer_bytes);

  CUtensorMap tmW;
  {
    const uint64_t dims[2] = {64, 64};
    const uint64_t str[1] = {128};
    const uint32_t box[2] = {64, 64};
    if (int e = make_tmap_bf16(&tmW, w->w_ab, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const size_t m_esz = m_dtype == B200_DTYPE_F32 ? 4 : 2;
  const size_t o_esz = out_dtype == B200_DTYPE_F32 ? 4 : 2;

  for (int bi = 0; bi < B; ++bi) {
    OpmProjParams pp;
    pp.m = static_cast<const uint8_t*>(m) + size_t(bi) * S * N * 64 * m_esz;
    pp.mask = mask + (mask_ndim == 3 ? size_t(bi) * S * N : 0);
    pp.mask_s_stride = mask_ndim == 3 ? N : 0;
    pp.ln_w = w->ln_w;
    pp.ln_b = w->ln_b;
    pp.aT = aT;
    pp.bT = bT;
    pp.S = S;
    pp.N = N;
    pp.Sp = Sp;
    pp.num_tiles = N * ((S + 127) / 128);
    pp.eps = 1e-5f;
    pp.row_counters = reinterpret_cast<int*>(inv) + 1;
    const int grid = pp.num_tiles < 2 * sm_count() ? pp.num_tiles : 2 * sm_count();
    if (m_dtype == B200_DTYPE_F32)
      B200_LAUNCH(opm_proj_kernel<true>, grid, opm_proj::THREADS, opm_proj::SMEM_BYTES, stream, tmW, pp);
    else
      B200_LAUNCH(opm_proj_kernel<false>, grid, opm_proj::THREADS, opm_proj::SMEM_BYTES, stream, tmW, pp);
    const float* scale_ptr = ext_scale;
    if (mask_ndim == 3 && !ext_scale) {
      B200_LAUNCH(opm_inv_row_count_kernel, grid_for(S, 8), 256, 0, stream, pp.mask, S, N, pp.row_counters, inv);
      scale_ptr = inv;
    }
    for (int i0 = 0; i0 < N; i0 += CI) {
      const int ci = (N - i0) < CI ? (N - i0) : CI;
      {
        BmmLaunch a{aT + size_t(i0) * 32 * Sp, bT + size_t(j0) * 32 * Sp, outer, 1, ci * 32, nj * 32, S, Sp, Sp, 0, 0, 0, 0};
        a.scale_ptr = scale_ptr;
        a.opm_ntok = nj;
        if (int e = launch_bmm(a, stream)) return e;
      }
      {
        void* dst = static_cast<uint8_t*>(out) + (size_t(bi) * N * nj + size_t(i0) * nj) * 128 * o_esz;
        BmmLaunch a{outer, w->w_o, dst, 1, ci * nj, 128, 1024, 1024, 1024, 128, 0, 0, 0};
        a.bias = add_bias ? w->bias_o : nullptr;
        a.out_f32 = out_dtype == B200_DTYPE_F32;
        if (residual) a.residual = residual + (size_t(bi) * N * nj + size_t(i0) * nj) * 128;
        if (int e = launch_bmm(a, stream)) return e;
      }
    }
  }
  return B200_OK;
}

int b200_opm_fwd(const void* m, const uint8_t* mask, int mask_ndim, void* out, const b200_opm_weights* w, int B,
                 int S, int N, int m_dtype, int out_dtype, void* workspace, size_t workspace_bytes,
                 b200_stream_t stream) {
  return opm_run(m, mask, mask_ndim, out, w, B, S, N, 0, N, nullptr, true, m_dtype, out_dtype, workspace, workspace_bytes,
                 stream);
}

int b200_opm_add_fwd(const void* m, const uint8_t* mask, int mask_ndim, const float* residual, float* out,
                     const b200_opm_weights* w, int B, int S, int N, int m_dtype, void* workspace, size_t workspace_bytes,
                     b200_stream_t stream) {
  B200_CHECK_ARG(residual && residual != out && aligned(residual, 16), "residual must be 16-byte aligned and not the output");
  return opm_run(m, mask, mask_ndim, out, w, B, S, N, 0, N, nullptr, true, m_dtype, B200_DTYPE_F32, workspace, workspace_bytes,
                 stream, residual);
}

int b200_opm_cols_fwd(const void* m, const uint8_t* mask, void* out, const b200_opm_weights* w, int S, int N, int j0,
                      int nj, const float* scale, int add_bias, int m_dtype, int out_dtype, void* workspace,
                      size_t workspace_bytes, b200_stream_t stream) {
  if (j0 < 0 || nj <= 0 || j0 + nj > N) return fail(B200_ERR_INVALID_ARGUMENT, "column range [%d, %d) outside [0, %d)", j0, j0 + nj, N);
  if (!scale) return fail(B200_ERR_INVALID_ARGUMENT, "scale is NULL");
  return opm_run(m, mask, 3, out, w, 1, S, N, j0, nj, scale, add_bias != 0, m_dtype, out_dtype, workspace, workspace_bytes,
                 stream);
}

// ------------------------------------------------------------------------------------------------ attention core
int b200_attention_core_fwd(const b200_attention_core_args* a, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(a != nullptr, "args is NULL");
  B200_CHECK_ARG(a->qk && a->vT && a->bias && a->mask && a->out, "qk/vT/bias/mask/out is NULL");
  B200_CHECK_ARG(a->head_dim_padded == 32 || a->head_dim_padded == 64, "head_dim_padded must be 32 or 64");
  B200_CHECK_ARG(a->N > 0 && a->H > 0 && a->batch > 0, "N/H/batch must be positive");
  B200_CHECK_ARG(a->head_dim_out > 0 && a->head_dim_out % 8 == 0 && a->head_dim_out <= a->head_dim_padded,
                 "head_dim_out must be a multiple of 8 and <= head_dim_padded");
  B200_CHECK_ARG(a->qk_width % 8 == 0 && a->v_pitch % 8 == 0 && a->bias_pitch % 8 == 0 && a->out_pitch % 8 == 0 &&
                     a->q_col0 % 8 == 0 && a->k_col0 % 8 == 0 && a->out_col0 % 8 == 0 && a->gate_col0 % 8 == 0 &&
                     a->gate_pitch % 8 == 0,
                 "pitches and column offsets must be multiples of 8 elements");
  B200_CHECK_ARG(a->bias_div > 0 && a->mask_div > 0 && a->bias_groups > 0, "bias_div/mask_div/bias_groups must be positive");
  B200_CHECK_ARG(aligned(a->qk, 16) && aligned(a->vT, 16) && aligned(a->bias, 16) && aligned(a->out, 16) &&
                     (!a->gate || aligned(a->gate, 16)), "operands must be 16-byte aligned");
  FlashLaunch l;
  l.qk = a->qk;
  l.qk_width = a->qk_width;
  l.qk_b_stride = a->qk_batch_stride;
  l.vT = a->vT;
  l.v_pitch = a->v_pitch;
  l.bias = a->bias;
  l.bias_pitch = a->bias_pitch;
  l.bias_groups = a->bias_groups;
  FlashParams& p = l.p;
  p.mask = a->mask;
  p.mask_div = a->mask_div;
  p.mask_row_stride = a->mask_row_stride;
  p.mask_key_stride = a->mask_key_stride;
  p.bias_div = a->bias_div;
  p.gate = static_cast<const __nv_bfloat16*>(a->gate);
  p.gate_activated = 0;
  p.gate_b_stride = a->gate_batch_stride;
  p.gate_pitch = a->gate_pitch;
  p.gate_col0 = a->gate_col0;
  p.out = static_cast<__nv_bfloat16*>(a->out);
  p.out_b_stride = a->out_batch_stride;
  p.out_pitch = a->out_pitch;
  p.out_col0 = a->out_col0;
  p.dh_out = a->head_dim_out;
  p.N = a->N;
  p.H = a->H;
  p.Bt = a->batch;
  p.q_col0 = a->q_col0;
  p.k_col0 = a->k_col0;
  p.v_row0 = 0;
  return launch_flash(l, a->head_dim_padded, static_cast<cudaStream_t>(stream));
}

// ------------------------------------------------------------------------------------------------ APB
struct ApbPlan {
  int dh, DH, W1, Nk;
  size_t off_sln, off_qkg, off_vT, off_zb, off_og, total;
};

static bool apb_plan(int B, int M, int N, int c_s, int H, ApbPlan* pl) {
  if (H <= 0 || H > 16 || c_s % H != 0) return false;
  pl->dh = c_s / H;
  if (pl->dh % 8 != 0 || pl->dh > 64 || c_s % 8 != 0) return false;
  pl->DH = pl->dh <= 32 ? 32 : 64;
  pl->W1 = 2 * H * pl->DH + c_s;
  pl->Nk = (N + 7) / 8 * 8;
  const size_t rows = size_t(B) * M * N;
  auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  size_t o = 0;
  pl->off_sln = o; o += up(rows * c_s * 2);
  pl->off_qkg = o; o += up(rows * pl->W1 * 2);
  pl->off_vT = o;  o += up(size_t(B) * M * H * pl->DH * pl->Nk * 2);
  pl->off_zb = o;  o += up(size_t(B) * H * N * pl->Nk * 2);
  pl->off_og = o;  o += up(rows * c_s * 2);
  pl->total = o;
  return true;
}

size_t b200_apb_workspace_bytes(int B, int M, int N, int c_s, int H) {
  ApbPlan pl;
  if (B <= 0 || M <= 0 || N <= 0 || !apb_plan(B, M, N, c_s, H, &pl)) return 0;
  return pl.total;
}

// Where the output projection goes instead of `out`: x += mul * (its result), x of its own dtype.
struct ApbOutput {
  void* x;
  bool f32;
  const float* mul;
  int mul_pitch;
};

static int apb_run(const void* s, const void* z, const void* ext_bias, int64_t ext_bias_pitch, const uint8_t* mask,
                   void* out, const b200_apb_weights* w, int B, int M, int N, int c_s, int H, int s_dtype, int z_dtype,
                   bool add_residual, void* workspace, size_t workspace_bytes, b200_stream_t stream_,
                   const ApbOutput* into = nullptr) {
  if (int e = b200_check_device()) return e;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  B200_CHECK_ARG(s && (z || ext_bias) && mask && out && w, "s/z/mask/out/w is NULL");
  B200_CHECK_ARG(w->w_qkg && w->b_qkg && w->w_v && w->w_z && w->ln_z_w && w->w_o, "a weight pointer is NULL");
  B200_CHECK_ARG(B > 0 && M > 0 && N > 0, "B=%d, M=%d, N=%d must be positive", B, M, N);
  B200_CHECK_ARG((s_dtype | 1) == 1 && (z_dtype | 1) == 1, "unknown dtype");
  ApbPlan pl;
  B200_CHECK_ARG(apb_plan(B, M, N, c_s, H, &pl),
                 "unsupported c_s=%d, H=%d: need H <= 16, head dim a multiple of 8 and <= 64", c_s, H);
  B200_CHECK_ARG(aligned(s, 32) && (!z || aligned(z, 32)) && aligned(out, 32), "s/z/out must be 32-byte aligned");
  B200_CHECK_ARG(!ext_bias || (aligned(ext_bias, 16) && ext_bias_pitch % 8 == 0 && ext_bias_pitch >= N),
                 "bias must be 16-byte aligned with a pitch that is a multiple of 8 and >= N");
  if (!workspace || workspace_bytes < pl.total || !aligned(workspace, 1024))
    return fail(B200_ERR_WORKSPACE, "workspace must be 1024-byte aligned and hold %zu bytes (got %zu)", pl.total,
                workspace_bytes);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __nv_bfloat16* s_ln = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_sln);
  __nv_bfloat16* qkg = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_qkg);
  __nv_bfloat16* vT = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_vT);
  __nv_bfloat16* zb = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_zb);
  __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_og);
  const int BM = B * M;
  const int64_t rows = int64_t(BM) * N;
  const int HD = H * pl.DH;

  // 1. LayerNorm (or plain conversion) of the single track; bf16 rows without a LayerNorm are used as they are
  if (!w->ln_s_w && s_dtype == B200_DTYPE_BF16) {
    s_ln = static_cast<__nv_bfloat16*>(const_cast<void*>(s));
  } else if (int e = launch_rows_to_bf16(s, s_dtype == B200_DTYPE_F32, s_ln, w->ln_s_w, w->ln_s_b, rows, c_s,
                                         w->ln_s_w != nullptr, stream)) {
    return e;
  }
  // 2. q | k | g projection (heads padded to DH, q pre-scaled) and V^T per batch item
  {
    BmmLaunch a{s_ln, w->w_qkg, qkg, 1, int(rows), pl.W1, c_s, c_s, c_s, pl.W1, 0, 0, 0};
    a.bias = w->b_qkg;
    if (int e = launch_bmm(a, stream)) return e;
  }
  {  // one launch for all batch items: they share the A operand
    BmmLaunch a{w->w_v, s_ln, vT, BM, HD, N, c_s, c_s, c_s, pl.Nk, 0, int64_t(N) * c_s, int64_t(HD) * pl.Nk};
    if (int e = launch_bmm(a, stream)) return e;
  }
  // 3. pair bias, one pass over z per batch element (unless the caller supplies it)
  const size_t z_esz = z_dtype == B200_DTYPE_F32 ? 4 : 2;
  for (int b = 0; b < B && !ext_bias; ++b) {
    if (int e = launch_pair_bias(static_cast<const uint8_t*>(z) + size_t(b) * N * N * kD * z_esz,
                                 z_dtype == B200_DTYPE_F32, w->ln_z_w, w->ln_z_b, w->w_z,
                                 zb + size_t(b) * H * N * pl.Nk, N, N, (long long)N * kD * z_esz, (long long)kD * z_esz,
                                 (long long)N * pl.Nk, pl.Nk, H, stream))
      return e;
  }
  // 4. attention core
  {
    FlashLaunch a;
    a.qk = qkg;
    a.qk_width = pl.W1;
    a.qk_b_stride = int64_t(N) * pl.W1;
    a.vT = vT;
    a.v_pitch = pl.Nk;
    a.bias = ext_bias ? ext_bias : static_cast<const void*>(zb);
    a.bias_pitch = ext_bias ? ext_bias_pitch : pl.Nk;
    a.bias_groups = B;
    FlashParams& p = a.p;
    p.mask = mask;
    p.mask_div = M;
    p.mask_row_stride = N;
    p.mask_key_stride = 1;
    p.bias_div = M;
    p.gate = qkg;
    p.gate_activated = 0;
    p.gate_b_stride = int64_t(N) * pl.W1;
    p.gate_pitch = pl.W1;
    p.gate_col0 = 2 * HD;
    p.out = og;
    p.out_b_stride = int64_t(N) * c_s;
    p.out_pitch = c_s;
    p.out_col0 = 0;
    p.dh_out = pl.dh;
    p.N = N;
    p.H = H;
    p.Bt = BM;
    p.q_col0 = 0;
    p.k_col0 = HD;
    p.v_row0 = 0;
    if (int e = launch_flash(a, pl.DH, stream)) return e;
  }
  // 5. output projection
  {
    BmmLaunch a{og, w->w_o, out, 1, int(rows), c_s, c_s, c_s, c_s, c_s, 0, 0, 0};
    a.out_f32 = s_dtype == B200_DTYPE_F32;
    a.residual = add_residual ? s : nullptr;
    if (into) {
      a.C = into->x;
      a.residual = into->x;
      a.out_f32 = into->f32;
      a.mul = into->mul;
      a.mul_pitch = into->mul_pitch;
    }
    if (int e = launch_bmm(a, stream)) return e;
  }
  return B200_OK;
}

int b200_apb_fwd(const void* s, const void* z, const uint8_t* mask, void* out, const b200_apb_weights* w, int B,
                 int M, int N, int c_s, int H, int s_dtype, int z_dtype, void* workspace, size_t workspace_bytes,
                 b200_stream_t stream) {
  if (!z) return fail(B200_ERR_INVALID_ARGUMENT, "z is NULL");
  return apb_run(s, z, nullptr, 0, mask, out, w, B, M, N, c_s, H, s_dtype, z_dtype, false, workspace,
                 workspace_bytes, stream);
}

int b200_apb_fwd_bias(const void* s, const void* bias, int64_t bias_pitch, const uint8_t* mask, void* out,
                      const b200_apb_weights* w, int B, int M, int N, int c_s, int H, int s_dtype, void* workspace,
                      size_t workspace_bytes, b200_stream_t stream) {
  if (!bias) return fail(B200_ERR_INVALID_ARGUMENT, "bias is NULL");
  return apb_run(s, nullptr, bias, bias_pitch, mask, out, w, B, M, N, c_s, H, s_dtype, B200_DTYPE_F32, false,
                 workspace, workspace_bytes, stream);
}

int b200_pair_bias_fwd(const void* z, const float* ln_w, const float* ln_b, const void* w_z, void* out, int n_rows,
                       int n_cols, int64_t z_row_stride, int64_t out_plane, int64_t out_pitch, int H, int transposed,
                       int z_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(z && ln_w && w_z && out, "z/ln_w/w_z/out is NULL");
  B200_CHECK_ARG(n_rows > 0 && n_cols > 0 && H > 0 && H <= 16, "n_rows/n_cols must be positive, 1 <= H <= 16");
  B200_CHECK_ARG((z_dtype | 1) == 1, "unknown z_dtype %d", z_dtype);
  B200_CHECK_ARG(z_row_stride >= int64_t(n_cols) * kD && z_row_stride % 8 == 0, "row stride smaller than a row");
  const int n_lines = transposed ? n_cols : n_rows, n_pos = transposed ? n_rows : n_cols;
  B200_CHECK_ARG(out_pitch >= n_pos && out_plane >= int64_t(n_lines) * out_pitch, "output pitch/plane too small");
  B200_CHECK_ARG(aligned(z, 32) && aligned(w_z, 16), "z must be 32-byte aligned, w_z 16-byte aligned");
  const long long esz = z_dtype == B200_DTYPE_F32 ? 4 : 2;
  const long long row_b = z_row_stride * esz, col_b = kD * esz;
  return launch_pair_bias(z, z_dtype == B200_DTYPE_F32, ln_w, ln_b, w_z, static_cast<__nv_bfloat16*>(out), n_lines, n_pos,
                          transposed ? col_b : row_b, transposed ? row_b : col_b, out_plane, out_pitch, H,
                          static_cast<cudaStream_t>(stream));
}

// ------------------------------------------------------------------------------------------------ triangle attention
// A slab holds `lines` complete attention rows: for the starting node a line is a row of z (the slab must span all
// columns), for the ending node a line is a column (the slab must span all rows); `pos` is the token axis attended over.
struct TriAttPlan {
  int lines, pos, Nk;
  size_t off_qkg, off_vT, off_tb, off_og, total;
};

static void triatt_plan(int lines, int pos, bool own_bias, TriAttPlan* pl) {
  pl->lines = lines;
  pl->pos = pos;
  pl->Nk = (pos + 7) / 8 * 8;
  auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  size_t o = 0;
  pl->off_qkg = o; o += up(size_t(lines) * pos * 384 * 2);
  pl->off_vT = o;  o += up(size_t(lines) * kD * pl->Nk * 2);
  pl->off_tb = o;  o += own_bias ? up(size_t(4) * pos * pl->Nk * 2) : 0;
  pl->off_og = o;  o += up(size_t(lines) * pos * kD * 2);
  pl->total = o;
}

static int triatt_slab(const void* z, const uint8_t* mask, const void* ext_bias, int64_t ext_bias_pitch, void* out,
                       const b200_triatt_weights* w, int n_rows, int n_cols, bool ending, bool add_residual, bool f32,
                       void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  const int lines = ending ? n_cols : n_rows, pos = ending ? n_rows : n_cols;
  TriAttPlan pl;
  triatt_plan(lines, pos, ext_bias == nullptr, &pl);
  if (!workspace || workspace_bytes < pl.total || !aligned(workspace, 1024))
    return fail(B200_ERR_WORKSPACE, "workspace must be 1024-byte aligned and hold %zu bytes (got %zu)", pl.total,
                workspace_bytes);
  if (!ext_bias && n_rows != n_cols)
    return fail(B200_ERR_INVALID_ARGUMENT, "a rectangular slab needs the triangle bias of the whole pair tensor");
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __nv_bfloat16* qkg = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_qkg);
  __nv_bfloat16* vT = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_vT);
  __nv_bfloat16* tb = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_tb);
  __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_og);
  const long long esz = f32 ? 4 : 2;
  const long long row_b = (long long)n_cols * kD * esz, col_b = kD * esz;
  const long long line_b = ending ? col_b : row_b, pos_b = ending ? row_b : col_b;

  CUtensorMap tmW;
  {
    const uint64_t dims[2] = {128, 512};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 128};
    if (int e = make_tmap_bf16(&tmW, w->w_qkgv, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  const int half_tiles = line_half_tiles(lines, pos, (pos + 127) / 128 * 128);
  CUtensorMap tmQKG, tmVT;  // [128 rows][64 values] boxes: a tile's (or a run's 64) pairs x channels of q|k|g, channels x keys of V^T
  {
    const uint64_t dims[3] = {384, uint64_t(pos), uint64_t(lines)};
    const uint64_t str[2] = {768, uint64_t(pos) * 768};
    const uint32_t box[3] = {64, half_tiles & 1 ? 64u : 128u, 1};
    if (int e = make_tmap_bf16(&tmQKG, qkg, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  {
    const uint64_t dims[3] = {uint64_t(pos), uint64_t(kD), uint64_t(lines)};
    const uint64_t str[2] = {uint64_t(pl.Nk) * 2, uint64_t(pl.Nk) * kD * 2};
    const uint32_t box[3] = {64, 128, 1};
    if (int e = make_tmap_bf16(&tmVT, vT, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  CUtensorMap tmWB;  // the 8 rows of the bias weights that hold the 4 heads, as two 64-channel halves
  {
    const uint64_t dims[2] = {128, 16};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 8};
    if (int e = make_tmap_bf16(&tmWB, w->w_b, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return e;
  }
  TriAttProjParams pp;
  pp.z = z;
  pp.ln_w = w->ln_w;
  pp.ln_b = w->ln_b;
  pp.g_bias = w->g_bias;
  pp.qkg = qkg;
  pp.vT = vT;
  pp.n_lines = lines;
  pp.n_pos = pos;
  pp.Nk = pl.Nk;
  pp.z_line_stride = line_b;
  pp.z_pos_stride = pos_b;
  pp.half_tiles = half_tiles;
  pp.num_tiles = (lines * half_tiles + 1) / 2;
  pp.eps = 1e-5f;
  // Without a bias from the caller the projection kernel writes the triangle bias of the same rows itself.
  pp.tri_bias = ext_bias ? nullptr : tb;
  pp.bias_plane = (long long)pos * pl.Nk;
  pp.bias_pitch = pl.Nk;
  pp.bias_scale = 1.4426950408889634f;
  const int grid = pp.num_tiles < sm_count() ? pp.num_tiles : sm_count();
  auto go = [&](auto half) -> int {
    if (f32) B200_LAUNCH((triatt_proj_kernel<true, half.value>), grid, triatt_proj::THREADS, triatt_proj::SMEM_BYTES, stream, tmW, tmQKG, tmVT, tmWB, pp);
    else B200_LAUNCH((triatt_proj_kernel<false, half.value>), grid, triatt_proj::THREADS, triatt_proj::SMEM_BYTES, stream, tmW, tmQKG, tmVT, tmWB, pp);
    return 0;
  };
  if (int e = half_tiles & 1 ? go(std::true_type()) : go(std::false_type())) return e;
  {
    FlashLaunch a;
    a.qk = qkg;
    a.qk_width = 384;
    a.qk_b_stride = int64_t(pos) * 384;
    a.vT = vT;
    a.v_pitch = pl.Nk;
    a.bias = ext_bias ? ext_bias : static_cast<const void*>(tb);
    a.bias_pitch = ext_bias ? ext_bias_pitch : pl.Nk;
    a.bias_groups = 1;
    FlashParams& p = a.p;
    p.mask = mask;
    p.mask_div = 1;
    // line l attends over keys k with mask[l][k] (starting node) or mask[k][l] (ending node)
    p.mask_row_stride = ending ? 1 : n_cols;
    p.mask_key_stride = ending ? n_cols : 1;
    p.bias_div = lines;
    p.gate = qkg;
    p.gate_activated = 1;  // the projection kernel stores sigmoid(g)
    p.gate_b_stride = int64_t(pos) * 384;
    p.gate_pitch = 384;
    p.gate_col0 = 256;
    p.out = og;
    p.out_b_stride = int64_t(pos) * kD;
    p.out_pitch = kD;
    p.out_col0 = 0;
    p.dh_out = 32;
    p.N = pos;
    p.H = 4;
    p.Bt = lines;
    p.q_col0 = 0;
    p.k_col0 = 128;
    p.v_row0 = 0;
    if (add_residual && out == z && line_attention_fits(a))
      return launch_line_attention(a, w->w_o, out, f32, line_b / esz, pos_b / esz, stream);
    if (int e = launch_flash(a, 32, stream)) return e;
  }
  {
    // Pair (line, pos) of the ending node lives in row pos * lines + line: a batch item per line, its rows a line of pairs apart, so
    // that lines of any length leave by TMA tiles (stored by the lanes where a line is not whole tiles of 128: 20 us against 10 for
    // 203 tokens).  In bf16 those lines are read back and rounded once, 13 us.  The starting node's and lines of whole tiles are reduced
    // into memory, with a rounding of the update and one of the sum: read back, a whole call takes 72 us instead of 66 at 256
    // tokens and 316 instead of 300 at 512.
    BmmLaunch a{og, w->w_o, out, 1, lines * pos, kD, kD, kD, kD, kD, 0, 0, 0};
    if (ending) {
      a.batch = lines, a.M = pos, a.ldc = int64_t(lines) * kD;
      a.sa = int64_t(pos) * kD, a.sc = kD;
      a.b_shared = true;
    }
    a.out_f32 = f32;
    a.residual = add_residual ? z : nullptr;
    a.round_once = ending && !f32 && pos % 128 != 0;
    if (int e = launch_bmm(a, stream)) return e;
  }
  return B200_OK;
}

static bool triatt_weights_ok(const b200_triatt_weights* w) {
  return w && w->w_qkgv && w->g_bias && w->w_b && w->w_o && w->ln_w && w->ln_b;
}

size_t b200_triatt_workspace_bytes(int N) {
  if (N <= 0) return 0;
  TriAttPlan pl;
  triatt_plan(N, N, true, &pl);
  return pl.total;
}

size_t b200_triatt_slab_workspace_bytes(int n_rows, int n_cols, int ending) {
  if (n_rows <= 0 || n_cols <= 0) return 0;
  TriAttPlan pl;
  triatt_plan(ending ? n_cols : n_rows, ending ? n_rows : n_cols, false, &pl);
  return pl.total;
}

int b200_triatt_fwd(const void* z, const uint8_t* mask, void* out, const b200_triatt_weights* w, int B, int N,
                    int ending, int add_residual, int z_dtype, void* workspace, size_t workspace_bytes,
                    b200_stream_t stream_) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(z && mask && out, "z/mask/out is NULL");
  B200_CHECK_ARG(triatt_weights_ok(w), "a weight pointer is NULL");
  B200_CHECK_ARG(B > 0 && N > 0, "B=%d, N=%d must be positive", B, N);
  B200_CHECK_ARG((z_dtype | 1) == 1, "unknown z_dtype %d", z_dtype);
  B200_CHECK_ARG(aligned(z, 32) && aligned(out, 32), "z/out must be 32-byte aligned");
  const bool f32 = z_dtype == B200_DTYPE_F32;
  const size_t esz = f32 ? 4 : 2;
  for (int bi = 0; bi < B; ++bi) {
    const size_t off = size_t(bi) * N * N * kD * esz;
    if (int e = triatt_slab(static_cast<const uint8_t*>(z) + off, mask + size_t(bi) * N * N, nullptr, 0,
                            static_cast<uint8_t*>(out) + off, w, N, N, ending != 0, add_residual != 0, f32, workspace,
                            workspace_bytes, static_cast<cudaStream_t>(stream_)))
      return e;
  }
  return B200_OK;
}

int b200_triatt_slab_fwd(const void* z, const uint8_t* mask, const void* bias, int64_t bias_pitch, void* out,
                         const b200_triatt_weights* w, int n_rows, int n_cols, int ending, int add_residual, int z_dtype,
                         void* workspace, size_t workspace_bytes, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(z && mask && bias && out, "z/mask/bias/out is NULL");
  B200_CHECK_ARG(triatt_weights_ok(w), "a weight pointer is NULL");
  B200_CHECK_ARG(n_rows > 0 && n_cols > 0, "n_rows=%d, n_cols=%d must be positive", n_rows, n_cols);
  B200_CHECK_ARG((z_dtype | 1) == 1, "unknown z_dtype %d", z_dtype);
  B200_CHECK_ARG(aligned(z, 32) && aligned(out, 32) && aligned(bias, 16), "z/out must be 32-byte aligned, bias 16-byte");
  const int pos = ending ? n_rows : n_cols;
  B200_CHECK_ARG(bias_pitch % 8 == 0 && bias_pitch >= pos, "bias pitch must be a multiple of 8 and >= %d", pos);
  return triatt_slab(z, mask, bias, bias_pitch, out, w, n_rows, n_cols, ending != 0, add_residual != 0,
                     z_dtype == B200_DTYPE_F32, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

// ------------------------------------------------------------------------------------------------ single-track helpers

int b200_rows_to_bf16(const void* x, void* y, const float* w, const float* b, int64_t rows, int cols, int x_dtype,
                      int normalize, int silu, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && y, "x/y is NULL");
  B200_CHECK_ARG(rows >= 0 && cols > 0 && cols % 8 == 0 && cols <= 1024, "cols=%d must be a multiple of 8, <= 1024", cols);
  B200_CHECK_ARG((x_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x, 32) && aligned(y, 16), "x must be 32-byte aligned, y 16-byte aligned");
  if (rows == 0) return B200_OK;
  return launch_rows_to_bf16(x, x_dtype == B200_DTYPE_F32, static_cast<__nv_bfloat16*>(y), w, b, rows, cols,
                             normalize != 0, static_cast<cudaStream_t>(stream), silu != 0);
}

int b200_rows2_to_bf16(const void* x1, int cols1, const void* x2, int cols2, void* y, const float* w, const float* b,
                       int64_t rows, int x_dtype, int normalize, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x1 && x2 && y, "x1/x2/y is NULL");
  B200_CHECK_ARG(rows >= 0 && cols1 > 0 && cols2 > 0 && cols1 % 8 == 0 && cols2 % 8 == 0 && cols1 + cols2 <= 1024,
                 "cols1=%d and cols2=%d must be positive multiples of 8 with a sum <= 1024", cols1, cols2);
  B200_CHECK_ARG((x_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x1, 32) && aligned(x2, 32) && aligned(y, 16), "x1/x2 must be 32-byte aligned, y 16-byte aligned");
  if (rows == 0) return B200_OK;
  return launch_rows_to_bf16(x1, x_dtype == B200_DTYPE_F32, static_cast<__nv_bfloat16*>(y), w, b, rows, cols1 + cols2,
                             normalize != 0, static_cast<cudaStream_t>(stream), false, x2, cols1);
}

int b200_window_bias_fwd(const void* z, const float* ln_w, const float* ln_b, const float* w_z, float* bias,
                         int64_t windows, int W, int Hk, int c_z, int heads, int z_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(z && ln_w && w_z && bias, "z/ln_w/w_z/bias is NULL");
  B200_CHECK_ARG(windows >= 0 && W > 0 && Hk > 0, "need windows >= 0 and W, Hk > 0");
  B200_CHECK_ARG(c_z > 0 && c_z % 4 == 0 && c_z <= 128, "c_z=%d must be a multiple of 4, at most 128", c_z);
  B200_CHECK_ARG(aligned(z, 16) && aligned(bias, 4), "z must be 16-byte aligned");
  B200_CHECK_ARG(heads > 0 && heads <= kWindowMaxHeads, "heads=%d must be in 1..%d", heads, kWindowMaxHeads);
  B200_CHECK_ARG((z_dtype | 1) == 1, "unknown dtype");
  if (windows == 0) return B200_OK;
  WindowBiasParams p{z, ln_w, ln_b, w_z, bias, windows * W * Hk, W * Hk, c_z, heads, 1e-5f};
  if (c_z == 16 && aligned(z, 32)) {
    const int grid = grid_for(p.pairs, 256);
    if (z_dtype == B200_DTYPE_F32) B200_LAUNCH(window_bias16_kernel<true>, grid, 256, 0, static_cast<cudaStream_t>(stream), p);
    else B200_LAUNCH(window_bias16_kernel<false>, grid, 256, 0, static_cast<cudaStream_t>(stream), p);
    return B200_OK;
  }
  int lpr = 1;
  while (lpr * 4 < c_z) lpr *= 2;  // lanes per pair: four channels each
  const int grid = grid_for(p.pairs * lpr, 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (z_dtype == B200_DTYPE_F32) B200_LAUNCH(window_bias_kernel<true>, grid, 256, 0, st, p, lpr);
  else B200_LAUNCH(window_bias_kernel<false>, grid, 256, 0, st, p, lpr);
  return B200_OK;
}

// qkv / gate rows of qkv_pitch / gate_pitch elements.
static int window_attention_run(const void* qkv, int qkv_pitch, const void* gate, int gate_pitch, const float* bias,
                                const uint8_t* mask, void* out, int B, int M, int NW, int W, int Hk, int heads, int head_dim,
                                cudaStream_t st) {
  B200_CHECK_ARG(qkv && gate && bias && mask && out, "qkv/gate/bias/mask/out is NULL");
  B200_CHECK_ARG(B > 0 && M > 0 && NW > 0 && W > 0 && Hk >= W && Hk % 8 == 0 && (Hk - W) % 2 == 0,
                 "need B, M, NW, W > 0 and Hk >= W, a multiple of 8, with Hk - W even (W=%d, Hk=%d)", W, Hk);
  B200_CHECK_ARG(heads > 0 && heads * W <= 256, "heads * W = %d exceeds the 256 threads of a window's CTA", heads * W);
  B200_CHECK_ARG(head_dim == 16 || head_dim == 32 || head_dim == 64, "head_dim=%d must be 16, 32 or 64", head_dim);
  B200_CHECK_ARG(2ll * Hk * heads * head_dim * 2 + Hk + 16 <= 227 * 1024, "the key window does not fit in shared memory");
  B200_CHECK_ARG((int64_t)B * M * NW < (int64_t(1) << 31), "too many windows");
  B200_CHECK_ARG(aligned(qkv, 16) && aligned(gate, 16) && aligned(out, 16) && aligned(bias, 16),
                 "qkv/gate/out/bias must be 16-byte aligned");
  WindowAttnParams p{static_cast<const __nv_bfloat16*>(qkv), static_cast<const __nv_bfloat16*>(gate), qkv_pitch, gate_pitch,
                     bias, mask, static_cast<__nv_bfloat16*>(out), NW, W, Hk, heads, M, 1.0f / sqrtf(float(head_dim))};
  if (head_dim == 16) return launch_window_attention<16>(p, B * M, st);
  if (head_dim == 32) return launch_window_attention<32>(p, B * M, st);
  return launch_window_attention<64>(p, B * M, st);
}

// The pair bias and the attention of all samples: one kernel where it serves the shapes, else by way of `bias`.
static int window_pair_run(const void* qkv, int qkv_pitch, const void* gate, int gate_pitch, const void* z, const float* ln_w,
                           const float* ln_b, const float* w_z, const uint8_t* mask, void* out, float* bias, int B, int M, int NW,
                           int W, int Hk, int heads, int head_dim, int c_z, int z_dtype, cudaStream_t st) {
  const WindowPairParams p{{static_cast<const __nv_bfloat16*>(qkv), static_cast<const __nv_bfloat16*>(gate), qkv_pitch, gate_pitch, nullptr,
                            mask, static_cast<__nv_bfloat16*>(out), NW, W, Hk, heads, M, 1.0f / sqrtf(float(head_dim))},
                           z, ln_w, ln_b, w_z, 1e-5f, 1};
  const bool args = qkv && gate && z && ln_w && w_z && mask && out && B > 0 && M > 0 && NW > 0 && W > 0 && heads > 0 &&
                    (z_dtype | 1) == 1 && aligned(qkv, 16) && aligned(gate, 16) && aligned(out, 16);
  if (!args || !window_pair_fits(p.a, B, head_dim, c_z, z)) {  // the two calls check their arguments
    if (int e = b200_window_bias_fwd(z, ln_w, ln_b, w_z, bias, int64_t(B) * NW, W, Hk, c_z, heads, z_dtype, st)) return e;
    return window_attention_run(qkv, qkv_pitch, gate, gate_pitch, bias, mask, out, B, M, NW, W, Hk, heads, head_dim, st);
  }
  const bool f32 = z_dtype == B200_DTYPE_F32;
  return head_dim == 16 ? launch_window_pair<16>(p, B, f32, st) : launch_window_pair<32>(p, B, f32, st);
}

int b200_window_pair_attention_fwd(const void* qkv, int qkv_pitch, const void* gate, int gate_pitch, const void* z,
                                   const float* ln_w, const float* ln_b, const float* w_z, const uint8_t* mask, void* out,
                                   float* bias, int B, int M, int NW, int W, int Hk, int heads, int head_dim, int c_z,
                                   int z_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(qkv_pitch >= 3 * heads * head_dim && gate_pitch >= heads * head_dim && qkv_pitch % 8 == 0 && gate_pitch % 8 == 0,
                 "pitches must be multiples of 8 and hold a row");
  B200_CHECK_ARG(bias, "bias is NULL");
  return window_pair_run(qkv, qkv_pitch, gate, gate_pitch, z, ln_w, ln_b, w_z, mask, out, bias, B, M, NW, W, Hk, heads, head_dim,
                         c_z, z_dtype, static_cast<cudaStream_t>(stream));
}

int b200_window_attention_fwd(const void* qkv, const void* gate, const float* bias, const uint8_t* mask, void* out, int B,
                              int M, int NW, int W, int Hk, int heads, int head_dim, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  return window_attention_run(qkv, 3 * heads * head_dim, gate, heads * head_dim, bias, mask, out, B, M, NW, W, Hk, heads, head_dim,
                              static_cast<cudaStream_t>(stream));
}

int b200_window_attention_pitched_fwd(const void* qkv, int qkv_pitch, const void* gate, int gate_pitch, const float* bias,
                                      const uint8_t* mask, void* out, int B, int M, int NW, int W, int Hk, int heads,
                                      int head_dim, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(qkv_pitch >= 3 * heads * head_dim && gate_pitch >= heads * head_dim && qkv_pitch % 8 == 0 && gate_pitch % 8 == 0,
                 "pitches must be multiples of 8 and hold a row");
  return window_attention_run(qkv, qkv_pitch, gate, gate_pitch, bias, mask, out, B, M, NW, W, Hk, heads, head_dim,
                              static_cast<cudaStream_t>(stream));
}

int b200_pair_outer_sum(const float* a, const float* c, const float* extra, float* z, int n_i, int n_j, int cols,
                        b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(a && c && z, "a/c/z is NULL");
  B200_CHECK_ARG(n_i >= 0 && n_j >= 0 && cols > 0 && cols % 8 == 0, "cols=%d must be a positive multiple of 8", cols);
  B200_CHECK_ARG(aligned(a, 32) && aligned(c, 32) && aligned(z, 32) && (!extra || aligned(extra, 32)),
                 "a/c/extra/z must be 32-byte aligned");
  if (n_i == 0 || n_j == 0) return B200_OK;
  B200_LAUNCH(pair_outer_sum_kernel, grid_for((int64_t)n_i * n_j * (cols / 8), 256), 256, 0,
              static_cast<cudaStream_t>(stream), a, c, extra, z, n_i, n_j, cols);
  return B200_OK;
}

int b200_msa_features(const float* msa, const float* has_deletion, const float* deletion_value, const float* paired, void* out,
                      int64_t rows, int nt, int pitch, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(msa && has_deletion && deletion_value && out, "msa/has_deletion/deletion_value/out is NULL");
  B200_CHECK_ARG(rows >= 0 && nt > 0 && pitch % 8 == 0 && pitch >= int64_t(nt) + (paired ? 3 : 2),
                 "need nt > 0 and a pitch that is a multiple of 8 and holds every feature (nt=%d, pitch=%d)", nt, pitch);
  B200_CHECK_ARG(aligned(msa, 4) && aligned(has_deletion, 4) && aligned(deletion_value, 4) && (!paired || aligned(paired, 4)) &&
                     aligned(out, 16),
                 "out must be 16-byte aligned");
  if (rows == 0) return B200_OK;
  B200_LAUNCH(msa_features_kernel, grid_for(rows * (pitch / 8), 256), 256, 0, static_cast<cudaStream_t>(stream), msa, has_deletion,
              deletion_value, paired, static_cast<__nv_bfloat16*>(out), rows, nt, pitch);
  return B200_OK;
}

int b200_add_rows(const float* x, const void* y, float* out, int64_t rows, int64_t period, int cols, int y_dtype,
                  b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && y && out, "x/y/out is NULL");
  B200_CHECK_ARG(rows >= 0 && period > 0 && cols > 0 && cols % 8 == 0, "need period > 0 and cols a positive multiple of 8");
  B200_CHECK_ARG((y_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x, 32) && aligned(y, 32) && aligned(out, 32), "x/y/out must be 32-byte aligned");
  if (rows == 0) return B200_OK;
  const int grid = grid_for(rows * (cols / 8), 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (y_dtype == B200_DTYPE_F32) B200_LAUNCH(add_rows_kernel<true>, grid, 256, 0, st, x, y, out, rows, period, cols);
  else B200_LAUNCH(add_rows_kernel<false>, grid, 256, 0, st, x, y, out, rows, period, cols);
  return B200_OK;
}

int b200_linear_bf16(const void* x, const void* w, const float* bias, const void* residual, void* out, int64_t rows,
                     int in_features, int out_features, int out_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && w && out, "x/w/out is NULL");
  B200_CHECK_ARG(rows > 0 && rows < (int64_t(1) << 31), "rows out of range");
  B200_CHECK_ARG(in_features > 0 && in_features % 8 == 0 && out_features > 0 && out_features % 8 == 0,
                 "in_features=%d and out_features=%d must be positive multiples of 8", in_features, out_features);
  B200_CHECK_ARG((out_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x, 16) && aligned(w, 16) && aligned(out, 32) && (!residual || aligned(residual, 32)),
                 "x/w must be 16-byte aligned, out/residual 32-byte aligned");
  BmmLaunch a{x, w, out, 1, int(rows), out_features, in_features, in_features, in_features, out_features, 0, 0, 0};
  a.bias = bias;
  a.residual = residual;
  a.out_f32 = out_dtype == B200_DTYPE_F32;
  return launch_bmm(a, static_cast<cudaStream_t>(stream));
}

int b200_swiglu_fwd(const void* h12, void* h, int64_t rows, int hidden, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(h12 && h, "h12/h is NULL");
  B200_CHECK_ARG(rows >= 0 && hidden > 0 && hidden % 8 == 0, "hidden=%d must be a positive multiple of 8", hidden);
  B200_CHECK_ARG(aligned(h12, 16) && aligned(h, 16), "h12/h must be 16-byte aligned");
  if (rows == 0) return B200_OK;
  B200_LAUNCH(swiglu_rows_kernel, grid_for(rows * (hidden / 8), 256), 256, 0, static_cast<cudaStream_t>(stream),
              static_cast<const __nv_bfloat16*>(h12), static_cast<__nv_bfloat16*>(h), rows, hidden);
  return B200_OK;
}

int b200_adaln_fwd(const void* x, const float* cond, int cond_width, int alpha_col, int beta_col, float lns, void* y,
                   int64_t rows, int cols, int x_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && cond && y, "x/cond/y is NULL");
  B200_CHECK_ARG(rows >= 0 && cols > 0 && cols % 8 == 0 && cols <= 1024, "cols=%d must be a multiple of 8, <= 1024", cols);
  B200_CHECK_ARG(cond_width % 8 == 0 && alpha_col % 8 == 0 && beta_col % 8 == 0 && alpha_col + cols <= cond_width &&
                     beta_col + cols <= cond_width, "bad conditioning layout");
  B200_CHECK_ARG((x_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x, 32) && aligned(cond, 32) && aligned(y, 16), "x/cond must be 32-byte aligned, y 16-byte");
  if (rows == 0) return B200_OK;
  return launch_adaln(x, x_dtype == B200_DTYPE_F32, cond, cond_width, alpha_col, beta_col, lns, static_cast<__nv_bfloat16*>(y),
                      nullptr, rows, cols, static_cast<cudaStream_t>(stream));
}

int b200_gated_residual_fwd(void* x, const void* h, const float* cond, int cond_width, int gamma_col, int64_t rows,
                            int cols, int x_dtype, int h_dtype, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && h && cond, "x/h/cond is NULL");
  B200_CHECK_ARG(rows >= 0 && cols > 0 && cols % 8 == 0, "cols=%d must be a positive multiple of 8", cols);
  B200_CHECK_ARG(cond_width % 8 == 0 && gamma_col % 8 == 0 && gamma_col + cols <= cond_width, "bad conditioning layout");
  B200_CHECK_ARG((x_dtype | 1) == 1 && (h_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x, 32) && aligned(h, 32) && aligned(cond, 32), "x/h/cond must be 32-byte aligned");
  if (rows == 0) return B200_OK;
  const int grid = grid_for(rows * (cols / 8), 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool xf = x_dtype == B200_DTYPE_F32, hf = h_dtype == B200_DTYPE_F32;
  if (xf && hf) B200_LAUNCH(gated_residual_rows_kernel<true, true>, grid, 256, 0, st, x, h, cond, cond_width, gamma_col,
                            rows, cols);
  else if (xf) B200_LAUNCH(gated_residual_rows_kernel<true, false>, grid, 256, 0, st, x, h, cond, cond_width, gamma_col,
                           rows, cols);
  else if (hf) B200_LAUNCH(gated_residual_rows_kernel<false, true>, grid, 256, 0, st, x, h, cond, cond_width, gamma_col,
                           rows, cols);
  else B200_LAUNCH(gated_residual_rows_kernel<false, false>, grid, 256, 0, st, x, h, cond, cond_width, gamma_col, rows,
                   cols);
  return B200_OK;
}

int b200_masked_softmax_rows(const void* logits, const uint8_t* mask, void* out, int H, int n_rows, int n, int pitch,
                             b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(logits && mask && out, "logits/mask/out is NULL");
  B200_CHECK_ARG(H > 0 && n > 0 && n_rows > 0 && pitch >= n && pitch % 8 == 0,
                 "need H, n_rows, n > 0 and a pitch >= n that is a multiple of 8");
  B200_CHECK_ARG(aligned(logits, 16) && aligned(out, 16), "logits/out must be 16-byte aligned");
  B200_LAUNCH(masked_softmax_rows_kernel, grid_for((int64_t)H * n_rows, 8), 256, 0, static_cast<cudaStream_t>(stream),
              static_cast<const __nv_bfloat16*>(logits), mask, static_cast<__nv_bfloat16*>(out), H, n_rows, n, pitch);
  return B200_OK;
}

int b200_pwa_values(const void* w_m, const void* mn, void* vT, int S, int n, int c_m, int H, int pitch, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(w_m && mn && vT, "w_m/mn/vT is NULL");
  B200_CHECK_ARG(S > 0 && n > 0 && H > 0 && c_m > 0 && c_m % 8 == 0, "S, n, H must be positive, c_m=%d a multiple of 8", c_m);
  B200_CHECK_ARG(pitch >= n && pitch % 8 == 0, "pitch=%d must be a multiple of 8 and >= n", pitch);
  B200_CHECK_ARG(aligned(w_m, 16) && aligned(mn, 16) && aligned(vT, 16), "w_m/mn/vT must be 16-byte aligned");
  // v_h^T[s] = W_m[h] . mn[s]^T of every head and MSA row in one launch: one A for all S batch items, 32 rows of C a head.
  // (A launch per head: 8 x 6.3 us for 128 rows of 256 tokens.)
  BmmLaunch a{w_m, mn, vT, S, 32 * H, pitch, c_m, c_m, c_m, pitch, 0, int64_t(n) * c_m, int64_t(32) * pitch};
  a.b_rows = n;
  a.row_groups = H;
  a.group_stride = int64_t(S) * 32 * pitch;
  return launch_bmm(a, static_cast<cudaStream_t>(stream));
}

int b200_pwa_gate(const void* o, const void* g, void* og, int S, int n, int H, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(o && g && og, "o/g/og is NULL");
  B200_CHECK_ARG(S > 0 && n > 0 && H > 0, "S, n, H must be positive");
  B200_CHECK_ARG(aligned(o, 16) && aligned(g, 16) && aligned(og, 16), "o/g/og must be 16-byte aligned");
  B200_LAUNCH(pwa_gate_kernel, grid_for((int64_t)S * n * H * 4, 256), 256, 0, static_cast<cudaStream_t>(stream),
              static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(g), static_cast<__nv_bfloat16*>(og),
              S, n, H);
  return B200_OK;
}

int b200_split_rows(const void* x, void* y, const float* w, const float* b, int64_t rows, int cols, float eps,
                    int normalize, int order, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && y, "x/y is NULL");
  B200_CHECK_ARG(rows >= 0 && cols > 0 && cols % 8 == 0, "cols=%d must be a positive multiple of 8", cols);
  B200_CHECK_ARG(!normalize || cols <= 1024, "LayerNorm rows hold at most 1024 channels");
  B200_CHECK_ARG(order == 0 || order == 1, "order must be 0 (hi|hi|lo) or 1 (hi|lo|hi)");
  B200_CHECK_ARG(aligned(x, 32) && aligned(y, 16), "x must be 32-byte aligned, y 16-byte aligned");
  if (rows == 0) return B200_OK;
  B200_LAUNCH(split_rows_kernel, grid_for(rows, 8), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const
              float*>(x), static_cast<__nv_bfloat16*>(y), w, b, rows, cols, eps, normalize, order);
  return B200_OK;
}

int b200_gate_rows_f32(const float* a, int64_t a_pitch, const float* b, int64_t b_pitch, const uint8_t* rowmask,
                       float* out, int64_t rows, int cols, int mode, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(a && b && out, "a/b/out is NULL");
  B200_CHECK_ARG(rows >= 0 && cols > 0 && cols % 4 == 0 && a_pitch % 4 == 0 && b_pitch % 4 == 0,
                 "cols and the pitches must be multiples of 4");
  B200_CHECK_ARG(mode >= 0 && mode <= 2, "mode must be 0 (a * sigmoid(b)), 1 (silu(a) * b) or 2 (a)");
  B200_CHECK_ARG(aligned(a, 16) && aligned(b, 16) && aligned(out, 16), "a/b/out must be 16-byte aligned");
  if (rows == 0) return B200_OK;
  B200_LAUNCH(gate_rows_f32_kernel, grid_for(rows * (cols / 4), 256), 256, 0, static_cast<cudaStream_t>(stream), a,
              a_pitch, b, b_pitch, rowmask, out, rows, cols, mode);
  return B200_OK;
}

int b200_softmax_bias_f32(float* s, const float* bias, const uint8_t* keymask, int64_t groups, int n, int H, int bias_div,
                          b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(s && keymask, "s/keymask is NULL");
  B200_CHECK_ARG(groups > 0 && n > 0 && H > 0 && bias_div > 0 && groups % ((int64_t)H * bias_div) == 0,
                 "groups must be a multiple of H * bias_div");
  B200_LAUNCH(softmax_bias_f32_kernel, grid_for(groups * n, 8), 256, 0, static_cast<cudaStream_t>(stream), s, bias,
              keymask, groups, n, H, bias_div, H * bias_div);
  return B200_OK;
}

int b200_pack_bf16(const b200_pack_segment* segments, int n, void* dst, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(segments && dst && n > 0 && n <= B200_PACK_MAX, "need 1..%d segments", B200_PACK_MAX);
  B200_CHECK_ARG(aligned(dst, 16), "dst must be 16-byte aligned");
  PackParams p;
  p.dst = static_cast<__nv_bfloat16*>(dst);
  int64_t most = 0;
  for (int i = 0; i < n; ++i) {
    const b200_pack_segment& s = segments[i];
    B200_CHECK_ARG(s.groups >= 0 && s.group >= 0 && s.pitch > 0 && s.group <= s.pitch && s.group % 8 == 0 && s.pitch % 8 == 0 &&
                       s.stride >= s.pitch && s.stride % 8 == 0 &&
                       s.dst_off >= 0 && s.dst_off % 8 == 0 && int64_t(s.groups) * s.pitch < (int64_t(1) << 31),
                   "segment %d: sizes and offsets must be multiples of 8", i);
    B200_CHECK_ARG(aligned(s.src, 32), "segment %d: the source must be 32-byte aligned", i);
    p.seg[i] = s;
    if (int64_t(s.groups) * s.pitch > most) most = int64_t(s.groups) * s.pitch;
  }
  if (most == 0) return B200_OK;
  B200_LAUNCH(pack_bf16_kernel, dim3(unsigned(grid_for(most / 8, 256)), unsigned(n)), 256, 0, static_cast<cudaStream_t>(stream), p);
  g_launch_count.fetch_sub(1, std::memory_order_relaxed);  // preparation, not one of the kernels a forward counts
  return B200_OK;
}

// ------------------------------------------------------------------------------------------------ trunk stack
static size_t round_up_1k(size_t x) { return (x + 1023) / 1024 * 1024; }
static size_t swiglu_workspace(int64_t rows, int cols, int64_t hidden) {
  const size_t h12 = hidden % 64 ? round_up_1k(size_t(rows) * 2 * hidden * 2) : 0;
  return round_up_1k(size_t(rows) * cols * 2) + h12 + round_up_1k(size_t(rows) * hidden * 2);
}
static bool has_triatt(const b200_trunk_block& w) { return w.tri_att_start.w_o != nullptr; }
static bool has_single(const b200_trunk_block& w) { return w.attention.w_o != nullptr; }
static size_t trunk_bias_bytes(int B, int N, int heads) {
  return round_up_1k(size_t(B) * heads * N * ((N + 7) / 8 * 8) * 2);
}
static size_t trunk_scratch_bytes(const b200_trunk_block* blocks, int N) {
  const size_t tm = b200_trimul_workspace_bytes(N), ta = has_triatt(blocks[0]) ? b200_triatt_workspace_bytes(N) : 0;
  return round_up_1k(tm > ta ? tm : ta);
}

size_t b200_trunk_workspace_bytes(const b200_trunk_block* blocks, int B, int N, int heads) {
  if (!blocks || B <= 0 || N <= 0) return 0;
  return trunk_scratch_bytes(blocks, N) + (has_single(blocks[0]) ? 2 * trunk_bias_bytes(B, N, heads) : 0) +
         round_up_1k(size_t(B) * N * N);
}

size_t b200_trunk_side_workspace_bytes(const b200_trunk_block* blocks, int n_blocks, int B, int N, int c_s, int heads) {
  if (!blocks || n_blocks <= 0 || B <= 0 || N <= 0 || !has_single(blocks[0])) return 0;
  size_t need = b200_apb_workspace_bytes(B, 1, N, c_s, heads);
  const size_t rows = size_t(B) * N;
  for (int i = 0; i < n_blocks; ++i) {
    const size_t n = swiglu_workspace(int64_t(rows), c_s, blocks[i].transition_s.hidden);
    if (n > need) need = n;
  }
  return need;
}

// The events that order the two streams of a trunk call: two "bias ready", two "bias read", one for the joins, and one for z
// read by a pair bias on the side stream.  Kept per host thread and device -- an event may be recorded again as soon as the
// waits on it have been enqueued.
struct TrunkEvents {
  cudaEvent_t ev[6] = {};
  int dev = -1;
  void drop() {
    for (cudaEvent_t& e : ev) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
  }
  ~TrunkEvents() { drop(); }
};

static int trunk_events(cudaEvent_t** out) {
  static thread_local TrunkEvents pool;
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  if (pool.dev != dev) {
    pool.drop();
    for (cudaEvent_t& e : pool.ev) B200_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    pool.dev = dev;
  }
  *out = pool.ev;
  return 0;
}

// Makes `stream` wait for what has been enqueued on `side`, at the latest when the scope ends: a call that fails on its way
// must not leave kernels on the side stream that still read the workspace its next call will write, nor a fork open in a
// stream that is being captured.
struct SideJoin {
  cudaStream_t side, stream;
  cudaEvent_t ev;  // null: nothing to join
  int join() {
    if (!ev) return B200_OK;
    const cudaEvent_t e = ev;
    ev = nullptr;
    B200_CUDA(cudaEventRecord(e, side));
    B200_CUDA(cudaStreamWaitEvent(stream, e, 0));
    return B200_OK;
  }
  ~SideJoin() {  // a failed call: its own error stays the one that is reported
    if (ev && cudaEventRecord(ev, side) == cudaSuccess) (void)cudaStreamWaitEvent(stream, ev, 0);
  }
};

// SwiGLU transition of any width: [LayerNorm,] fc1 | fc2 product with the SwiGLU in its epilogue (hidden a multiple of 64;
// otherwise a row kernel of its own), fc3 product.  x fp32 or bf16 [rows][cols], out [rows][out_cols]; residual: added into
// out (== x's values); mul: gate of the fc3 product, as in BmmLaunch.
static int swiglu_transition(const void* x, bool x_f32, void* out, bool out_f32, bool residual, const float* mul, int mul_pitch,
                             const b200_swiglu_weights& w, int64_t rows, int cols, int out_cols, uint8_t* ws, cudaStream_t stream) {
  const int hidden = int(w.hidden);
  const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
  if (x_f32 || w.ln_w) {
    __nv_bfloat16* xr = reinterpret_cast<__nv_bfloat16*>(ws);
    if (int e = launch_rows_to_bf16(x, x_f32, xr, w.ln_w, w.ln_b, rows, cols, w.ln_w != nullptr, stream)) return e;
    xb = xr;
  }
  ws += round_up_1k(size_t(rows) * cols * 2);
  __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(ws);
  if (hidden % 64 == 0) {
    BmmLaunch a{xb, w.w12, h, 1, int(rows), 2 * hidden, cols, cols, cols, hidden, 0, 0, 0};
    a.swiglu = true;
    if (int e = launch_bmm(a, stream)) return e;
  } else {
    __nv_bfloat16* h12 = reinterpret_cast<__nv_bfloat16*>(ws + round_up_1k(size_t(rows) * hidden * 2));
    BmmLaunch a{xb, w.w12, h12, 1, int(rows), 2 * hidden, cols, cols, cols, 2 * hidden, 0, 0, 0};
    if (int e = launch_bmm(a, stream)) return e;
    B200_LAUNCH(swiglu_rows_kernel, grid_for(rows * (hidden / 8), 256), 256, 0, stream, h12, h, rows, hidden);
  }
  BmmLaunch b{h, w.w3, out, 1, int(rows), out_cols, hidden, hidden, hidden, out_cols, 0, 0, 0};
  b.out_f32 = out_f32;
  b.residual = residual ? out : nullptr;
  b.mul = mul;
  b.mul_pitch = mul_pitch;
  return launch_bmm(b, stream);
}

// Accurate triangle multiplication: hs (hi | lo rows), the operands a and b (hi and lo planes; later ts), and in fp32 t, the
// projected t and the gate logits.
static size_t accurate_rows_bytes(int N) { return round_up_1k(size_t(N) * ((N + 7) / 8 * 8) * 256 * 2); }

size_t b200_accurate_trimul_workspace_bytes(int N) {
  if (N <= 0) return 0;
  return 6 * accurate_rows_bytes(N);
}

int b200_accurate_trimul_fwd(const float* z, const uint8_t* mask, float* out, const void* w_in, const void* w_p_out,
                             const void* w_g_out, const float* ln_in_w, const float* ln_in_b, const float* ln_out_w,
                             const float* ln_out_b, int N, int incoming, int add_residual, void* workspace,
                             size_t workspace_bytes, b200_stream_t stream_) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(z && mask && out && w_in && w_p_out && w_g_out && ln_in_w && ln_in_b && ln_out_w && ln_out_b,
                 "an argument is NULL");
  B200_CHECK_ARG(N > 0 && N <= 32768, "N=%d out of range", N);
  B200_CHECK_ARG(aligned(z, 32) && aligned(out, 16) && aligned(w_in, 16) && aligned(w_p_out, 16) && aligned(w_g_out, 16),
                 "z must be 32-byte aligned, out and the weights 16-byte aligned");
  B200_CHECK_ARG(workspace && aligned(workspace, 1024) && workspace_bytes >= b200_accurate_trimul_workspace_bytes(N),
                 "workspace missing, misaligned or too small");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int pitch = (N + 7) / 8 * 8;
  const int64_t rows = int64_t(N) * pitch, pairs = int64_t(N) * N;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __nv_bfloat16* hs = reinterpret_cast<__nv_bfloat16*>(ws);
  const size_t part = accurate_rows_bytes(N);
  __nv_bfloat16* a = reinterpret_cast<__nv_bfloat16*>(ws + part);
  __nv_bfloat16* b = a + part / 2;
  __nv_bfloat16* ts = a;  // after the contraction has read a
  float* t = reinterpret_cast<float*>(ws + 3 * part);
  float* po = reinterpret_cast<float*>(ws + 4 * part);
  float* go = reinterpret_cast<float*>(ws + 5 * part);
  // incoming walks the pairs column by column: (line, pos) is pair (pos, line)
  const long long ls = incoming ? 1 : N, ps = incoming ? N : 1;
  B200_LAUNCH(ln_split128_kernel, grid_for(rows, 32), 256, 0, stream, z, hs, ln_in_w, ln_in_b, (long long)rows, N, pitch, ls,
              ps, 1);
  {
    BmmLaunch m{hs, w_in, a, 1, int(rows), 512, 384, 256, 384, rows, 0, 0, int64_t(part / 2)};
    m.a_fold = 2;
    m.gate_mask = mask;
    m.mask_pitch = pitch;
    m.mask_n = N;
    m.mask_line = ls;
    m.mask_pos = ps;
    if (int e = launch_bmm(m, stream)) return e;
  }
  {
    BmmLaunch m{a, b, t, 128, N, N, pitch, pitch, pitch, pitch, int64_t(N) * pitch, int64_t(N) * pitch, int64_t(N) * pitch};
    m.out_f32 = 1;
    m.parts = true;
    if (int e = launch_bmm(m, stream)) return e;
  }
  B200_LAUNCH(ln_split_channels_kernel, dim3((N + 31) / 32, N), 256, 0, stream, t, ts, ln_out_w, ln_out_b, N, N, pitch);
  {
    BmmLaunch m{ts, w_p_out, po, 1, int(pairs), 128, 384, 256, 384, 128, 0, 0, 0};
    m.out_f32 = 1;
    m.a_fold = 2;
    if (int e = launch_bmm(m, stream)) return e;
    m.A = hs, m.B = w_g_out, m.C = go, m.M = int(rows);
    if (int e = launch_bmm(m, stream)) return e;
  }
  B200_LAUNCH(gate_pairs_kernel, grid_for(pairs * 32, 256), 256, 0, stream, po, go, add_residual ? z : nullptr, out, N, pitch,
              incoming);
  return B200_OK;
}

size_t b200_accurate_transition_workspace_bytes(int64_t rows, int cols, int hidden) {
  if (rows <= 0 || cols <= 0 || hidden <= 0) return 0;
  return round_up_1k(size_t(rows) * cols * 4) + size_t(rows) * hidden * 4;
}

int b200_accurate_transition_fwd(const float* x, float* out, const void* w12, const void* w3, const float* ln_w,
                                 const float* ln_b, int64_t rows, int cols, int hidden, int out_cols, int normalize,
                                 int add_residual, void* workspace, size_t workspace_bytes, b200_stream_t stream_) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && out && w12 && w3, "x/out/w12/w3 is NULL");
  B200_CHECK_ARG(rows >= 0 && rows < (int64_t(1) << 31), "rows out of range");
  B200_CHECK_ARG(cols > 0 && cols <= 1024 && cols % 64 == 0 && hidden > 0 && hidden % 64 == 0 && out_cols > 0 && out_cols % 8 == 0,
                 "cols=%d and hidden=%d must be multiples of 64 (cols <= 1024), out_cols=%d of 8", cols, hidden, out_cols);
  B200_CHECK_ARG(!add_residual || out_cols == cols, "a residual needs out_cols == cols");
  B200_CHECK_ARG(aligned(x, 32) && aligned(out, 16) && aligned(w12, 16) && aligned(w3, 16),
                 "x must be 32-byte aligned, out and the weights 16-byte aligned");
  if (rows == 0) return B200_OK;
  B200_CHECK_ARG(workspace && aligned(workspace, 1024) &&
                     workspace_bytes >= b200_accurate_transition_workspace_bytes(rows, cols, hidden),
                 "workspace missing, misaligned or too small");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  __nv_bfloat16* xs = static_cast<__nv_bfloat16*>(workspace);
  __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(static_cast<uint8_t*>(workspace) + round_up_1k(size_t(rows) * cols * 4));
  if (cols == 128) {  // rows that fit a warp's registers, four at a time
    B200_LAUNCH(ln_split128_kernel, grid_for(rows, 32), 256, 0, stream, x, xs, ln_w, ln_b, (long long)rows, int(rows),
                int(rows), 0ll, 1ll, normalize);
  } else {
    B200_LAUNCH(split_rows_kernel, grid_for(rows, 8), 256, 0, stream, x, xs, ln_w, ln_b, rows, cols, 1e-5f, normalize, 2);
  }
  BmmLaunch m{xs, w12, h, 1, int(rows), 2 * hidden, 3 * cols, 2 * cols, 3 * cols, 2 * hidden, 0, 0, 0};
  m.swiglu = m.split = true;
  m.a_fold = cols / 64;
  if (int e = launch_bmm(m, stream)) return e;
  BmmLaunch o{h, w3, out, 1, int(rows), out_cols, 3 * hidden, 2 * hidden, 3 * hidden, out_cols, 0, 0, 0};
  o.out_f32 = 1;
  o.a_fold = hidden / 64;
  o.residual = add_residual ? x : nullptr;
  return launch_bmm(o, stream);
}

size_t b200_swiglu_transition_workspace_bytes(int64_t rows, int cols, int64_t hidden) {
  return rows > 0 && cols > 0 && hidden > 0 ? swiglu_workspace(rows, cols, hidden) : 0;
}

int b200_swiglu_transition_fwd(const void* x, void* out, const b200_swiglu_weights* w, int64_t rows, int cols, int out_cols,
                               int add_residual, int x_dtype, void* workspace, size_t workspace_bytes, b200_stream_t stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(x && out && w && w->w12 && w->w3, "x/out/weights is NULL");
  B200_CHECK_ARG(rows >= 0 && rows < (int64_t(1) << 31), "rows out of range");
  B200_CHECK_ARG(cols > 0 && cols % 8 == 0 && cols <= 1024 && out_cols > 0 && out_cols % 8 == 0 && w->hidden > 0 && w->hidden % 8 == 0,
                 "widths must be multiples of 8 and the input width at most 1024");
  B200_CHECK_ARG((x_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(!add_residual || x == out, "the residual form works in place");
  // bf16 rows without a LayerNorm are the product's operand as they are, others are read 32 bytes at a time
  B200_CHECK_ARG(aligned(x, x_dtype == B200_DTYPE_BF16 && !w->ln_w ? 16 : 32) && aligned(out, 32),
                 "out must be 32-byte aligned, x 32-byte (16 for bf16 without a LayerNorm)");
  if (rows == 0) return B200_OK;
  if (!workspace || workspace_bytes < swiglu_workspace(rows, cols, w->hidden) || !aligned(workspace, 1024))
    return fail(B200_ERR_WORKSPACE, "workspace must be 1024-byte aligned and hold %zu bytes (got %zu)",
                swiglu_workspace(rows, cols, w->hidden), workspace_bytes);
  const bool f32 = x_dtype == B200_DTYPE_F32;
  return swiglu_transition(x, f32, out, f32, add_residual != 0, nullptr, 0, *w, rows, cols, out_cols,
                           static_cast<uint8_t*>(workspace), static_cast<cudaStream_t>(stream));
}

// ------------------------------------------------------------------------------------------------ conditioned block
struct CondPlan {
  size_t off_cn, off_cond, off_y, off_rest, total;
};
static void cond_plan(const b200_cond_layer* l, int64_t rows, CondPlan* pl) {
  size_t o = 0;
  pl->off_cn = o; o += round_up_1k(size_t(rows) * l->dim_cond * 2);
  pl->off_cond = o; o += round_up_1k(size_t(rows) * 6 * l->dim * 4);
  pl->off_y = o; o += round_up_1k(size_t(rows) * l->dim * 2);
  pl->off_rest = o;
  size_t attn;
  if (l->window_queries) {
    attn = round_up_1k(size_t(rows) * 4 * l->dim * 2) + round_up_1k(size_t(rows) * l->dim * 2) +
           round_up_1k(size_t(l->B) * l->N * l->window_keys * l->heads * 4);
  } else {
    attn = b200_apb_workspace_bytes(l->B, l->M, l->N, l->dim, l->heads);
  }
  const size_t tr = l->transition_fused.w13 ? round_up_1k(size_t(rows) * l->dim * 2) : swiglu_workspace(rows, l->dim, l->transition.hidden);
  pl->total = o + (attn > tr ? attn : tr);
}

size_t b200_cond_layer_workspace_bytes(const b200_cond_layer* l) {
  if (!l || l->B <= 0 || l->M <= 0 || l->N <= 0 || l->dim <= 0) return 0;
  CondPlan pl;
  cond_plan(l, int64_t(l->B) * l->M * l->N, &pl);
  return pl.total;
}

// The two kernels around the attention of a windowed block of 128 channels; maps and launch.
static int cond_rows_map(CUtensorMap* m, const void* base, bool f32, int64_t rows, int cols) {
  const uint64_t dims[2] = {uint64_t(cols), uint64_t(rows)};
  const uint64_t str[1] = {uint64_t(cols) * (f32 ? 4 : 2)};
  const uint32_t box[2] = {f32 ? 32u : 64u, 128};
  return make_tmap(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, 2, dims, str, box,
                   CU_TENSOR_MAP_SWIZZLE_128B);
}

static bool cond_block_fits(const b200_cond_layer* l, int x_dtype) {
  const int64_t hidden = l->transition_fused.hidden;
  return l->window_queries && l->dim == 128 && l->dim_cond == 128 && x_dtype == B200_DTYPE_F32 && l->transition_fused.w13 &&
         l->transition_fused.w3 && (hidden == 256 || hidden == 512);
}

static CondBlockParams cond_block_params(const b200_cond_layer* l, const void* c, int64_t rows) {
  return CondBlockParams{c, l->ln_c_w, l->ln_c_b, l->b_cond, l->b_qkvg, rows, int((rows + 127) / 128),
                         int(l->transition_fused.hidden / 64), l->lns_scale, 1e-5f};
}

static int launch_cond_in(const b200_cond_layer* l, const void* x, const void* c, int c_dtype, void* qkvg, int64_t rows,
                          cudaStream_t stream) {
  CondInMaps m;
  memset(&m, 0, sizeof(m));
  if (int e = cond_rows_map(&m.w_cond, l->w_cond, false, 768, 128)) return e;
  if (int e = cond_rows_map(&m.w_qkvg, l->w_qkvg, false, 512, 128)) return e;
  if (int e = cond_rows_map(&m.x, x, true, rows, 128)) return e;
  if (int e = cond_rows_map(&m.qkvg, qkvg, false, rows, 512)) return e;
  const CondBlockParams p = cond_block_params(l, c, rows);
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  if (c_dtype == B200_DTYPE_F32) B200_LAUNCH(cond_in_kernel<true>, grid, cond_block::THREADS, cond_block::InLayout::SMEM_BYTES, stream, m, p);
  else B200_LAUNCH(cond_in_kernel<false>, grid, cond_block::THREADS, cond_block::InLayout::SMEM_BYTES, stream, m, p);
  return B200_OK;
}

static int launch_cond_out(const b200_cond_layer* l, const void* x, const void* c, int c_dtype, const void* og, void* out, int64_t rows,
                           cudaStream_t stream) {
  CondOutMaps m;
  memset(&m, 0, sizeof(m));
  const int hidden = int(l->transition_fused.hidden);
  if (int e = cond_rows_map(&m.w_cond, l->w_cond, false, 768, 128)) return e;
  if (int e = cond_rows_map(&m.w_o, l->w_o, false, 128, 128)) return e;
  if (int e = cond_rows_map(&m.w13, l->transition_fused.w13, false, 2 * hidden, 128)) return e;
  if (int e = cond_rows_map(&m.w3, l->transition_fused.w3, false, 128, hidden)) return e;
  if (int e = cond_rows_map(&m.og, og, false, rows, 128)) return e;
  if (int e = cond_rows_map(&m.x, x, true, rows, 128)) return e;
  if (int e = cond_rows_map(&m.out, out, true, rows, 128)) return e;
  const CondBlockParams p = cond_block_params(l, c, rows);
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  if (c_dtype == B200_DTYPE_F32) B200_LAUNCH(cond_out_kernel<true>, grid, cond_block::THREADS, cond_block::OutLayout::SMEM_BYTES, stream, m, p);
  else B200_LAUNCH(cond_out_kernel<false>, grid, cond_block::THREADS, cond_block::OutLayout::SMEM_BYTES, stream, m, p);
  return B200_OK;
}

int b200_cond_layer_fwd(const b200_cond_layer* l, const void* x, const void* pairs, const void* bias, int64_t bias_pitch,
                        const void* c, const uint8_t* mask, void* out, int x_dtype, int c_dtype, int pairs_dtype,
                        void* workspace, size_t workspace_bytes, b200_stream_t stream_) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(l && x && c && mask && out && (pairs || bias), "an argument is NULL");
  B200_CHECK_ARG(l->B > 0 && l->M > 0 && l->N > 0 && l->heads > 0, "B/M/N/heads must be positive");
  B200_CHECK_ARG(l->dim > 0 && l->dim % 32 == 0 && l->dim <= 1024 && l->dim_cond > 0 && l->dim_cond % 8 == 0 && l->dim_cond <= 1024,
                 "dim=%d must be a multiple of 32, dim_cond=%d of 8, both <= 1024", l->dim, l->dim_cond);
  B200_CHECK_ARG((x_dtype | 1) == 1 && (c_dtype | 1) == 1 && (pairs_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(x, 32) && aligned(c, 32) && aligned(out, 32), "x/c/out must be 32-byte aligned");
  B200_CHECK_ARG(l->w_cond && l->b_cond && (l->transition_fused.w13 || l->transition.w12), "a weight pointer is NULL");
  const int64_t rows = int64_t(l->B) * l->M * l->N;
  B200_CHECK_ARG(rows < (int64_t(1) << 31), "too many rows");
  CondPlan pl;
  cond_plan(l, rows, &pl);
  if (!workspace || workspace_bytes < pl.total || !aligned(workspace, 1024))
    return fail(B200_ERR_WORKSPACE, "workspace must be 1024-byte aligned and hold %zu bytes (got %zu)", pl.total, workspace_bytes);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __nv_bfloat16* cn = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_cn);
  float* cond = reinterpret_cast<float*>(ws + pl.off_cond);
  __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(ws + pl.off_y);
  uint8_t* rest = ws + pl.off_rest;
  const int D = l->dim, CW = 6 * D;
  const bool xf32 = x_dtype == B200_DTYPE_F32;
  if (cond_block_fits(l, x_dtype)) {
    const int W = l->window_queries, Hk = l->window_keys, NW = l->N / W;
    B200_CHECK_ARG(l->N % W == 0, "N=%d is not a multiple of the query window %d", l->N, W);
    B200_CHECK_ARG(pairs && l->w_qkvg && l->b_qkvg && l->w_o && l->ln_z_w && l->w_z, "a window weight pointer is NULL");
    B200_CHECK_ARG(D % l->heads == 0, "dim=%d is not a multiple of heads=%d", D, l->heads);
    __nv_bfloat16* qkvg = reinterpret_cast<__nv_bfloat16*>(rest);
    __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(rest + round_up_1k(size_t(rows) * 4 * D * 2));
    float* wb = reinterpret_cast<float*>(rest + round_up_1k(size_t(rows) * 4 * D * 2) + round_up_1k(size_t(rows) * D * 2));
    if (int e = launch_cond_in(l, x, c, c_dtype, qkvg, rows, stream)) return e;
    if (int e = window_pair_run(qkvg, 4 * D, qkvg + 3 * D, 4 * D, pairs, l->ln_z_w, l->ln_z_b, l->w_z, mask, og, wb, l->B, l->M, NW, W, Hk,
                                l->heads, D / l->heads, l->dim_pairwise, pairs_dtype, stream))
      return e;
    return launch_cond_out(l, x, c, c_dtype, og, out, rows, stream);
  }
  // alpha1 | beta1 | gamma1 | alpha2 | beta2 | gamma2 = Linear(silu(LayerNorm(c)))
  if (int e = launch_rows_to_bf16(c, c_dtype == B200_DTYPE_F32, cn, l->ln_c_w, l->ln_c_b, rows, l->dim_cond, true, stream, true)) return e;
  {
    BmmLaunch a{cn, l->w_cond, cond, 1, int(rows), CW, l->dim_cond, l->dim_cond, l->dim_cond, CW, 0, 0, 0};
    a.bias = l->b_cond;
    a.out_f32 = 1;
    if (int e = launch_bmm(a, stream)) return e;
  }
  auto adaln = [&](const void* in, int alpha, void* copy) -> int {
    return launch_adaln(in, xf32, cond, CW, alpha * D, (alpha + 1) * D, l->lns_scale, y, copy, rows, D, stream);
  };
  auto gated_residual = [&](const __nv_bfloat16* h, int gamma) -> int {
    const int grid = grid_for(rows * (D / 8), 256);
    if (xf32) B200_LAUNCH((gated_residual_rows_kernel<true, false>), grid, 256, 0, stream, out, h, cond, CW, gamma * D, rows, D);
    else B200_LAUNCH((gated_residual_rows_kernel<false, false>), grid, 256, 0, stream, out, h, cond, CW, gamma * D, rows, D);
    return 0;
  };
  // out = x + gamma1 * attention(adaln(x)); x is copied on the way, the output projection adds into the copy
  if (int e = adaln(x, 0, x == out ? nullptr : out)) return e;
  if (l->window_queries) {
    const int W = l->window_queries, Hk = l->window_keys, NW = l->N / W;
    B200_CHECK_ARG(l->N % W == 0, "N=%d is not a multiple of the query window %d", l->N, W);
    B200_CHECK_ARG(pairs && l->w_qkvg && l->b_qkvg && l->w_o && l->ln_z_w && l->w_z, "a window weight pointer is NULL");
    B200_CHECK_ARG(D % l->heads == 0, "dim=%d is not a multiple of heads=%d", D, l->heads);
    __nv_bfloat16* qkvg = reinterpret_cast<__nv_bfloat16*>(rest);
    __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(rest + round_up_1k(size_t(rows) * 4 * D * 2));
    float* wb = reinterpret_cast<float*>(rest + round_up_1k(size_t(rows) * 4 * D * 2) + round_up_1k(size_t(rows) * D * 2));
    {
      BmmLaunch a{y, l->w_qkvg, qkvg, 1, int(rows), 4 * D, D, D, D, 4 * D, 0, 0, 0};
      a.bias = l->b_qkvg;
      if (int e = launch_bmm(a, stream)) return e;
    }
    if (int e = window_pair_run(qkvg, 4 * D, qkvg + 3 * D, 4 * D, pairs, l->ln_z_w, l->ln_z_b, l->w_z, mask, og, wb, l->B, l->M, NW, W, Hk,
                                l->heads, D / l->heads, l->dim_pairwise, pairs_dtype, stream))
      return e;
    BmmLaunch a{og, l->w_o, out, 1, int(rows), D, D, D, D, D, 0, 0, 0};
    a.residual = out;
    a.out_f32 = xf32;
    a.mul = cond + 2 * D;
    a.mul_pitch = CW;
    if (int e = launch_bmm(a, stream)) return e;
  } else {
    const ApbOutput into{out, xf32, cond + 2 * D, CW};
    if (int e = apb_run(y, pairs, bias, bias_pitch, mask, out, &l->attention, l->B, l->M, l->N, D, l->heads, B200_DTYPE_BF16, pairs_dtype,
                        false, rest, workspace_bytes - pl.off_rest, stream, &into))
      return e;
  }
  // out += gamma2 * transition(adaln(out))
  if (int e = adaln(out, 3, nullptr)) return e;
  if (l->transition_fused.w13) {
    __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(rest);
    const b200_transition_weights& tw = l->transition_fused;
    if (int e = b200_transition_hidden_fwd(y, h, tw.w13, tw.w3, nullptr, nullptr, rows, int(tw.hidden), 0, 0, B200_DTYPE_BF16, stream)) return e;
    return gated_residual(h, 5);
  }
  return swiglu_transition(y, false, out, xf32, true, cond + 5 * D, CW, l->transition, rows, D, D, rest, stream);
}

int b200_trunk_fwd(const b200_trunk_block* blocks, int n_blocks, const void* z_in, void* z, void* s,
                   const uint8_t* token_mask, const uint8_t* pair_mask, int B, int N, int c_s, int heads, int s_dtype,
                   int z_dtype, void* workspace, size_t workspace_bytes, void* side_workspace, size_t side_bytes,
                   b200_stream_t stream_, b200_stream_t side_stream) {
  if (int e = b200_check_device()) return e;
  B200_CHECK_ARG(blocks && n_blocks > 0, "need at least one block");
  B200_CHECK_ARG(z_in && z && (token_mask || pair_mask), "z_in/z/mask is NULL");
  B200_CHECK_ARG(B > 0 && N > 0, "B=%d, N=%d must be positive", B, N);
  B200_CHECK_ARG((s_dtype | 1) == 1 && (z_dtype | 1) == 1, "unknown dtype");
  B200_CHECK_ARG(aligned(z, 32) && aligned(z_in, 32), "z must be 32-byte aligned");
  const bool single = has_single(blocks[0]);
  if (single) {
    B200_CHECK_ARG(s && token_mask && aligned(s, 32), "the single track needs s (32-byte aligned) and token_mask");
    B200_CHECK_ARG(c_s > 0 && c_s % 8 == 0 && c_s <= 1024 && heads > 0 && heads <= 16,
                   "c_s=%d must be a multiple of 8 and <= 1024, heads=%d <= 16", c_s, heads);
  }
  for (int i = 0; i < n_blocks; ++i) {
    const b200_trunk_block& w = blocks[i];
    B200_CHECK_ARG(trimul_weights_ok(&w.tri_mul_out) && trimul_weights_ok(&w.tri_mul_in), "block %d: bad triangle weights", i);
    B200_CHECK_ARG(has_triatt(w) == has_triatt(blocks[0]) && has_single(w) == single, "block %d: differs from block 0 in kind", i);
    B200_CHECK_ARG(!has_triatt(w) || (triatt_weights_ok(&w.tri_att_start) && triatt_weights_ok(&w.tri_att_end)),
                   "block %d: bad triangle attention weights", i);
    B200_CHECK_ARG(!single || (w.transition_s.w12 && w.transition_s.w3 && w.transition_s.hidden > 0 && w.transition_s.hidden % 8 == 0),
                   "block %d: bad single transition weights", i);
  }
  const size_t need = b200_trunk_workspace_bytes(blocks, B, N, heads);
  const size_t side_need = b200_trunk_side_workspace_bytes(blocks, n_blocks, B, N, c_s, heads);
  if (!workspace || workspace_bytes < need || !aligned(workspace, 1024) ||
      (side_need && (!side_workspace || side_bytes < side_need || !aligned(side_workspace, 1024))))
    return fail(B200_ERR_WORKSPACE, "workspaces must be 1024-byte aligned and hold %zu and %zu bytes (got %zu, %zu)", need,
                side_need, workspace_bytes, side_bytes);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  cudaStream_t side = side_stream ? static_cast<cudaStream_t>(side_stream) : stream;
  const bool two = single && side != stream;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const size_t scratch = trunk_scratch_bytes(blocks, N), bias_bytes = single ? trunk_bias_bytes(B, N, heads) : 0;
  __nv_bfloat16* bias[2] = {reinterpret_cast<__nv_bfloat16*>(ws + scratch),
                            reinterpret_cast<__nv_bfloat16*>(ws + scratch + bias_bytes)};
  cudaEvent_t* ev = nullptr;
  if (two) {
    if (int e = trunk_events(&ev)) return e;
    B200_CUDA(cudaEventRecord(ev[4], stream));  // s, and all that was enqueued before this call
    B200_CUDA(cudaStreamWaitEvent(side, ev[4], 0));
  }
  SideJoin forked{side, stream, two ? ev[4] : nullptr};
  if (!pair_mask) {
    uint8_t* pm = ws + scratch + 2 * bias_bytes;
    B200_LAUNCH(pair_mask_kernel, grid_for(int64_t(B) * N * N, 1024), 256, 0, stream, token_mask, pm, B, N);
    pair_mask = pm;
  }
  const bool zf32 = z_dtype == B200_DTYPE_F32, sf32 = s_dtype == B200_DTYPE_F32;
  const size_t zsz = zf32 ? 4 : 2;
  const int Nk = (N + 7) / 8 * 8;
  // The pair bias of a block reads z, which the next block writes for the first time two kernels on: where it and that block's first
  // projection leave each other SMs, a tile each, it runs on the side stream beside them (4 blocks, us, on the main stream / beside:
  // 24 tokens 450 / 441, 64 469 / 461; with 80 tokens and more the two would take turns).
  const bool beside = two && 2 * N <= sm_count();
  for (int i = 0; i < n_blocks; ++i) {
    const b200_trunk_block& w = blocks[i];
    if (int e = trimul_fwd_impl(i == 0 ? z_in : z, pair_mask, z, &w.tri_mul_out, B, N, 0, 1, z_dtype, ws, scratch, stream,
                                beside && i > 0 ? ev[5] : nullptr))
      return e;
    if (int e = trimul_fwd_impl(z, pair_mask, z, &w.tri_mul_in, B, N, 1, 1, z_dtype, ws, scratch, stream)) return e;
    if (has_triatt(w)) {
      if (int e = b200_triatt_fwd(z, pair_mask, z, &w.tri_att_start, B, N, 0, 1, z_dtype, ws, scratch, stream)) return e;
      if (int e = b200_triatt_fwd(z, pair_mask, z, &w.tri_att_end, B, N, 1, 1, z_dtype, ws, scratch, stream)) return e;
    }
    const b200_transition_weights& tz = w.transition_z;
    if (int e = b200_transition_hidden_fwd(z, z, tz.w13, tz.w3, tz.ln_w, tz.ln_b, int64_t(B) * N * N, int(tz.hidden),
                                           tz.ln_w != nullptr, 1, z_dtype, stream))
      return e;
    if (!single) continue;
    const int k = i & 1;
    if (two && !beside && i >= 2) B200_CUDA(cudaStreamWaitEvent(stream, ev[2 + k], 0));  // block i - 2 has read this bias buffer
    if (beside) {
      B200_CUDA(cudaEventRecord(ev[k], stream));
      B200_CUDA(cudaStreamWaitEvent(side, ev[k], 0));
    }
    for (int b = 0; b < B; ++b)
      if (int e = launch_pair_bias(static_cast<const uint8_t*>(z) + size_t(b) * N * N * kD * zsz, zf32, w.attention.ln_z_w,
                                   w.attention.ln_z_b, w.attention.w_z, bias[k] + size_t(b) * heads * N * Nk, N, N,
                                   (long long)N * kD * zsz, (long long)kD * zsz, (long long)N * Nk, Nk, heads, beside ? side : stream))
        return e;
    if (beside) {
      B200_CUDA(cudaEventRecord(ev[5], side));
    } else if (two) {
      B200_CUDA(cudaEventRecord(ev[k], stream));
      B200_CUDA(cudaStreamWaitEvent(side, ev[k], 0));
    }
    if (int e = apb_run(s, nullptr, bias[k], Nk, token_mask, s, &w.attention, B, 1, N, c_s, heads, s_dtype, B200_DTYPE_F32,
                        true, side_workspace, side_bytes, side))
      return e;
    if (two && !beside) B200_CUDA(cudaEventRecord(ev[2 + k], side));
    if (int e = swiglu_transition(s, sf32, s, sf32, true, nullptr, 0, w.transition_s, int64_t(B) * N, c_s, c_s,
                                  static_cast<uint8_t*>(side_workspace), side))
      return e;
  }
  return forked.join();
}

}  // extern "C"
