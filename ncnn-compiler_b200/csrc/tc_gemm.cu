#include "tc_gemm.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

namespace nb {

bool tc_pdl_enabled() {
  static const bool on = [] {
    const char* f = std::getenv("NCNN_B200_PDL");
    return f == nullptr || f[0] != '0';
  }();
  return on;
}

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
using EncodeIm2colFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                    const cuuint64_t*, const cuuint64_t*, const int*, const int*,
                                    cuuint32_t, cuuint32_t, const cuuint32_t*,
                                    CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn g_encode_tiled = nullptr;
EncodeIm2colFn g_encode_im2col = nullptr;
std::once_flag g_driver_once;
std::string g_driver_error;

void load_driver_entry_points() {
  std::call_once(g_driver_once, [] {
    cudaDriverEntryPointQueryResult query;
    void* fn = nullptr;
    cudaError_t err =
        cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &query);
    if (err != cudaSuccess || query != cudaDriverEntryPointSuccess || fn == nullptr) {
      g_driver_error = "cuTensorMapEncodeTiled is not available from this driver";
      return;
    }
    g_encode_tiled = reinterpret_cast<EncodeTiledFn>(fn);
    fn = nullptr;
    err = cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &query);
    if (err != cudaSuccess || query != cudaDriverEntryPointSuccess || fn == nullptr) {
      g_driver_error = "cuTensorMapEncodeIm2col is not available from this driver";
      return;
    }
    g_encode_im2col = reinterpret_cast<EncodeIm2colFn>(fn);
  });
}

CUtensorMapSwizzle swizzle_for(int row_bytes) {
  return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                          : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                             : CU_TENSOR_MAP_SWIZZLE_32B);
}

CUtensorMapDataType dtype_for(int kind) {
  return kind == GEMM_I8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                         : (kind == GEMM_BF16X3 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32);
}

int elem_bytes(int kind) { return tc_elem_bytes(kind); }

std::string encode_tiled_2d(CUtensorMap* map, int kind, const void* base, uint64_t inner,
                            uint64_t outer, uint64_t outer_stride_bytes, uint32_t box_inner,
                            uint32_t box_outer, int row_bytes) {
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {outer_stride_bytes};
  const cuuint32_t box[2] = {box_inner, box_outer};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r = g_encode_tiled(map, dtype_for(kind), 2, const_cast<void*>(base), dims,
                                    strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                    swizzle_for(row_bytes), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    return "cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)) +
           " (inner " + std::to_string(inner) + ", outer " + std::to_string(outer) + ", stride " +
           std::to_string(outer_stride_bytes) + ")";
  }
  return {};
}

std::string encode_im2col(CUtensorMap* map, int kind, const void* base, const TcIm2colView& v,
                          uint32_t channels_per_pixel, uint32_t pixels, int row_bytes) {
  const cuuint64_t dims[4] = {v.C, v.W, v.H, v.N};
  const cuuint64_t strides[3] = {v.stride_w, v.stride_h, v.stride_n};
  // Bounding box of filter-origin positions: the first is -pad, the last is the
  // origin of the last output pixel; TMA wants it relative to the tensor's far edge.
  const int last_w = -v.pad_l + (v.OW - 1) * v.stride_conv_w;
  const int last_h = -v.pad_t + (v.OH - 1) * v.stride_conv_h;
  const int lower[2] = {-v.pad_l, -v.pad_t};
  const int upper[2] = {last_w - (static_cast<int>(v.W) - 1), last_h - (static_cast<int>(v.H) - 1)};
  const cuuint32_t elem_strides[4] = {1, static_cast<cuuint32_t>(v.stride_conv_w),
                                      static_cast<cuuint32_t>(v.stride_conv_h), 1};
  const CUresult r = g_encode_im2col(
      map, dtype_for(kind), 4, const_cast<void*>(base), dims, strides, lower, upper,
      channels_per_pixel, pixels, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
      swizzle_for(row_bytes), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    return "cuTensorMapEncodeIm2col failed with code " + std::to_string(static_cast<int>(r)) +
           " (C " + std::to_string(v.C) + ", W " + std::to_string(v.W) + ", H " +
           std::to_string(v.H) + ", N " + std::to_string(v.N) + ", strides " +
           std::to_string(v.stride_w) + "/" + std::to_string(v.stride_h) + "/" +
           std::to_string(v.stride_n) + ", corners " + std::to_string(lower[0]) + "," +
           std::to_string(lower[1]) + " / " + std::to_string(upper[0]) + "," +
           std::to_string(upper[1]) + ")";
  }
  return {};
}

// Shared memory that the rings and buffers of a CTA may fill: 227 KB per block, minus 1 KB of alignment slack, minus the
// kernels' static shared memory (barriers and flags, 208 to 272 bytes), and 1 KB of room for that to grow.
constexpr int kTcSmemBudget = 224 * 1024;
constexpr int kDrainBytes = 8 * kDrainWarpBytes;  // shared memory of the eight epilogue warps

int res_mode_of(const TcEpilogue& e) {
  return e.res0 == nullptr ? RES_NONE : (e.res_bf16 ? RES_BF16X2 : (e.res1 != nullptr ? RES_SPLIT : RES_F32));
}

int out_elem_bytes(int out_mode) { return out_mode == OUT_I8 ? 1 : (out_mode == OUT_BF16X2 ? 2 : 4); }

// The formats that kernels of a kind are compiled for; the rest (networks that mix kinds in unusual ways) goes out
// element by element.
bool drains(int kind, int out_mode, int res_mode) {
  if (res_mode == RES_SPLIT && kind != GEMM_TF32X3) return false;
  switch (out_mode) {
    case OUT_F32:
    case OUT_CHW: return true;
    case OUT_I8: return kind == GEMM_I8 && res_mode == RES_NONE;
    case OUT_BF16X2: return kind == GEMM_BF16X3 || kind == GEMM_TF32X3;
    case OUT_F32_SPLIT: return kind == GEMM_TF32X3;
    default: return kind == GEMM_TF32;
  }
}

// True when tc_drain can write these results: rows (of `N` columns, `ldo` apart) made of 16-byte pieces in every format
// that takes part.  *wide: of 32-byte pieces, so that stores and loads are whole sectors.
bool direct_rows(int kind, const TcEpilogue& e, int N, int* wide) {
  bool ok = drains(kind, e.out_mode, res_mode_of(e)), all32 = true;
  auto plane = [&](const void* p, int es) {
    if (p == nullptr) return;
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    ok = ok && at % 16 == 0 && e.ldo * es % 16 == 0 && static_cast<long long>(N) * es % 16 == 0;
    all32 = all32 && at % 32 == 0 && e.ldo * es % 32 == 0;
  };
  if (e.out_mode == OUT_I8) {
    plane(e.outq, 1);
  } else if (e.out_mode != OUT_CHW) {
    plane(e.out0, out_elem_bytes(e.out_mode));
    plane(e.out1, out_elem_bytes(e.out_mode));
  }
  const int rs = e.res_bf16 ? 2 : 4;
  plane(e.res0, rs);
  plane(e.res1, rs);
  for (int i = 0; i < e.side_count; ++i) plane(e.side_q[i], 1);
  *wide = all32 ? 1 : 0;
  return ok;
}

// Tile width: every multiple of 16 up to 128 is a legal UMMA N.  Cost model:
// waves over the SMs times (columns computed + a fixed per-tile term for the
// A traffic and pipeline fill, which do not shrink with the tile).
int choose_block_n(long long tiles_m, int N, int sm_count, int step) {
  int best = step;
  double best_cost = 1e300;
  for (int bn = step; bn <= 128; bn += step) {
    const long long tiles = tiles_m * ((N + bn - 1) / bn);
    const long long waves = (tiles + sm_count - 1) / sm_count;
    const double cost = static_cast<double>(waves) * (bn + 24);
    if (cost < best_cost - 1e-9 || (std::fabs(cost - best_cost) <= 1e-9 && bn > best)) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

// NCNN_B200_PAIR=0 in the environment keeps every tile at 128 rows.
bool pair_enabled() {
  const char* f = std::getenv("NCNN_B200_PAIR");
  return f == nullptr || f[0] != '0';
}

int env_int(const char* name, int fallback);

// NCNN_B200_SPLIT_K=0 in the environment never puts the chunks of a tile on different CTAs: one CTA adds up the same chunks.
bool split_k_enabled() { return env_int("NCNN_B200_SPLIT_K", 1) != 0; }

// The chunks of a contraction's sums, from the layer alone (see kTcChunkFrom); p.k_blocks blocks of p.row_bytes.
void set_chunks(TcGemmParams& p, int kind, int full_row_bytes) {
  p.chunks = 1;
  p.chunk_blocks = p.k_blocks;
  p.split_k = 0;
  const int per_block = full_row_bytes / p.row_bytes;  // a pair plan's half-size blocks
  const int full = p.k_blocks / per_block;
  if (kind != GEMM_BF16X3 || !p.a_im2col || full < kTcChunkFrom) return;
  const int chunks = (full + kTcChunkBlocks - 1) / kTcChunkBlocks;
  const int blocks = (full + chunks - 1) / chunks;
  p.chunks = (full + blocks - 1) / blocks;
  p.chunk_blocks = blocks * per_block;
}

// Chunks side by side: the tile width that does it fastest, or 0 where whole tiles are as fast.  In units of one K block
// at 16 columns (0.40 us; 128 columns take 1.3 of them, measured): a unit's chunk and its share of the latency of
// publishing and adding sums, and those sums' way through L2, against the whole tiles' K blocks.
int split_width(const TcGemmParams& p, const TcEpilogue& e, int N, int block_n, int sm_count) {
  if (p.chunks < 2 || e.sk_ws == nullptr || e.sk_flags == nullptr || !split_k_enabled()) return 0;
  auto tiles_of = [&](int bn) { return static_cast<long long>(p.tiles_m) * ((N + bn - 1) / bn); };
  auto waves = [&](long long units) { return static_cast<double>((units + sm_count - 1) / sm_count); };
  double best = 0.9 * waves(tiles_of(block_n)) * p.k_blocks * (1.0 + block_n / 400.0);
  int width = 0;
  for (int bn = 16; bn <= 128; bn += 16) {
    const long long tiles = tiles_of(bn), units = tiles * p.chunks;
    if (tiles * 8 > e.sk_flag_count || static_cast<size_t>(units) * kTcBlockM * bn * 4 > e.sk_ws_bytes) continue;
    const double cost = waves(units) * (p.chunk_blocks + 3) * (1.0 + bn / 400.0) + 5.0 + static_cast<double>(units) * bn / 1600.0;
    if (cost < best) {
      best = cost;
      width = bn;
    }
  }
  return width;
}

// InnerProduct and Gemm of too few rows to fill the SMs: the tile width and the chunks of K that are expected to take the
// least time, the chunks of a tile on different CTAs.  Clocks as in gemm_clocks (a block's copies, or its MMAs and the gap
// between blocks), and for the chunks' sums their way through L2.
// fp32 sums round by where K is cut, so a layer has one way to cut it: the chunks that are best for a full tile of 128 rows
// (with fewer rows others would be up to 4 % better by these clocks).  Calls of up to three tiles of rows that come here are all
// cut so, or (where chunks gain nothing) all whole; the rows choose the tile width, which no bit depends on, and whether a tile's chunks
// lie apart or follow one another in one CTA, which costs 0 to 5 % over whole tiles and rounds like chunks apart (4096 -> 1000,
// 300 rows: 4.4e-6 of the result's norm off in chunks, 1.4e-5 whole).  Contractions of up to 26 blocks of bf16 pairs (1664 values)
// are never cut: a network's last layer then gives a batch of any size the bits of its images run one by one (1536 -> 1000,
// 33 rows: 16.5 us whole, 12.7 in chunks; chunks for every batch would cost calls of thousands of rows 8 to 20 %).  Whole
// numbers are exact however they are cut.
// Whole calls in us, before (workers that share tiles, tc_gemm2.cuh, or whole tiles) -> in chunks:
//            2048 -> 1024          3000 -> 700           2816 -> 2816           4096 -> 4096
//   fp32     64 rows 24.7 -> 16.4  64 rows 34.6 -> 14.4  64 rows 30.8 -> 20.5   64 rows 32.8 -> 28.7
//            128     34.2 -> 14.4  128     48.4 -> 16.5  128     39.7 -> 22.7   128     39.4 -> 33.9
//            1000    26.7 -> 30.8  1000    36.8 -> 34.9  1000    49.3 -> 54.2   1000    87.4 -> 84.3
//   int8     128     11.0 -> 12.8  300     12.9 -> 18.5  64      12.3 -> 14.5   64      23.4 -> 19.1, 128 30.7 -> 18.5
// and of more than one tile of rows, chunks in one CTA against chunks apart (their number behind the layer; ! is not taken):
//            2048 -> 1024 (4)      3000 -> 700 (6)       2816 -> 2816 (4)       4096 -> 1000 (8)       2048 -> 2048 (4)
//   fp32     200 rows 22.7 / 18.7  200 rows 30.1 / 22.5  200 rows 28.8 / 28.9!  200 rows 37.9 / 32.8   200 rows 22.7 / 26.8!
//            384      22.8 / 23.8! 384      30.9 / 28.8! 384      30.9 / 45.9!  384      39.2 / 48.6!  384      24.7 / 35.6!
// so they lie apart where the clocks below say so (of three tiles, 4096 -> 512 37.1 / 31.2); int8, whose blocks are short, is
// cut from 28 blocks on and up to two tiles.
struct RowsSplit {
  int block_n = 0, chunk_blocks = 0, chunks = 1;
  bool apart = false;  // the chunks of a tile on different CTAs
  double clocks = 1e300;
};
// The best of whole tiles and tiles in `only` chunks apart (0: in any number of them).
RowsSplit best_rows_split(int kind, long long M, int k_blocks, const TcEpilogue& e, int N, int sm_count, int only) {
  RowsSplit best;
  const bool i8 = kind == GEMM_I8;
  const long long tiles_m = (M + kTcBlockM - 1) / kTcBlockM;
  for (int bn = 16; bn <= 128 && bn < N + 16; bn += 16) {
    const long long tiles = tiles_m * ((N + bn - 1) / bn);
    const double mmas = i8 ? 4.0 : 12.0;
    const double block = std::max(tc_planes(kind) * 3.0 * (kTcBlockM + bn), mmas * std::max(39.0, (kTcBlockM + bn) / 4.0) + 330.0);
    for (int chunks = 1; chunks <= std::min(32, k_blocks / 2); ++chunks) {
      if (only != 0 && chunks != 1 && chunks != only) continue;
      const int blocks = (k_blocks + chunks - 1) / chunks;
      if ((k_blocks + blocks - 1) / blocks != chunks) continue;
      const long long units = tiles * chunks;
      if (chunks > 1 && (tiles * 8 > e.sk_flag_count || static_cast<size_t>(units) * kTcBlockM * bn * 4 > e.sk_ws_bytes)) continue;
      // (a warp adds four chunks of 16 columns in ~700 clocks.  Two and three tiles of rows, fp32: fitted to 65 of the calls
      // above; the sums of that many tiles get in one another's way)
      const double sums = i8 || tiles_m == 1
                              ? 2500.0 + 700.0 * ((chunks + 3) / 4) * ((bn + 31) / 32) + static_cast<double>(tiles) * std::min<long long>(M, kTcBlockM) * chunks * bn / 500.0
                              : 44.0 * chunks * bn + static_cast<double>(M) * N * chunks / 130.0 - 5300.0;
      const double clocks = static_cast<double>((units + sm_count - 1) / sm_count) * blocks * block + 3000.0 + 12.0 * bn + (chunks > 1 ? sums : 0.0);
      if (clocks >= best.clocks) continue;
      best.clocks = clocks;
      best.block_n = bn;
      best.chunk_blocks = blocks;
      best.chunks = chunks;
    }
  }
  return best;
}
RowsSplit split_rows(int kind, long long M, int k_blocks, const TcEpilogue& e, int N, int sm_count) {
  if ((kind != GEMM_BF16X3 && kind != GEMM_I8) || e.sk_ws == nullptr || e.sk_flags == nullptr) return {};
  const bool i8 = kind == GEMM_I8;
  if (k_blocks < (i8 ? 28 : 27) || M > (i8 ? 2 : 3) * kTcBlockM) return {};
  if (i8) {
    RowsSplit rows = split_k_enabled() ? best_rows_split(kind, M, k_blocks, e, N, sm_count, 0) : RowsSplit{};
    rows.apart = rows.chunks > 1;
    return rows;
  }
  RowsSplit layer = best_rows_split(kind, kTcBlockM, k_blocks, e, N, sm_count, 0);
  layer.apart = layer.chunks > 1;
  if (layer.chunks == 1) return best_rows_split(kind, M, k_blocks, e, N, sm_count, 1);
  RowsSplit rows = best_rows_split(kind, M, k_blocks, e, N, sm_count, layer.chunks);
  rows.apart = rows.chunks > 1;
  if (M <= kTcBlockM) {
    if (!rows.apart) rows = layer;
    rows.clocks = layer.clocks;  // (what other forms are compared with: the same for all calls of one tile)
    return rows;
  }
  // (up to a tenth of the clocks' gain did not come: 2048 -> 1024, 300 rows 25.2 in chunks, 22.7 whole)
  const RowsSplit whole = best_rows_split(kind, M, k_blocks, e, N, sm_count, 1);
  if (M > 2 * kTcBlockM && rows.clocks > 0.8 * whole.clocks) rows = whole;
  if (rows.chunks == 1) {
    rows.chunks = layer.chunks;
    rows.chunk_blocks = layer.chunk_blocks;
    rows.apart = false;
  }
  return rows;
}

void finish_plan(TcLaunch* L, int kind, long long M, int N, const TcEpilogue& e, int sm_count) {
  TcGemmParams& p = L->p;
  p.M = static_cast<int>(M);
  p.N = N;
  p.tiles_m = static_cast<int>((M + kTcBlockM - 1) / kTcBlockM);
  // A lone tile brings the rows it has, in whole swizzle atoms of eight: rows past them are not filled with zeros by TMA, which
  // takes as long as bringing data, and hold whatever the ring held (a row of A reaches its own row of results only).
  // Whole calls, 128 rows -> those there are: int8 1001 -> 1537, 1 to 65 rows 12.4 -> 10.3 us, 4000 -> 2000, 4 rows 14.4 -> 12.4;
  // fp32 blocks, bound by their twelve MMAs, gain less: 4096 -> 4096, 9 rows 26.3 -> 24.8.
  p.a_rows = static_cast<int>(std::min<long long>(kTcBlockM, (M + 7) / 8 * 8));
  const int res_mode = res_mode_of(e);
  p.direct = direct_rows(kind, e, N, &p.wide) ? 1 : 0;
  p.block_n = choose_block_n(p.tiles_m, N, sm_count, 16);
  set_chunks(p, kind, p.row_bytes);
  if (const int width = split_width(p, e, N, p.block_n, sm_count)) {
    p.block_n = width;
    p.split_k = 1;
  }
  if (!p.a_im2col) {
    const RowsSplit rows = split_rows(kind, M, p.k_blocks, e, N, sm_count);
    if (rows.chunks > 1) {
      p.chunk_blocks = rows.chunk_blocks;
      p.chunks = rows.chunks;
      if (rows.apart && split_k_enabled()) {
        p.block_n = rows.block_n;
        p.split_k = 1;
      }
    }
  }
  p.sk_ws = e.sk_ws;
  p.sk_flags = e.sk_flags;
  p.tiles_n = (N + p.block_n - 1) / p.block_n;
  const int drain = kDrainBytes + (e.side_count > 0 ? 8 * 2 * kDrainSideBytes : 0);  // (room for two int8 copies)
  const int planes = tc_planes(kind);
  // a stage holds the A tile(s) and block_n rows of B, every sub-buffer 1 KB aligned
  const int b_bytes = (p.block_n * p.row_bytes + 1023) / 1024 * 1024;
  p.stage_bytes = planes * (kTcBlockM * p.row_bytes + b_bytes);
  const long long tiles_total = static_cast<long long>(p.tiles_m) * p.tiles_n;
  // Paired tiles: two 128-row halves share every B tile, so a K block moves 256 + block_n operand
  // rows for twice the output instead of 2 x (128 + block_n).  Worth it where the operand fetch sets
  // the pace (deep contractions over full 128-byte rows; the stem's 64-byte window rows ran 9%
  // slower paired) and the coarser tiles still fill the SMs wave by wave; the ring then holds two
  // (larger) stages.
  p.pair = 0;
  p.pair_rows = 0;
  if (pair_enabled() && p.chunks == 1 && p.k_blocks >= 6 && p.block_n <= 128 && p.row_bytes >= 128) {
    const int pair_stage = planes * (2 * kTcBlockM * p.row_bytes + b_bytes);
    const long long waves_single = (tiles_total + sm_count - 1) / sm_count;
    const double cost_single = static_cast<double>(waves_single) * (kTcBlockM + p.block_n);
    // whole waves of pairs first, single tiles for what is left; k waves of pairs cover
    // floor(k * SMs / tiles_n) tile rows of 256
    const int max_pair_rows = p.tiles_m / 2;
    double best = cost_single;
    int best_rows = 0;
    for (int k = 1; k <= 65; ++k) {  // up to 64 waves of pairs, then "all pairs"
      const int rows = k == 65 ? max_pair_rows
                               : static_cast<int>(std::min<long long>(max_pair_rows, static_cast<long long>(k) * sm_count / p.tiles_n));
      const long long pair_tiles = static_cast<long long>(rows) * p.tiles_n;
      const long long single_tiles = static_cast<long long>(p.tiles_m - 2 * rows) * p.tiles_n;
      const double cost = static_cast<double>((pair_tiles + sm_count - 1) / sm_count) * (2 * kTcBlockM + p.block_n) +
                          static_cast<double>((single_tiles + sm_count - 1) / sm_count) * (kTcBlockM + p.block_n);
      if (cost < best - 1e-9) {
        best = cost;
        best_rows = rows;
      }
      if (rows == max_pair_rows) break;
    }
    const long long tiles_mixed = static_cast<long long>(p.tiles_m - best_rows) * p.tiles_n;
    if (best_rows > 0 && best < 0.97 * cost_single && tiles_mixed * 10 >= 9ll * sm_count &&
        (kTcSmemBudget - drain) / pair_stage >= 2) {
      p.pair = 1;
      p.pair_rows = best_rows;
      p.tiles_m = p.tiles_m - best_rows;  // tile rows: best_rows pairs, then singles
      p.stage_bytes = pair_stage;
    }
  }
  const int budget = kTcSmemBudget - drain;
  // int8 K blocks are two to four MMAs over 12-32 KB: arming and releasing a ring stage (~450 cycles of barrier
  // hand-shake per block, more than the block's copies and MMAs take) sets the pace.  A stage then holds several
  // K blocks (a divisor of their count, at least three stages deep): one hand-shake for all of them.
  p.sub_blocks = 1;
  if (kind == GEMM_I8 && !p.pair && !p.split_k && env_int("NCNN_B200_SUB_BLOCKS", 1) != 0)
    for (int sub : {4, 3, 2})
      if (p.k_blocks % sub == 0 && budget / (sub * p.stage_bytes) >= 3) {
        p.sub_blocks = sub;
        break;
      }
  p.stages = std::max(2, std::min(kTcMaxStages, budget / (p.sub_blocks * p.stage_bytes)));
  L->smem_bytes = p.stages * p.sub_blocks * p.stage_bytes + drain + 1024;
  // never fewer bytes than half an SM's shared memory: two CTAs must not share an
  // SM, each allocates tensor memory for itself
  L->smem_bytes = std::max(L->smem_bytes, 120 * 1024);
  const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * (p.split_k ? p.chunks : 1);
  L->grid = static_cast<int>(std::min<long long>(units, sm_count));
  L->kind = kind;
  p.bias = e.bias;
  p.scale = e.scale;
  p.out0 = e.out0;
  p.out1 = e.out1;
  p.outq = e.outq;
  p.res0 = e.res0;
  p.res1 = e.res1;
  p.res_mode = res_mode;
  p.ldo = e.ldo;
  p.out_mode = e.out_mode;
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.out_scale = e.out_scale;
  p.status = e.status;
  p.trace = e.trace;
  p.side_count = e.side_count;
  p.side_ld = e.ldo;
  p.side_q0 = e.side_q[0];
  p.side_q1 = e.side_q[1];
  p.side_scale0 = e.side_scale[0];
  p.side_scale1 = e.side_scale[1];
}

// ---- CTA pairs (tc_gemm2.cuh)
// NCNN_B200_CTA2=0 keeps every contraction on the one-CTA kernel; NCNN_B200_STREAMK=0 never splits
// a tile between pairs, =1 always does where it can; NCNN_B200_CTA2_MIN_KB sets the shallowest
// contraction (K blocks per tile) that goes to pairs.
int env_int(const char* name, int fallback) {
  const char* f = std::getenv(name);
  return f == nullptr || f[0] == 0 ? fallback : std::atoi(f);
}

int max_pairs_resident(int kind, int smem_bytes, int sm_count);

// Launch attributes of the contraction kernels: clusters of two CTAs for the pair form, and programmatic
// stream serialisation: the kernel's preamble (barriers, tensor memory, descriptor prefetch) may run while
// the previous kernel of the stream drains; the kernel itself waits (grid_dependency_wait) before it
// touches any tensor.
struct KernelLaunchConfig {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attrs[2];
  KernelLaunchConfig(int grid, int threads, int smem_bytes, bool pair, cudaStream_t stream) {
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
    cfg.stream = stream;
    cfg.attrs = attrs;
    cfg.numAttrs = 0;
    if (pair) {
      attrs[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
      attrs[cfg.numAttrs].val.clusterDim.x = 2;
      attrs[cfg.numAttrs].val.clusterDim.y = 1;
      attrs[cfg.numAttrs].val.clusterDim.z = 1;
      ++cfg.numAttrs;
    }
    if (tc_pdl_enabled()) {
      attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attrs[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
      ++cfg.numAttrs;
    }
  }
};

// True when tc_gemm2_kernel takes this contraction (on CTA pairs, or on single CTAs with tiles split
// between them); fills the plan like finish_plan does.
// `half_blocks_ok`: K blocks of half the size (64-byte rows) address the same packed operands, so
// the plan may trade K-block size for ring stages.
bool finish_plan_workers(TcLaunch* L, int kind, long long M, int N, const TcEpilogue& e, int sm_count,
                         bool half_blocks_ok) {
  TcGemmParams& p = L->p;
  if (env_int("NCNN_B200_CTA2", 1) == 0 || sm_count < 2) return false;
  if (p.k_blocks < env_int("NCNN_B200_CTA2_MIN_KB", 6)) return false;
  const int res_mode = res_mode_of(e);
  p.direct = direct_rows(kind, e, N, &p.wide) ? 1 : 0;
  if (!p.direct || e.out_mode == OUT_CHW) return false;  // this kernel drains dense rows only
  if (e.side_count > 0) return false;  // int8 copies of the result: the one-CTA kernel writes those
  const int step = 16;
  auto even_width = [&](int widest) {
    const int n_tiles = (N + widest - 1) / widest;
    return ((N + n_tiles - 1) / n_tiles + step - 1) / step * step;
  };
  const int full_kb = p.k_blocks;
  const int forced_split = env_int("NCNN_B200_STREAMK", -1);
  const bool ws_given = e.sk_ws != nullptr && e.sk_flags != nullptr;

  // Form 1, CTA pairs: tiles of 256 rows x up to 256 columns.  Measured on ResNet-18 at batch 64: tiles of
  // 256 columns keep the tensor pipe busy through the whole main loop (the operand path of an SM carries half
  // the bytes per product); narrower pair tiles gain nothing over the one-CTA kernel's paired tiles and pay
  // more barrier hand-shakes per output.  Taken when whole tiles fill at least one wave of pairs.
  const int pair_bn = even_width(kTc2MaxBlockN);
  const long long pair_tiles = ((M + kTc2TileM - 1) / kTc2TileM) * ((N + pair_bn - 1) / pair_bn);
  const int one_bn = even_width(128);
  const long long one_tiles = ((M + kTcBlockM - 1) / kTcBlockM) * ((N + one_bn - 1) / one_bn);
  // Sums in chunks (the same in every form, so the batch may decide): tiles of 256 columns have no second accumulator
  // while the running sum takes its place, so the MMAs of a pair wait for every chunk to be added, and a wave of pair
  // tiles takes ~1.6 waves of the one-CTA kernel's, which has room for both.  Pairs where they still come out ahead: two
  // layers of 7x7x512 -> 512 and their edges, pairs / one CTA in us, with the waves of each: 192 images (1, 2) 207 / 228,
  // 208 (2, 3) 353 / 318, 256 (2, 3) 347 / 334, 296 (2, 4) 354 / 432, 448 (3, 5) 549 / 611, 512 (3, 6) 557 / 659; 768
  // channels, 128 images (2, 2) 483 / 318, 192 (2, 3) 493 / 512.  Operand rows of 64 bytes stay on pairs, which fetch
  // half of the weights each (14x14x392 -> 392, 64 images (2, 3) 303 / 379).
  const bool chunked = kind == GEMM_BF16X3 && p.a_im2col && p.row_bytes == 128 && full_kb >= kTcChunkFrom;
  const long long pair_waves = (pair_tiles + sm_count / 2 - 1) / (sm_count / 2), one_waves = (one_tiles + sm_count - 1) / sm_count;
  const bool pairs_win = pair_tiles >= sm_count / 2 && (!chunked || 3 * pair_waves < 2 * one_waves);
  const bool pair_form = pair_bn >= env_int("NCNN_B200_CTA2_MIN_BN", 192) && (pairs_win || env_int("NCNN_B200_CTA2_ALWAYS", 0) != 0);
  // Form 2, single CTAs with split tiles: tiles of 128 rows x up to 128 columns, every SM an equal share of
  // the K blocks.  Taken when whole tiles would leave SMs idle (few, deep tiles) and the workspace allows.
  const long long one_units = one_tiles * full_kb;
  const int one_workers = static_cast<int>(std::min<long long>(sm_count, one_units / 4));
  bool split_form = false;
  // Where a tile is cut depends on how many tiles there are, so a split layer rounds its fp32 sums
  // differently at different batch sizes.  Convolutions keep whole tiles (splitting them gained nothing
  // on the benchmark networks, and a batch then equals its images run one by one bit for bit);
  // InnerProduct and Gemm, where a handful of rows must stream megabytes of weights, are split.
  const bool may_split = forced_split == 1 || (forced_split != 0 && !p.a_im2col);
  if (!pair_form && ws_given && may_split && one_workers >= 2) {
    // Every worker ends with the tile it finishes, whose partial sums arrive no earlier than the other
    // workers finish theirs: publishing, waiting and adding them is an exposed tail worth about twenty
    // K blocks (measured on 3x3 convolutions of 256 and 512 channels at batch 64, where splitting lost).
    const double cost_whole = static_cast<double>((one_tiles + sm_count - 1) / sm_count) * full_kb;
    const double cost_split = static_cast<double>((one_units + one_workers - 1) / one_workers) + 20.0;
    split_form = forced_split == 1 || cost_split < 0.9 * cost_whole;
    // (chunks of K on different CTAs do the same without workers that wait, and win where rows are few.  A tile of many
    // workers waits for each of them: 4096 -> 512, 200 rows, 18 to a tile 55 us, whole 41; 4096 -> 4096, 2 to a tile 39.5 and 40.9)
    const double block = std::max(tc_planes(kind) * 3.0 * (kTcBlockM + one_bn), (kind == GEMM_I8 ? 4.0 : 12.0) * (kTcBlockM + one_bn) / 4.0);
    const double waits = kind == GEMM_BF16X3 ? 4000.0 * std::max(0.0, static_cast<double>(one_workers) / one_tiles - 2.5) : 0.0;
    if (forced_split != 1 && split_rows(kind, M, full_kb, e, N, sm_count).clocks < cost_split * block + 3000.0 + waits) split_form = false;
  }
  if (!pair_form && !split_form) return false;
  const int ctas = pair_form ? 2 : 1;
  const int tile_m = pair_form ? kTc2TileM : kTcBlockM;

  p.M = static_cast<int>(M);
  p.N = N;
  p.tiles_m = static_cast<int>((M + tile_m - 1) / tile_m);
  p.block_n = pair_form ? pair_bn : one_bn;
  p.tiles_n = (N + p.block_n - 1) / p.block_n;
  const int budget_all = kTcSmemBudget;
  const int planes = tc_planes(kind);
  // Full-size K blocks with a ring deep enough to cover the copy latency, else half-size ones.
  const int full_rb = p.row_bytes, full_cb = p.c_blocks, full_ke = p.k_elems;
  auto try_config = [&](bool half_blocks, int min_stages) {
    const int rb = half_blocks ? full_rb / 2 : full_rb;
    const int b_bytes = ((p.block_n / ctas) * rb + 1023) / 1024 * 1024;
    const int stage = planes * (kTcBlockM * rb + b_bytes);
    const int stages = std::min(kTcMaxStages, (budget_all - kDrainBytes) / stage);
    if (stages < min_stages) return false;
    p.row_bytes = rb;
    p.k_elems = half_blocks ? full_ke / 2 : full_ke;
    p.c_blocks = half_blocks ? full_cb * 2 : full_cb;
    p.k_blocks = half_blocks ? full_kb * 2 : full_kb;
    p.half_blocks = half_blocks ? 1 : 0;
    p.stage_bytes = stage;
    p.stages = stages;
    return true;
  };
  const bool halves = half_blocks_ok && full_rb == 128 && kind == GEMM_BF16X3;
  if (!try_config(false, 3) && !(halves && try_config(true, 4)) && !try_config(false, 2)) return false;
  p.pair = 0;
  p.pair_rows = 0;
  p.sub_blocks = 1;
  L->smem_bytes = std::max(p.stages * p.stage_bytes + kDrainBytes + 1024, 120 * 1024);
  L->kind = kind;
  L->cta2 = ctas;
  // workers: one per TPC (pairs) or per SM, all resident at once
  int workers = pair_form ? std::min(sm_count / 2, max_pairs_resident(kind, L->smem_bytes, sm_count)) : sm_count;
  if (workers < 1) return false;
  const long long tiles = static_cast<long long>(p.tiles_m) * p.tiles_n;
  const long long units = tiles * p.k_blocks;
  if (forced_split == 1) workers = static_cast<int>(std::max<long long>(1, std::min<long long>(workers, units / 4)));
  // Splitting tiles pays when whole tiles leave SMs idle in the last wave; the worker that finishes a
  // split tile spends about three K blocks' time on the partial sums.
  const double cost_whole = static_cast<double>((tiles + workers - 1) / workers) * p.k_blocks;
  const double cost_split = static_cast<double>((units + workers - 1) / workers) + 20.0 * p.k_blocks / full_kb;
  const size_t ws_need = static_cast<size_t>(ctas * workers) * kTcBlockM * p.block_n * 4;
  const bool can_split = ws_given && e.sk_ws_bytes >= ws_need && e.sk_flag_count >= 2 * ctas * workers &&
                         units >= 4ll * workers;
  if (split_form) {
    if (!can_split && units < 4ll * workers) workers = static_cast<int>(std::max<long long>(1, units / 4));
    p.streamk = ws_given && e.sk_ws_bytes >= static_cast<size_t>(workers) * kTcBlockM * p.block_n * 4 &&
                        e.sk_flag_count >= 2 * workers
                    ? 1
                    : 0;
    if (!p.streamk) {
      p.row_bytes = full_rb;
      p.k_elems = full_ke;
      p.c_blocks = full_cb;
      p.k_blocks = full_kb;
      p.half_blocks = 0;
      L->cta2 = 0;
      return false;
    }
  } else {
    p.streamk = can_split && may_split && (forced_split == 1 || cost_split < 0.95 * cost_whole) ? 1 : 0;
  }
  set_chunks(p, kind, full_rb);
  if (p.streamk) p.chunks = 1;  // (forced: a tile is cut where the workers' shares end)
  if (!p.streamk) workers = static_cast<int>(std::min<long long>(workers, tiles));
  p.sk_ws = e.sk_ws;
  p.sk_flags = e.sk_flags;
  L->grid = ctas * workers;
  p.bias = e.bias;
  p.scale = e.scale;
  p.out0 = e.out0;
  p.out1 = e.out1;
  p.outq = e.outq;
  p.res0 = e.res0;
  p.res1 = e.res1;
  p.res_mode = res_mode;
  p.ldo = e.ldo;
  p.out_mode = e.out_mode;
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.out_scale = e.out_scale;
  p.status = e.status;
  p.trace = e.trace;
  p.side_count = e.side_count;
  p.side_ld = e.ldo;
  p.side_q0 = e.side_q[0];
  p.side_q1 = e.side_q[1];
  p.side_scale0 = e.side_scale[0];
  p.side_scale1 = e.side_scale[1];
  return true;
}

}  // namespace

int tc_row_bytes(int kind, int channels) {
  if (kind == GEMM_I8) {
    if (channels % 16 != 0) return 0;
    return channels > 64 ? 128 : (channels > 32 ? 64 : 32);
  }
  // bf16 rows: 64 channels when they divide evenly, else 32 per block; a last block that
  // reaches past the tensor is zero-filled by TMA (pixel rows must stay 16-byte multiples)
  if (kind == GEMM_BF16X3) return channels % 64 == 0 ? 128 : (channels % 8 == 0 ? 64 : 0);
  if (channels % 4 != 0) return 0;
  return 128;
}

int tc_k_elems(int kind, int channels) {
  const int rb = tc_row_bytes(kind, channels);
  if (rb == 0) return 0;
  return rb / tc_elem_bytes(kind);
}

std::string tc_plan_conv_tiles(TcLaunch* L, int kind, const TcIm2colView& v, int out_channels, const TcEpilogue& e, int sm_count) {
  load_driver_entry_points();
  if (!g_driver_error.empty()) return g_driver_error;
  const int rb = tc_row_bytes(kind, static_cast<int>(v.C));
  if (rb == 0) return "channel count is not addressable by TMA (row not a multiple of 16 bytes)";
  TcGemmParams& p = L->p;
  std::memset(&p, 0, sizeof(p));
  p.row_bytes = rb;
  p.k_elems = rb / tc_elem_bytes(kind);
  p.a_rows = kTcBlockM;
  p.c_blocks = static_cast<int>((v.C + p.k_elems - 1) / p.k_elems);
  p.k_blocks = v.KH * v.KW * p.c_blocks;
  p.a_im2col = 1;
  p.OH = v.OH;
  p.OW = v.OW;
  p.KW = v.KW;
  p.stride_h = v.stride_conv_h;
  p.stride_w = v.stride_conv_w;
  p.pad_t = v.pad_t;
  p.pad_l = v.pad_l;
  p.dil_h = v.dil_h;
  p.dil_w = v.dil_w;
  const long long M = static_cast<long long>(v.N) * v.OH * v.OW;
  if (M > 0x7fffffffll) return "too many output pixels for one launch";
  L->cta2 = 0;
  if (!finish_plan_workers(L, kind, M, out_channels, e, sm_count, v.C % 64 == 0))
    finish_plan(L, kind, M, out_channels, e, sm_count);
  return {};
}

std::string tc_encode_conv(TcLaunch* L, int kind, const TcIm2colView& v, const void* w0, const void* w1, int out_channels) {
  const TcGemmParams& p = L->p;
  const uint32_t b_box_rows = static_cast<uint32_t>(L->cta2 == 2 ? p.block_n / 2 : p.block_n);
  const int prb = p.row_bytes;  // the pair plan may have halved the K blocks

  std::string err = encode_im2col(&L->map_a0, kind, v.plane0, v, p.k_elems, static_cast<uint32_t>(p.a_rows), prb);
  if (!err.empty()) return err;
  if (tc_planes(kind) == 2) {
    err = encode_im2col(&L->map_a1, kind, v.plane1, v, p.k_elems, static_cast<uint32_t>(p.a_rows), prb);
    if (!err.empty()) return err;
  } else {
    L->map_a1 = L->map_a0;
  }
  const uint64_t k_total = static_cast<uint64_t>(p.k_blocks) * p.k_elems;
  err = encode_tiled_2d(&L->map_b0, kind, w0, k_total, out_channels,
                        k_total * elem_bytes(kind), p.k_elems, b_box_rows, prb);
  if (!err.empty()) return err;
  if (tc_planes(kind) == 2) {
    err = encode_tiled_2d(&L->map_b1, kind, w1, k_total, out_channels,
                          k_total * elem_bytes(kind), p.k_elems, b_box_rows, prb);
    if (!err.empty()) return err;
  } else {
    L->map_b1 = L->map_b0;
  }
  return {};
}

std::string tc_plan_conv(TcLaunch* L, int kind, const TcIm2colView& v, const void* w0, const void* w1, int out_channels, const TcEpilogue& e,
                         int sm_count) {
  const std::string err = tc_plan_conv_tiles(L, kind, v, out_channels, e, sm_count);
  return err.empty() ? tc_encode_conv(L, kind, v, w0, w1, out_channels) : err;
}

std::string tc_plan_gemm(TcLaunch* L, int kind, const void* a0, const void* a1, long long M, int K,
                         long long lda, const void* w0, const void* w1, int N,
                         const TcEpilogue& e, int sm_count) {
  load_driver_entry_points();
  if (!g_driver_error.empty()) return g_driver_error;
  const int es = elem_bytes(kind);
  if ((lda * es) % 16 != 0) return "row stride of A is not a multiple of 16 bytes";
  if (M > 0x7fffffffll) return "too many rows for one launch";
  TcGemmParams& p = L->p;
  std::memset(&p, 0, sizeof(p));
  p.row_bytes = 128;
  p.k_elems = 128 / es;
  p.a_rows = kTcBlockM;
  p.c_blocks = (K + p.k_elems - 1) / p.k_elems;
  p.k_blocks = p.c_blocks;
  p.a_im2col = 0;
  p.OH = p.OW = p.KW = 1;
  p.stride_h = p.stride_w = p.dil_h = p.dil_w = 1;
  L->cta2 = 0;
  if (!finish_plan_workers(L, kind, M, N, e, sm_count, K % 64 == 0)) finish_plan(L, kind, M, N, e, sm_count);
  const uint32_t b_box_rows = static_cast<uint32_t>(L->cta2 == 2 ? p.block_n / 2 : p.block_n);
  const int prb = p.row_bytes;  // the pair plan may have halved the K blocks
  std::string err = encode_tiled_2d(&L->map_a0, kind, a0, K, M, lda * es, p.k_elems, static_cast<uint32_t>(p.a_rows), prb);
  if (!err.empty()) return err;
  if (tc_planes(kind) == 2) {
    err = encode_tiled_2d(&L->map_a1, kind, a1, K, M, lda * es, p.k_elems, static_cast<uint32_t>(p.a_rows), prb);
    if (!err.empty()) return err;
  } else {
    L->map_a1 = L->map_a0;
  }
  const uint64_t k_total = static_cast<uint64_t>(p.k_blocks) * p.k_elems;
  err = encode_tiled_2d(&L->map_b0, kind, w0, k_total, N, k_total * es, p.k_elems, b_box_rows, prb);
  if (!err.empty()) return err;
  if (tc_planes(kind) == 2) {
    err = encode_tiled_2d(&L->map_b1, kind, w1, k_total, N, k_total * es, p.k_elems, b_box_rows, prb);
    if (!err.empty()) return err;
  } else {
    L->map_b1 = L->map_b0;
  }
  return {};
}

namespace {

// Calls f(std::integral_constant<int, EPI>) for the epilogue form of a launch (see `drains`).
template <int KIND, bool CHW, class F>
cudaError_t with_form(int out_mode, bool res, F&& f) {
#define NB_FORM(OUT, RES) \
  if (out_mode == OUT && res == RES) return f(std::integral_constant<int, epi_form(OUT, RES)>{})
  NB_FORM(OUT_F32, false);
  NB_FORM(OUT_F32, true);
  if constexpr (CHW) {
    NB_FORM(OUT_CHW, false);
    NB_FORM(OUT_CHW, true);
  }
  if constexpr (KIND == GEMM_I8) {
    NB_FORM(OUT_I8, false);
  }
  if constexpr (KIND == GEMM_BF16X3 || KIND == GEMM_TF32X3) {
    NB_FORM(OUT_BF16X2, false);
    NB_FORM(OUT_BF16X2, true);
  }
  if constexpr (KIND == GEMM_TF32X3) {
    NB_FORM(OUT_F32_SPLIT, false);
    NB_FORM(OUT_F32_SPLIT, true);
  }
  if constexpr (KIND == GEMM_TF32) {
    NB_FORM(OUT_F32_TF32, false);
    NB_FORM(OUT_F32_TF32, true);
  }
#undef NB_FORM
  return cudaErrorInvalidValue;
}

// Opts a kernel in to `smem` bytes of dynamic shared memory, once per device (the attribute belongs to a device's context).
template <class K>
cudaError_t opt_in(K kernel, int smem) {
  static std::mutex mutex;
  static std::map<std::pair<const void*, int>, cudaError_t> done;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mutex);
  const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), device);
  const auto it = done.find(key);
  if (it != done.end()) return it->second;
  return done[key] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

template <class K, class... Args>
cudaError_t launch_opted(K kernel, int max_smem, KernelLaunchConfig& lc, const Args&... args) {
  const cudaError_t e = opt_in(kernel, max_smem);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&lc.cfg, kernel, args...);
}

template <int KIND>
int pairs_resident(int smem_bytes, int sm_count) {
  KernelLaunchConfig wc(sm_count / 2 * 2, kTc2Threads, smem_bytes, true, nullptr);
  int clusters = 0;
  const auto kernel = tc_gemm2_kernel<KIND, true, epi_form(OUT_F32, false)>;
  if (opt_in(kernel, kTcSmemBudget + 1024) != cudaSuccess || cudaOccupancyMaxActiveClusters(&clusters, kernel, &wc.cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return clusters;
}

// how many CTA pairs of the kernel the device runs at once (no device: as many as there are TPCs)
int max_pairs_resident(int kind, int smem_bytes, int sm_count) {
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    cudaGetLastError();
    return sm_count / 2;
  }
  switch (kind) {
    case GEMM_TF32: return pairs_resident<GEMM_TF32>(smem_bytes, sm_count);
    case GEMM_TF32X3: return pairs_resident<GEMM_TF32X3>(smem_bytes, sm_count);
    case GEMM_BF16X3: return pairs_resident<GEMM_BF16X3>(smem_bytes, sm_count);
    default: return pairs_resident<GEMM_I8>(smem_bytes, sm_count);
  }
}

template <int KIND>
cudaError_t launch_workers(const TcLaunch& L, cudaStream_t stream) {
  const bool pair = L.cta2 == 2;
  KernelLaunchConfig wc(L.grid, kTc2Threads, L.smem_bytes, pair, stream);
  return with_form<KIND, false>(L.p.out_mode, L.p.res_mode != RES_NONE, [&](auto form) {
    constexpr int EPI = decltype(form)::value;
    if (pair) return launch_opted(tc_gemm2_kernel<KIND, true, EPI>, kTcSmemBudget + 1024, wc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
    return launch_opted(tc_gemm2_kernel<KIND, false, EPI>, kTcSmemBudget + 1024, wc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
  });
}

cudaError_t tc_launch_workers(const TcLaunch& L, cudaStream_t stream) {
  cudaError_t e;
  switch (L.kind) {
    case GEMM_TF32: e = launch_workers<GEMM_TF32>(L, stream); break;
    case GEMM_TF32X3: e = launch_workers<GEMM_TF32X3>(L, stream); break;
    case GEMM_BF16X3: e = launch_workers<GEMM_BF16X3>(L, stream); break;
    default: e = launch_workers<GEMM_I8>(L, stream); break;
  }
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <int KIND>
cudaError_t launch_gemm(const TcLaunch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, kTcThreads, L.smem_bytes, false, stream);
  const int max_smem = kTcSmemBudget + 1024;  // contents + alignment slack
  // (int8 copies of an fp32 result are written by instantiations of their own)
  if constexpr (KIND == GEMM_I8) {
    if (L.p.side_count > 0) {
      if (!L.p.direct || L.p.out_mode != OUT_F32)
        return launch_opted(tc_gemm_kernel<KIND, kEpiAny, true>, max_smem, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
      if (L.p.res_mode != RES_NONE)
        return launch_opted(tc_gemm_kernel<KIND, epi_form(OUT_F32, true), true>, max_smem, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
      return launch_opted(tc_gemm_kernel<KIND, epi_form(OUT_F32, false), true>, max_smem, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
    }
  }
  if (!L.p.direct) return launch_opted(tc_gemm_kernel<KIND, kEpiAny>, max_smem, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
  return with_form<KIND, true>(L.p.out_mode, L.p.res_mode != RES_NONE, [&](auto form) {
    return launch_opted(tc_gemm_kernel<KIND, decltype(form)::value>, max_smem, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
  });
}

}  // namespace

cudaError_t tc_launch(const TcLaunch& L, cudaStream_t stream) {
  if (L.cta2) return tc_launch_workers(L, stream);
  cudaError_t e;
  switch (L.kind) {
    case GEMM_TF32: e = launch_gemm<GEMM_TF32>(L, stream); break;
    case GEMM_TF32X3: e = launch_gemm<GEMM_TF32X3>(L, stream); break;
    case GEMM_BF16X3: e = launch_gemm<GEMM_BF16X3>(L, stream); break;
    default: e = launch_gemm<GEMM_I8>(L, stream); break;
  }
  return e != cudaSuccess ? e : cudaGetLastError();
}

// ------------------------------------------------------------------ patch-resident convolution
namespace {

std::string encode_tiled_4d(CUtensorMap* map, bool bf16, const void* base, int C, int W, int H, int N, uint32_t box_c,
                            uint32_t box_w, uint32_t box_h, CUtensorMapSwizzle swizzle) {
  const cuuint64_t es = bf16 ? 2 : 4;
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(C), static_cast<cuuint64_t>(W), static_cast<cuuint64_t>(H),
                              static_cast<cuuint64_t>(N)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(C) * es, static_cast<cuuint64_t>(C) * es * W,
                                 static_cast<cuuint64_t>(C) * es * W * H};
  const cuuint32_t box[4] = {box_c, box_w, box_h, 1};
  const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
  const CUresult r = g_encode_tiled(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                                    const_cast<void*>(base), dims, strides,
                                    box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return "cuTensorMapEncodeTiled (4-D) failed with code " + std::to_string(static_cast<int>(r));
  return {};
}

}  // namespace

bool tc_halo_applies(int kind, int C, int KH, int KW, int stride_h, int stride_w, int dil_h, int dil_w, int OH,
                     int OW, int out_channels, int out_mode) {
  if (kind != GEMM_TF32 && kind != GEMM_TF32X3 && kind != GEMM_BF16X3) return false;
  if (stride_h != 1 || stride_w != 1 || dil_h != 1 || dil_w != 1) return false;
  if (KH * KW < 2 || KH > 7 || KW > 7) return false;  // a 1x1 filter has nothing to reuse
  if (C % (kind == GEMM_BF16X3 ? 64 : 32) != 0 || out_channels % 4 != 0 || out_mode == OUT_I8) return false;
  if (out_mode == OUT_BF16X2 && out_channels % 32 != 0) return false;
  const double covered = static_cast<double>((OH + kHaloTileH - 1) / kHaloTileH * kHaloTileH) *
                         ((OW + kHaloTileW - 1) / kHaloTileW * kHaloTileW);
  return static_cast<double>(OH) * OW / covered >= 0.70;
}

std::string tc_plan_conv_halo(TcHaloLaunch* L, int kind, const TcHaloConv& c, const TcEpilogue& e, int sm_count,
                              bool pair) {
  load_driver_entry_points();
  if (!g_driver_error.empty()) return g_driver_error;
  TcHaloParams& p = L->p;
  std::memset(&p, 0, sizeof(p));
  const int planes = tc_planes(kind);
  const bool a_bf16 = kind == GEMM_BF16X3;
  const int res_mode = res_mode_of(e);
  if (e.out_mode == OUT_CHW || e.out_mode == OUT_I8 || e.side_count > 0 || !direct_rows(kind, e, c.out_channels, &p.wide))
    return "the patch-resident kernel writes channel-last rows of 16-byte pieces";
  if (e.ldo != c.out_channels) return "the patch-resident kernel writes dense channel-last rows";
  p.images = c.images;
  p.OH = c.OH;
  p.OW = c.OW;
  p.N = c.out_channels;
  p.tiles_y = (c.OH + kHaloTileH - 1) / kHaloTileH;
  p.tiles_x = (c.OW + kHaloTileW - 1) / kHaloTileW;
  // an MMA of any N <= 128 costs the same issue time: take the widest tile
  const int step = pair ? 32 : 16;
  const int widest = pair ? 256 : 128;  // a pair's CTA holds half of the weight rows of a tap
  {
    const int n_tiles = (c.out_channels + widest - 1) / widest;
    p.block_n = ((c.out_channels + n_tiles - 1) / n_tiles + step - 1) / step * step;
  }
  p.tiles_n = (c.out_channels + p.block_n - 1) / p.block_n;
  const int ctas = pair ? 2 : 1;
  L->pair = pair ? 1 : 0;
  if (pair && (p.block_n / 2) % 8 != 0) return "a pair's half of the weight tile must be whole 8-row groups";
  p.k_elems = 128 / tc_elem_bytes(kind);
  p.c_blocks = c.C / p.k_elems;
  p.taps = c.KH * c.KW;
  p.KW = c.KW;
  p.pad_t = c.pad_t;
  p.pad_l = c.pad_l;
  p.patch_h = kHaloTileH + c.KH - 1;
  p.patch_w = kHaloTileW + c.KW - 1;
  p.patch_bytes = (p.patch_h * p.patch_w * 128 + 1023) / 1024 * 1024;
  p.b_bytes = ((p.block_n / ctas) * 128 + 1023) / 1024 * 1024;
  p.bias = e.bias;
  p.res_mode = res_mode;
  p.out0 = e.out0;
  p.out1 = e.out1;
  p.res0 = e.res0;
  p.res1 = e.res1;
  p.out_mode = e.out_mode;
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.status = e.status;
  p.trace = e.trace;
  const int fixed = 2 * planes * p.patch_bytes + kDrainBytes;
  p.stages = (kTcSmemBudget - fixed) / (planes * p.b_bytes);
  p.stages = std::min(p.stages, kTcMaxStages);
  if (p.stages < 2) return "shared memory cannot hold the patch buffers and two weight stages";
  L->smem_bytes = fixed + p.stages * planes * p.b_bytes + 1024;
  L->smem_bytes = std::max(L->smem_bytes, 120 * 1024);
  const long long pixel_tiles = static_cast<long long>(c.images) * p.tiles_y * p.tiles_x;
  const long long tiles = ((pixel_tiles + ctas - 1) / ctas) * p.tiles_n;
  if (pixel_tiles * p.tiles_n > 0x7fffffffll) return "too many tiles for one launch";
  L->grid = ctas * static_cast<int>(std::min<long long>(tiles, sm_count / ctas));
  L->kind = kind;

  std::string err = encode_tiled_4d(&L->map_a0, a_bf16, c.in0, c.C, c.W, c.H, c.images, p.k_elems, p.patch_w,
                                    p.patch_h, CU_TENSOR_MAP_SWIZZLE_128B);
  if (err.empty() && planes == 2)
    err = encode_tiled_4d(&L->map_a1, a_bf16, c.in1, c.C, c.W, c.H, c.images, p.k_elems, p.patch_w, p.patch_h,
                          CU_TENSOR_MAP_SWIZZLE_128B);
  if (!err.empty()) return err;
  const uint64_t k_total = static_cast<uint64_t>(p.taps) * p.c_blocks * p.k_elems;
  err = encode_tiled_2d(&L->map_b0, kind, c.w0, k_total, c.out_channels, k_total * tc_elem_bytes(kind), p.k_elems,
                        p.block_n / ctas, 128);
  if (err.empty() && planes == 2)
    err = encode_tiled_2d(&L->map_b1, kind, c.w1, k_total, c.out_channels, k_total * tc_elem_bytes(kind), p.k_elems,
                          p.block_n / ctas, 128);
  if (!err.empty()) return err;
  return err;
}

cudaError_t tc_launch_halo(const TcHaloLaunch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, kHaloThreads, L.smem_bytes, L.pair != 0, stream);
  auto launch = [&](auto kind) {
    constexpr int KIND = decltype(kind)::value;
    return with_form<KIND, false>(L.p.out_mode, L.p.res_mode != RES_NONE, [&](auto form) {
      constexpr int EPI = decltype(form)::value;
      if (L.pair) return launch_opted(tc_conv_halo_kernel<KIND, true, EPI>, kTcSmemBudget + 1024, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
      return launch_opted(tc_conv_halo_kernel<KIND, false, EPI>, kTcSmemBudget + 1024, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
    });
  };
  cudaError_t e;
  if (L.kind == GEMM_BF16X3) e = launch(std::integral_constant<int, GEMM_BF16X3>{});
  else if (L.kind == GEMM_TF32X3) e = launch(std::integral_constant<int, GEMM_TF32X3>{});
  else e = launch(std::integral_constant<int, GEMM_TF32>{});
  return e != cudaSuccess ? e : cudaGetLastError();
}

// ------------------------------------------------------------------ convolution of few pixels
namespace {

// Expected clocks of a layer's launch.  A K block takes what its MMAs take (128 bytes of operands a clock, or the tensor
// rate) or what its copies take (~3 clocks a row of 128 bytes, ~2 of 64), whichever is longer.
double mma_clocks(int m, int n) { return std::max({m == 64 ? 23.0 : 39.0, (m + n) / 4.0, n * m / (m == 64 ? 128.0 : 256.0)}); }
double k_block_clocks(int row_bytes, int m, int n, double rows) {
  return std::max(row_bytes / 32 * 3 * mma_clocks(m, n), rows * (row_bytes == 128 ? 3.0 : 2.0)) + 20.0;
}

double gemm_clocks(const TcLaunch& L, int sm_count) {
  const TcGemmParams& p = L.p;
  const double fixed = 3000.0 + 12.0 * p.block_n + (p.split_k || p.streamk ? 3000.0 : 0.0);
  if (L.cta2 == 2) {
    const double block = k_block_clocks(p.row_bytes, 128, p.block_n, 2.0 * (kTcBlockM + p.block_n / 2));
    const long long tiles = static_cast<long long>(p.tiles_m) * p.tiles_n, workers = L.grid / 2;
    return fixed + static_cast<double>((tiles + workers - 1) / workers) * p.k_blocks * block;
  }
  // (what lies between two blocks is hidden behind wide MMAs only)
  const double block = std::max(k_block_clocks(p.row_bytes, 128, p.block_n, 2.0 * (kTcBlockM + p.block_n)),
                                p.row_bytes / 32 * 3 * mma_clocks(128, p.block_n) + 330.0);
  const long long singles = static_cast<long long>(p.tiles_m - p.pair_rows) * p.tiles_n * (p.split_k ? p.chunks : 1);
  const long long pairs = static_cast<long long>(p.pair_rows) * p.tiles_n;
  const double pair_block = p.pair ? std::max(2.0 * p.row_bytes / 32 * 3 * mma_clocks(128, p.block_n), 6.0 * (2 * kTcBlockM + p.block_n)) : 0.0;
  const int blocks = p.split_k ? p.chunk_blocks : p.k_blocks;
  return fixed + blocks * (static_cast<double>((singles + sm_count - 1) / sm_count) * block + static_cast<double>((pairs + sm_count - 1) / sm_count) * pair_block);
}

}  // namespace

std::string tc_plan_conv_patch(TcPatchLaunch* L, int kind, const TcIm2colView& v, const void* w0, const void* w1,
                               int out_channels, const TcEpilogue& e, int sm_count, const TcLaunch& gemm, bool always) {
  const int stride = v.stride_conv_h;
  if (kind != GEMM_BF16X3 || v.stride_conv_w != stride || (stride != 1 && stride != 2) || v.dil_h != 1 || v.dil_w != 1 || v.KH > 16 || v.KW > 16)
    return "the patch kernel takes bf16 pairs, strides of 1 or 2 and no dilation";
  int wide = 0;
  if (e.out_mode == OUT_I8 || e.side_count > 0 || !direct_rows(kind, e, out_channels, &wide)) return "the patch kernel writes rows of 16-byte pieces";
  const int rb = tc_row_bytes(kind, static_cast<int>(v.C));
  if (rb == 0) return "channel count is not addressable by TMA";
  TcGemmParams g{};  // K blocks and chunks as tc_gemm_kernel has them
  g.row_bytes = rb;
  g.k_elems = rb / 2;
  g.c_blocks = static_cast<int>((v.C + g.k_elems - 1) / g.k_elems);
  g.k_blocks = v.KH * v.KW * g.c_blocks;
  g.a_im2col = 1;
  set_chunks(g, kind, rb);
  const int taps = v.KH * v.KW;
  if (taps < 2) return "a 1x1 filter has nothing to reuse";
  // (a single tile of few K blocks stays with tc_gemm_kernel because the test of that kernel's waits asks for it there, not
  // because it is faster: whole calls of 64 -> 64, 4x4 to 11x11 pixels, and of 64 -> 256, 11x11, take 10.4 us there and 8.3 here)
  if (!always && gemm.cta2 == 0 && gemm.p.tiles_m == 1 && g.k_blocks <= 9) return "a single short tile";
  // The model ranks tile shapes well and both kernels' tiles roughly: with operand rows of 128 bytes this kernel came out
  // ahead up to 0.68 of the other's clocks, with rows of 64 bytes (channel counts that are no multiple of 64) up to 0.81.
  // 3x3 layers, launches by events (~8 us of which are the events'), other kernel -> this one:
  //   64 channels, 56x56     1 image 13.3 -> 11.6    4: 15.4 -> 15.3      8: 21.6 -> 19.5    16: 24.2 -> 27.7 (0.97)
  //   128, 28x28             1: 17.4 -> 13.4         3: 17.5 -> 17.3      6: 17.6 -> 19.5 (0.75)
  //   256, 14x14             1: 25.5 -> 17.4         8: 25.6 -> 23.0     16: 27.7 -> 26.9    24: 27.6 -> 39.9 (1.13)
  //   512, 7x7 (in chunks)   1: 21.6 -> 17.3         2: 21.2 -> 19.6      4: 21.5 -> 25.1 (0.82)
  //   256 -> 512, stride 2   1: 25.6 -> 19.5         8: 25.6 -> 20.1     12: 25.6 -> 30.4 (1.09)
  //   96, 28x28              1: 19.4 -> 13.3        16: 29.7 -> 19.5     32: 40.2 -> 27.7    64: 42.0 -> 48.2 (0.87)
  //   168, 50x50             1: 30.8 -> 21.5         8: 97.4 -> 66.6     12: 125 -> 87       16: 128 -> 119 (0.87)
  TcPatchParams best{};
  double best_clocks = always ? 1e300 : (rb == 128 ? 0.68 : 0.81) * gemm_clocks(gemm, sm_count);
  // one tile shape: 8 or 16 rows of 8 pixels, `bn` columns, groups of all taps of a channel block or of a filter row
  auto consider = [&](int th, int bn, bool whole_groups) {
    TcPatchParams p{};
    p.images = static_cast<int>(v.N);
    p.tile_h = th;
    p.tiles_y = (v.OH + th - 1) / th;
    p.tiles_x = (v.OW + kPatchTileW - 1) / kPatchTileW;
    p.block_n = bn;
    p.tiles_n = (out_channels + bn - 1) / bn;
    const long long tiles = static_cast<long long>(v.N) * p.tiles_y * p.tiles_x * p.tiles_n;
    if (tiles > (1 << 24)) return;
    p.subs = stride;
    p.row_step = stride;
    p.patch_h = (th - 1) * stride + v.KH;
    p.patch_w = ((kPatchTileW - 1) * stride + v.KW + stride - 1) / stride;
    p.sub_bytes = (p.patch_w * p.patch_h * rb + 1023) / 1024 * 1024;
    p.step_even = stride == 2 ? p.sub_bytes : rb;
    p.step_odd = stride == 2 ? rb - p.sub_bytes : rb;
    p.group = whole_groups ? taps : v.KW;
    if (g.chunks > 1 && g.chunk_blocks % p.group != 0) return;  // (a chunk holds whole groups)
    p.group_rows = p.group / v.KW;
    p.patch_groups = v.KH / p.group_rows;
    p.groups = g.k_blocks / p.group;
    p.chunk_groups = g.chunks > 1 ? g.chunk_blocks / p.group : p.groups;
    p.b_bytes = (bn * rb + 1023) / 1024 * 1024;
    p.acc_cols = (bn + 31) / 32 * 32;
    const int buf = 2 * p.subs * p.sub_bytes, stage = p.group * 2 * p.b_bytes, drain = 4 * kDrainWarpBytes;
    // two CTAs to an SM (of this kernel only: anything less than 110 KB would let in the others, which take all of
    // tensor memory), or one with deeper rings
    auto fits = [&](int budget, int bufs, int least) {
      p.patch_bufs = bufs;
      p.stages = std::min({kTcMaxStages, p.groups, (budget - drain - bufs * buf) / stage});
      return p.stages >= std::min(least, p.groups);
    };
    if (!fits(111 * 1024, 2, 2) && !fits(kTcSmemBudget, 3, 3) && !fits(kTcSmemBudget, 2, 2)) return;
    const double block = k_block_clocks(rb, 8 * th, bn, 2.0 * p.subs * p.patch_w * p.patch_h / taps + 2.0 * bn) + 350.0 / p.group;
    for (int split = 0; split <= (g.chunks > 1 ? 1 : 0); ++split) {
      const long long units = tiles * (split ? g.chunks : 1);
      if (split && (e.sk_ws == nullptr || e.sk_flags == nullptr || tiles * 4 > e.sk_flag_count ||
                    static_cast<size_t>(units) * kTcBlockM * bn * 4 > e.sk_ws_bytes))
        continue;
      const double waves = static_cast<double>((units + sm_count - 1) / sm_count);
      const double clocks = 3000.0 + 12.0 * bn + (split ? 3000.0 + static_cast<double>(units) * bn / 4.0 : 0.0) +
                            waves * ((split ? g.chunk_blocks : g.k_blocks) * block + 300.0);
      if (clocks >= best_clocks) continue;
      best_clocks = clocks;
      best = p;
      best.split_k = split;
    }
  };
  for (int th : {8, 16})
    for (int bn = 16; bn <= 128 && bn < out_channels + 16; bn += 16)
      for (bool whole_groups : {true, false}) consider(th, bn, whole_groups);
  if (best.tile_h == 0) return "other kernels are expected to be as fast";
  TcPatchParams& p = L->p;
  p = best;
  p.OH = v.OH;
  p.OW = v.OW;
  p.N = out_channels;
  p.c_blocks = g.c_blocks;
  p.k_elems = g.k_elems;
  p.row_bytes = rb;
  p.taps = taps;
  p.KW = v.KW;
  p.k_blocks = g.k_blocks;
  p.stride = stride;
  p.pad_t = v.pad_t;
  p.pad_l = v.pad_l;
  p.chunks = g.chunks;
  const int cols = p.acc_cols * (p.chunks > 1 && !p.split_k ? 3 : 2);
  p.tmem_cols = 32;
  while (p.tmem_cols < cols) p.tmem_cols *= 2;
  p.sk_ws = e.sk_ws;
  p.sk_flags = e.sk_flags;
  p.wide = wide;
  p.bias = e.bias;
  p.out0 = e.out0;
  p.out1 = e.out1;
  p.res0 = e.res0;
  p.res1 = e.res1;
  p.ldo = e.ldo;
  p.res_mode = res_mode_of(e);
  p.out_mode = e.out_mode;
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.status = e.status;
  const int contents = p.patch_bufs * 2 * p.subs * p.sub_bytes + p.stages * p.group * 2 * p.b_bytes + 4 * kDrainWarpBytes;
  L->smem_bytes = std::max(contents + 1024, 110 * 1024);
  if (p.tmem_cols > 256) L->smem_bytes = std::max(L->smem_bytes, 120 * 1024);
  L->kind = kind;
  const long long units = static_cast<long long>(p.images) * p.tiles_y * p.tiles_x * p.tiles_n * (p.split_k ? p.chunks : 1);
  L->grid = static_cast<int>(std::min<long long>(units, sm_count));

  const cuuint64_t dims[4] = {v.C, v.W, v.H, v.N};
  const cuuint64_t strides[3] = {v.stride_w, v.stride_h, v.stride_n};
  const cuuint32_t step = static_cast<cuuint32_t>(stride);  // (a copy skips every other column at stride 2)
  const cuuint32_t box[4] = {static_cast<cuuint32_t>(p.k_elems), (static_cast<cuuint32_t>(p.patch_w) - 1) * step + 1, static_cast<cuuint32_t>(p.patch_h), 1};
  const cuuint32_t elem_strides[4] = {1, step, 1, 1};
  if (box[1] > 256 || box[2] > 256) return "the patch does not fit a TMA box";
  for (int plane = 0; plane < 2; ++plane) {
    const CUresult r = g_encode_tiled(plane ? &L->map_a1 : &L->map_a0, dtype_for(kind), 4, const_cast<void*>(plane ? v.plane1 : v.plane0), dims,
                                      strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(rb),
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return "cuTensorMapEncodeTiled (patch) failed with code " + std::to_string(static_cast<int>(r));
  }
  const uint64_t k_total = static_cast<uint64_t>(p.k_blocks) * p.k_elems;
  std::string err = encode_tiled_2d(&L->map_b0, kind, w0, k_total, out_channels, k_total * 2, p.k_elems, p.block_n, rb);
  if (err.empty()) err = encode_tiled_2d(&L->map_b1, kind, w1, k_total, out_channels, k_total * 2, p.k_elems, p.block_n, rb);
  return err;
}

cudaError_t tc_launch_patch(const TcPatchLaunch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, kPatchThreads, L.smem_bytes, false, stream);
  const cudaError_t e = with_form<GEMM_BF16X3, true>(L.p.out_mode, L.p.res_mode != RES_NONE, [&](auto form) {
    return launch_opted(tc_conv_patch_kernel<GEMM_BF16X3, decltype(form)::value>, kTcSmemBudget + 1024, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
  });
  return e != cudaSuccess ? e : cudaGetLastError();
}

// ------------------------------------------------------------------ int8 convolution with its filter resident
std::string tc_plan_conv_i8(TcConvI8Launch* L, const TcIm2colView& v, const void* w, int out_channels, const TcEpilogue& e, int sm_count,
                            bool always) {
  load_driver_entry_points();
  if (!g_driver_error.empty()) return g_driver_error;
  const int taps = v.KH * v.KW;
  if (v.stride_conv_h != 1 || v.stride_conv_w != 1 || v.dil_h != 1 || v.dil_w != 1 || taps < 2 || v.KH > 16 || v.KW > 16)
    return "the kernel takes filters of several taps, stride 1 and no dilation";
  const int rb = tc_row_bytes(GEMM_I8, static_cast<int>(v.C));
  if (rb < 64) return "rows of 32 bytes or none";
  TcConvI8Params& p = L->p;
  std::memset(&p, 0, sizeof(p));
  const int res_mode = res_mode_of(e);
  if ((e.out_mode != OUT_I8 && e.out_mode != OUT_F32) || (e.side_count > 0 && e.out_mode != OUT_F32) || (res_mode != RES_NONE && res_mode != RES_F32) ||
      !direct_rows(GEMM_I8, e, out_channels, &p.wide))
    return "the kernel writes channel-last rows of 16-byte pieces";
  p.images = static_cast<int>(v.N);
  p.OH = v.OH;
  p.OW = v.OW;
  p.N = out_channels;
  p.tiles_y = (v.OH + kI8TileH - 1) / kI8TileH;
  p.tiles_x = (v.OW + kI8TileW - 1) / kI8TileW;
  const long long tiles = static_cast<long long>(v.N) * p.tiles_y * p.tiles_x;
  if (tiles > (1 << 28)) return "too many tiles for one launch";
  p.row_bytes = p.k_elems = rb;
  p.c_blocks = (static_cast<int>(v.C) + rb - 1) / rb;
  p.KH = v.KH;
  p.KW = v.KW;
  p.pad_t = v.pad_t;
  p.pad_l = v.pad_l;
  p.patch_h = kI8TileH + v.KH - 1;
  p.patch_w = kI8TileW + v.KW - 1;
  p.patch_bytes = (p.patch_h * p.patch_w * rb + 1023) / 1024 * 1024;
  p.drain_bytes = (e.out_mode == OUT_I8 ? kDrainSideBytes : kDrainWarpBytes) + e.side_count * kDrainSideBytes;
  const int blocks = taps * p.c_blocks;
  // the widest column block that leaves room for two patches and an epilogue group, then more groups, then more patches
  for (int parts = 1; parts <= (out_channels + 15) / 16; ++parts) {
    p.block_n = ((out_channels + parts - 1) / parts + 15) / 16 * 16;
    if (p.block_n > 256) continue;
    p.b_bytes = (p.block_n * rb + 1023) / 1024 * 1024;
    p.acc_cols = (p.block_n + 31) / 32 * 32;
    for (p.groups = kI8MaxGroups; p.groups >= 1; --p.groups) {
      if (p.groups * p.acc_cols > static_cast<int>(kTcTmemCols)) continue;
      p.patches = std::min(kI8MaxPatches, (kTcSmemBudget - blocks * p.b_bytes - 4 * p.groups * p.drain_bytes) / p.patch_bytes);
      if (p.patches >= 2) break;
    }
    if (p.groups >= 2) break;
  }
  if (p.groups < 2) return "the filter does not fit shared memory";
  p.accs = p.groups * std::min({static_cast<int>(kTcTmemCols) / (p.groups * p.acc_cols), kI8MaxAccs / p.groups, 2});
  p.tiles_n = (out_channels + p.block_n - 1) / p.block_n;
  if (p.tiles_n > sm_count) return "more column blocks than SMs";
  // Launches of ResNet-18's layers by events (~8 us of which are the events'), tc_gemm_kernel (or pairs of CTAs) -> this one; the
  // second figure of a pair is a layer that adds an fp32 residual and writes fp32 and an int8 copy:
  //   64 channels, 56x56           1 image 10.4, 12.6 -> 10.6, 13.3   4: 11.8, 14.1 -> 10.3, 13.7   64: 37, 51 -> 21, 41   256: 120, 160 -> 53, 116
  //       33x33 (57 % of the tiles filled), 256 images 47, 69 -> 33, 64;  16x16, 16 images (one wave) 12.0, 12.6 -> 10.4, 13.5
  //   128, 28x28 (77 %)            4: 11.2 -> 12.7   16: 14.4, 16.3 -> 13.5, 14.5   64: 20.5, 30.8 -> 18.5, 29.8   96: 22.6, 39.4 -> 22.4, 40.1
  //       256: 43, 86 -> 38, 88;  fp32 results without a residual  64: 22.5 -> 22.2   96: 24.5 -> 26.7   192: 38 -> 43   256: 47 -> 51
  //       17x17 (38 %), 256 images 22.5, 24.7 -> 31, 41
  //   256 (four column blocks), 14x14   4: 12.6, 15.2 -> 12.0, 14.3   16 (one wave): 14.4, 16.8 -> 12.5, 16.3   256: 38, 59 -> 43, 80
  //   512 (16), 7x7                1: 16.4 -> 12.5   4 (one wave): 16.4 -> 12.7   16: 16.6 -> 18.4
  // With one tile to a CTA nothing is reused, and what is left is a shorter chain: from 18 K blocks on.  With several the filter's
  // reuse wins, unless tiles are mostly empty or the pixels are read again for each of many column blocks.  Beside a filter of
  // 128-byte rows fp32 results have room for two epilogue groups, or for three and half of the columns, and the drain falls
  // behind: up to four tiles an SM (128 images, residual: 52.6 and 49.3, where the other kernel's last wave is short).
  const long long waves = (tiles + sm_count / p.tiles_n - 1) / (sm_count / p.tiles_n);
  const double filled = static_cast<double>(v.OH) * v.OW / (static_cast<double>(p.tiles_y) * p.tiles_x * kI8TileH * kI8TileW);
  const bool slow_drain = rb == 128 && e.out_mode == OUT_F32 && tiles > 4ll * sm_count;
  const bool pays = waves == 1 ? blocks >= 18 : p.tiles_n <= 2 && !slow_drain && filled >= (rb == 64 ? 0.5 : 0.7);
  if (!always && !pays) return "other kernels are expected to be as fast";
  p.bias = e.bias;
  p.scale = e.scale;
  p.out0 = e.out0;
  p.outq = e.outq;
  p.res0 = e.res0;
  p.ldo = e.ldo;
  p.res_mode = res_mode;
  p.far_res = p.res_mode == RES_F32 && static_cast<long long>(v.N) * v.OH * v.OW * e.ldo * 4 > (126ll << 20);
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.out_scale = e.out_scale;
  p.side_count = e.side_count;
  p.side_q0 = e.side_q[0];
  p.side_q1 = e.side_q[1];
  p.side_scale0 = e.side_scale[0];
  p.side_scale1 = e.side_scale[1];
  p.status = e.status;
  L->out_mode = e.out_mode;
  L->threads = 64 + 128 * p.groups;
  // never fewer bytes than half an SM's shared memory: each CTA takes all of tensor memory
  L->smem_bytes = std::max(blocks * p.b_bytes + p.patches * p.patch_bytes + 4 * p.groups * p.drain_bytes + 1024, 120 * 1024);
  L->grid = p.tiles_n * static_cast<int>(std::min<long long>(tiles, sm_count / p.tiles_n));

  const cuuint64_t dims[4] = {v.C, v.W, v.H, v.N};
  const cuuint64_t strides[3] = {v.stride_w, v.stride_h, v.stride_n};
  const cuuint32_t box[4] = {static_cast<cuuint32_t>(p.k_elems), static_cast<cuuint32_t>(p.patch_w), static_cast<cuuint32_t>(p.patch_h), 1};
  const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
  const CUresult r = g_encode_tiled(&L->map_a, dtype_for(GEMM_I8), 4, const_cast<void*>(v.plane0), dims, strides, box, elem_strides,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(rb), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return "cuTensorMapEncodeTiled (int8 patch) failed with code " + std::to_string(static_cast<int>(r));
  const uint64_t k_total = static_cast<uint64_t>(blocks) * p.k_elems;
  return encode_tiled_2d(&L->map_b, GEMM_I8, w, k_total, out_channels, k_total, p.k_elems, p.block_n, rb);
}

cudaError_t tc_launch_conv_i8(const TcConvI8Launch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, L.threads, L.smem_bytes, false, stream);
  const int max_smem = kTcSmemBudget + 1024;
  cudaError_t e;
  if (L.p.side_count > 0) {
    if (L.p.res_mode != RES_NONE) e = launch_opted(tc_conv_i8_kernel<epi_form(OUT_F32, true), true>, max_smem, lc, L.p, L.map_a, L.map_b);
    else e = launch_opted(tc_conv_i8_kernel<epi_form(OUT_F32, false), true>, max_smem, lc, L.p, L.map_a, L.map_b);
  } else {
    e = with_form<GEMM_I8, false>(L.out_mode, L.p.res_mode != RES_NONE, [&](auto form) {
      return launch_opted(tc_conv_i8_kernel<decltype(form)::value, false>, max_smem, lc, L.p, L.map_a, L.map_b);
    });
  }
  return e != cudaSuccess ? e : cudaGetLastError();
}

// ------------------------------------------------------------------ depthwise + projection
namespace {

struct DwProjShape {
  int block_n = 0, tiles_n = 0, stages = 0, patches = 0, drain_groups = 0, b_bytes = 0, x_plane_bytes = 0, x_row_bytes = 64, x_bufs = 0, accs = 2, e_bufs = 0;
  int a_slots = 0, smem = 0;
  bool ok = false;
};
bool dw_project_formats(int out_mode, int res_mode) { return (out_mode == OUT_BF16X2 || out_mode == OUT_F32) && res_mode != RES_SPLIT; }
// columns of a tile: N in as few tiles of at most 256 as it takes, all alike
void dw_project_columns(DwProjShape& r, int N) {
  const int n_tiles = (N + 255) / 256;
  r.block_n = ((N + n_tiles - 1) / n_tiles + 15) / 16 * 16;
  r.tiles_n = (N + r.block_n - 1) / r.block_n;
  r.b_bytes = (r.block_n * 64 + 1023) / 1024 * 1024;
}

// Shared-memory plan of the pair with one or two groups of epilogue warps.
DwProjShape dw_project_shape(int N, int out_mode, int res_mode, int C, int drain_groups) {
  DwProjShape r;
  if (!dw_project_formats(out_mode, res_mode)) return r;
  dw_project_columns(r, N);
  r.drain_groups = drain_groups;
  const int c_pad = (C + kDwpChannels - 1) / kDwpChannels * kDwpChannels;
  const int table = (c_pad * 10 * 4 + 1023) / 1024 * 1024;  // depthwise filter and bias
  const int stage = 2 * r.b_bytes;
  // Deep patch ring first (a patch load outlasts one block's arithmetic), then three weight stages (plenty); the last
  // resort is two of each.
  for (int min_stages : {3, 2}) {
    // (an even ring only: the two depthwise groups take alternate blocks, so with an even depth a slot always
    // belongs to the same group, which waits for its phases in order; with three slots a slot would alternate
    // between the groups, a group would wait for every second phase of it, and a parity wait cannot tell a
    // phase from the one two before it: a load delayed past a whole block's arithmetic let a group read a stale
    // patch, about once in 10^5 loads with the L2 flushed)
    for (int patches : {4, 2}) {
      const int fixed = patches * kDwpPatchBytes + 2 * 2 * kDwpAPlaneBytes + drain_groups * 4 * kDrainWarpBytes + table;
      const int stages = std::min(kDwpMaxStages, (kTcSmemBudget - fixed) / stage);
      if (stages >= min_stages) {
        r.stages = stages;
        r.patches = patches;
        r.smem = fixed + stages * stage + 1024;
        r.ok = true;
        return r;
      }
    }
  }
  return r;
}

// A second group hides the drain of a tile behind the next one, which counts on short chains of channel blocks; on long ones its
// 16 KB may be two of four patches or one of three weight stages, which count more.  Calls in us, one group / two where the
// rings differ: 48x48x32 -> 384, 30 images 137 / 117; 48x48x128 -> 208, 59 images 220 / 204; 24x24x192 -> 352, 106 images 181 / 173;
// 24x24x256 -> 320, 160 images 269 / 273; 48x48x288 -> 320, 38 images 258 / 262; 14x14x384 -> 288, 356 images 279 / 285; 48x48x672 -> 112,
// 35 images 326 / 333; 16x16x1152 -> 96, 137 images 238 / 244.  Where both leave the same rings two never lose.
// What has no room for two groups even with two patches and two stages is no pair: 1344 -> 256 takes 145 (14x14, 64 images), 489
// (256) and 469 us (28x28, 64) as one, 135, 490 and 469 as two launches.
DwProjShape dw_project_shape(int N, int out_mode, int res_mode, int C) {
  const DwProjShape one = dw_project_shape(N, out_mode, res_mode, C, 1), two = dw_project_shape(N, out_mode, res_mode, C, 2);
  const bool same_rings = two.patches == one.patches && std::min(two.stages, 3) == std::min(one.stages, 3);
  return !two.ok || C <= 8 * kDwpChannels || same_rings ? two : one;
}

// Shared and tensor memory plan of the whole block.  Where its weights do not stay, stride-2 blocks stream them (64 images of
// 28x28x384 -> 64: 47 us a call, 74 as three layers; 56x56x384 -> 128 139, 264).
// Eight operand tiles before two input patches: four (one for each quarter of a set) leave the depthwise warps waiting for
// the projection's MMAs, while a patch is needed by the expand MMAs only, which run ahead.
DwProjShape block_shape(int N, int out_mode, int res_mode, int C, int stride, int cin) {
  DwProjShape r;
  if (!dw_project_formats(out_mode, res_mode) || (stride != 1 && stride != 2)) return r;
  // One column tile: a second is a whole tile of the kernel, its expand and depthwise work done once more.  64 images of
  // 56x56x96 with 160 outputs in two: stride 1 227 us a call, 217 as expand layer and pair; stride 2 117, 102 as three layers.
  if (N > 128) return r;
  dw_project_columns(r, N);
  // Two accumulators beside one buffer of each half's expanded pixels, or two where they fit; past 96 columns at stride 2 one
  // accumulator (56x56x144 -> 128, 64 images: a call takes 108 us, 131 with two accumulators and two column tiles).
  const int pixels = blk_in_cols(stride), columns = static_cast<int>(kTcTmemCols);
  r.accs = 2 * r.block_n + 2 * pixels <= columns ? 2 : 1;
  r.e_bufs = 2 * r.block_n + 4 * pixels <= columns ? 2 : 1;
  r.x_row_bytes = cin <= 16 ? 32 : 64;
  r.x_plane_bytes = (dwp_patch_pixels(stride) * r.x_row_bytes + 1023) / 1024 * 1024;
  const int c_blocks = (C + kDwpChannels - 1) / kDwpChannels, c_pad = c_blocks * kDwpChannels;
  const int table = (kBlkTableRows * c_pad * 4 + 1023) / 1024 * 1024;
  const int fixed = table + dwp_tile_h(stride) * kDwpTileW / 32 * kDrainWarpBytes;
  const int stage = 2 * r.b_bytes;
  for (bool streamed : {false, true}) {
    if (streamed && stride == 1) break;
    const int weights = streamed ? 2 * 4 * kDwpChannels * r.x_row_bytes : 2 * c_pad * r.x_row_bytes + c_blocks * stage;
    for (int slots : {8, 4})
      for (int x_bufs : {2, 1}) {
        int smem = fixed + weights + x_bufs * 2 * r.x_plane_bytes + slots * 2 * blk_a_plane_bytes(stride);
        if (streamed) {
          r.stages = std::min(kBlkMaxStages, (kTcSmemBudget - smem) / stage);
          if (r.stages < (slots == 8 || x_bufs == 2 ? 4 : 2)) continue;
          smem += r.stages * stage;
        }
        if (smem > kTcSmemBudget) continue;
        r.x_bufs = x_bufs;
        r.a_slots = slots;
        r.smem = smem + 1024;
        r.ok = true;
        return r;
      }
  }
  return r;
}

// an image that fills less than 60 % of its tiles (7 x 7 fills 38 % of a 16 x 8 tile) is faster as separate layers
bool dw_project_fills(int H, int W, int stride) {
  const int th = dwp_tile_h(stride);
  const int tiles = ((H + th - 1) / th) * ((W + kDwpTileW - 1) / kDwpTileW);
  return env_int("NCNN_B200_FUSE_DW", 1) >= 2 || static_cast<long long>(H) * W * 10 >= 6ll * tiles * th * kDwpTileW;
}

// The pair splits its registers between its roles (setmaxnreg): with fewer at launch than the split counts on, the depthwise warps
// would wait for registers that nobody gives back, in an instruction that no time limit covers.
std::string pair_registers(int out_mode, bool res) {
  int regs = 0;
  const cudaError_t e = with_form<GEMM_BF16X3, false>(out_mode, res, [&](auto form) {
    cudaFuncAttributes a;
    const cudaError_t q = cudaFuncGetAttributes(&a, tc_dw_project_kernel<GEMM_BF16X3, 1, false, decltype(form)::value>);
    regs = q == cudaSuccess ? a.numRegs : 0;
    return q;
  });
  if (e != cudaSuccess) return std::string("attributes of the fused depthwise + projection kernel: ") + cudaGetErrorString(e);
  regs = env_int("NCNN_B200_TEST_PAIR_REGS", regs);  // (as if compiled for so many)
  if (regs != kDwpRegs)
    return "the fused depthwise + projection kernel was compiled for " + std::to_string(regs) + " registers a thread, its roles share " +
           std::to_string(kDwpRegs);
  return "";
}

}  // namespace

bool tc_dw_project_applies(int C, int N, int H, int W, int out_mode, bool has_res, bool res_bf16) {
  if (C % 4 != 0 || C < 8 || N % 8 != 0 || H < 1 || W < 1) return false;
  if (!dw_project_fills(H, W, 1)) return false;
  const int res_mode = !has_res ? RES_NONE : (res_bf16 ? RES_BF16X2 : RES_F32);
  if (out_mode == OUT_F32 && N % 4 != 0) return false;
  return dw_project_shape(N, out_mode, res_mode, C).ok;
}

bool tc_block_applies(int Cin, int C, int N, int OH, int OW, int stride, bool has_res) {
  if (Cin < 8 || Cin > 32 || Cin % 8 != 0 || C % 8 != 0 || C < 32 || N % 8 != 0 || OH < 1 || OW < 1) return false;
  if (has_res && stride != 1) return false;
  if (C > (kTcChunkFrom - 1) * kDwpChannels) return false;  // (a projection that deep may be summed in chunks, the block sums it whole)
  if (!dw_project_fills(OH, OW, stride)) return false;
  // whatever formats the planner gives the output and the residual later
  for (int out_mode : {OUT_F32, OUT_BF16X2})
    for (int res_mode : {RES_NONE, RES_F32, RES_BF16X2}) {
      if (!has_res && res_mode != RES_NONE) continue;
      if (has_res && res_mode == RES_NONE) continue;
      if (!block_shape(N, out_mode, res_mode, C, stride, Cin).ok) return false;
    }
  return true;
}

bool tc_block_streams(int Cin, int C, int N, int stride) { return block_shape(N, OUT_F32, RES_NONE, C, stride, Cin).stages > 0; }

std::string tc_plan_dw_project(TcDwProjLaunch* L, const TcDwProjConv& c, const TcEpilogue& e, int sm_count) {
  load_driver_entry_points();
  if (!g_driver_error.empty()) return g_driver_error;
  TcDwProjParams& p = L->p;
  std::memset(&p, 0, sizeof(p));
  const int res_mode = res_mode_of(e);
  if (!direct_rows(GEMM_BF16X3, e, c.out_channels, &p.wide)) return "the fused depthwise + projection kernel writes rows of 16-byte pieces";
  const bool expand = c.ex_w0 != nullptr;
  const int stride = c.stride;
  const DwProjShape shape = expand ? block_shape(c.out_channels, e.out_mode, res_mode, c.C, stride, c.Cin)
                                   : (stride == 1 ? dw_project_shape(c.out_channels, e.out_mode, res_mode, c.C) : DwProjShape{});
  if (!shape.ok) return "the fused depthwise + projection kernel does not take this output format, width or stride";
  if (e.ldo != c.out_channels) return "the fused depthwise + projection kernel writes dense channel-last rows";
  std::string err = expand ? std::string() : pair_registers(e.out_mode, res_mode != RES_NONE);
  if (!err.empty()) return err;
  const int x_channels = expand ? c.Cin : c.C;
  if ((reinterpret_cast<uintptr_t>(c.x) & 15) != 0 || (static_cast<size_t>(x_channels) * (expand ? 2 : 4)) % 16 != 0 ||
      (expand && (c.x1 == nullptr || (reinterpret_cast<uintptr_t>(c.x1) & 15) != 0)))
    return "input rows of the fused kernel must be 16-byte aligned";
  const int th = dwp_tile_h(stride);
  p.images = c.images;
  p.H = c.H;
  p.W = c.W;
  p.Hin = c.Hin;
  p.Win = c.Win;
  p.C = c.C;
  p.N = c.out_channels;
  p.tiles_y = (c.H + th - 1) / th;
  p.tiles_x = (c.W + kDwpTileW - 1) / kDwpTileW;
  p.block_n = shape.block_n;
  p.tiles_n = shape.tiles_n;
  p.c_blocks = (c.C + kDwpChannels - 1) / kDwpChannels;
  p.pad_t = c.pad_t;
  p.pad_l = c.pad_l;
  p.stages = shape.stages;
  p.patch_bufs = shape.patches;
  p.drain_groups = shape.drain_groups;
  p.b_bytes = shape.b_bytes;
  p.dw_weights = c.dw_weights;
  p.dw_bias = c.dw_bias;
  p.dw_act = c.dw_act;
  p.dw_act_a = c.dw_act_a;
  p.dw_act_b = c.dw_act_b;
  p.x_plane_bytes = shape.x_plane_bytes;
  p.x_row_bytes = shape.x_row_bytes;
  p.x_bufs = shape.x_bufs;
  p.accs = shape.accs;
  p.e_bufs = shape.e_bufs;
  p.a_slots = shape.a_slots;
  p.ex_ksteps = expand ? (shape.x_row_bytes == 32 ? 1 : (c.Cin + 15) / 16) : 0;
  p.ex_bias = c.ex_bias;
  p.ex_act = c.ex_act;
  p.ex_act_a = c.ex_act_a;
  p.ex_act_b = c.ex_act_b;
  p.bias = e.bias;
  p.res_mode = res_mode;
  p.out0 = e.out0;
  p.out1 = e.out1;
  p.res0 = e.res0;
  p.res1 = e.res1;
  p.out_mode = e.out_mode;
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.status = e.status;
  L->stride = stride;
  L->expand = expand;
  L->smem_bytes = std::max(shape.smem, 120 * 1024);
  const long long tiles = static_cast<long long>(c.images) * p.tiles_y * p.tiles_x * p.tiles_n;
  if (tiles > 0x7fffffffll) return "too many tiles for one launch";
  L->grid = static_cast<int>(std::min<long long>(tiles, sm_count));
  // input patches, [image][Hin][Win][channels], boxes of 32 channels x patch width x patch height: fp32 and dense
  // in shared memory for the depthwise filter; with the expand layer fused in, the bf16 planes of the block's input
  // as 64-byte-swizzled operand rows (channels past Cin read as zero)
  const uint32_t x_box = expand ? static_cast<uint32_t>(shape.x_row_bytes / 2) : kDwpChannels;
  const CUtensorMapSwizzle x_swizzle = !expand ? CU_TENSOR_MAP_SWIZZLE_NONE
                                               : (shape.x_row_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B);
  err = encode_tiled_4d(&L->map_x, expand, c.x, x_channels, c.Win, c.Hin, c.images, x_box, dwp_patch_w(stride),
                                    dwp_patch_h(stride), x_swizzle);
  if (err.empty() && expand)
    err = encode_tiled_4d(&L->map_x1, true, c.x1, x_channels, c.Win, c.Hin, c.images, x_box, dwp_patch_w(stride),
                          dwp_patch_h(stride), x_swizzle);
  // expand weights: [C][32] bf16 per plane (64-byte pitch), one block of 32 rows per copy, as many K columns as the rows hold
  if (err.empty() && expand) err = encode_tiled_2d(&L->map_e0, GEMM_BF16X3, c.ex_w0, 32, c.C, 64, x_box, kDwpChannels, shape.x_row_bytes);
  if (err.empty() && expand) err = encode_tiled_2d(&L->map_e1, GEMM_BF16X3, c.ex_w1, 32, c.C, 64, x_box, kDwpChannels, shape.x_row_bytes);
  if (!err.empty()) return err;
  const uint64_t k_total = static_cast<uint64_t>(p.c_blocks) * kDwpChannels;
  err = encode_tiled_2d(&L->map_b0, GEMM_BF16X3, c.w0, k_total, c.out_channels, k_total * 2, kDwpChannels, p.block_n, 64);
  if (err.empty())
    err = encode_tiled_2d(&L->map_b1, GEMM_BF16X3, c.w1, k_total, c.out_channels, k_total * 2, kDwpChannels, p.block_n, 64);
  if (!err.empty()) return err;
  return err;
}

cudaError_t tc_launch_dw_project(const TcDwProjLaunch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, L.expand ? kBlkThreads : kDwpThreads, L.smem_bytes, false, stream);
  constexpr int max_smem = kTcSmemBudget + 1024;
  const cudaError_t e = with_form<GEMM_BF16X3, false>(L.p.out_mode, L.p.res_mode != RES_NONE, [&](auto form) {
    constexpr int EPI = decltype(form)::value;
    if (!L.expand) return launch_opted(tc_dw_project_kernel<GEMM_BF16X3, 1, false, EPI>, max_smem, lc, L.p, L.map_x, L.map_x1, L.map_e0, L.map_e1, L.map_b0, L.map_b1);
    if (L.stride == 1) return launch_opted(tc_dw_project_kernel<GEMM_BF16X3, 1, true, EPI>, max_smem, lc, L.p, L.map_x, L.map_x1, L.map_e0, L.map_e1, L.map_b0, L.map_b1);
    if (L.p.stages > 0) return launch_opted(tc_dw_project_kernel<GEMM_BF16X3, 2, true, EPI, true>, max_smem, lc, L.p, L.map_x, L.map_x1, L.map_e0, L.map_e1, L.map_b0, L.map_b1);
    return launch_opted(tc_dw_project_kernel<GEMM_BF16X3, 2, true, EPI>, max_smem, lc, L.p, L.map_x, L.map_x1, L.map_e0, L.map_e1, L.map_b0, L.map_b1);
  });
  return e != cudaSuccess ? e : cudaGetLastError();
}

float tf32_round_host(float x) {
  // round to nearest, ties away from zero, onto 10 explicit mantissa bits
  uint32_t u;
  std::memcpy(&u, &x, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return x;
  u += 0x1000u;
  u &= 0xffffe000u;
  float r;
  std::memcpy(&r, &u, 4);
  return r;
}

void tc_pack_weights_f32(int kind, const float* w, int O, int I, int KH, int KW, int k_elems,
                         std::vector<float>* hi, std::vector<float>* lo) {
  const int c_blocks = (I + k_elems - 1) / k_elems;
  const size_t cpad = static_cast<size_t>(c_blocks) * k_elems;
  const size_t k_total = static_cast<size_t>(KH) * KW * cpad;
  hi->assign(static_cast<size_t>(O) * k_total, 0.0f);
  if (lo != nullptr) lo->assign(kind == GEMM_TF32X3 ? hi->size() : 0, 0.0f);
  for (int o = 0; o < O; ++o)
    for (int i = 0; i < I; ++i)
      for (int kh = 0; kh < KH; ++kh)
        for (int kw = 0; kw < KW; ++kw) {
          const float v = w[((static_cast<size_t>(o) * I + i) * KH + kh) * KW + kw];
          const size_t dst = o * k_total + (static_cast<size_t>(kh) * KW + kw) * cpad + i;
          const float h = tf32_round_host(v);
          (*hi)[dst] = h;
          if (kind == GEMM_TF32X3 && lo != nullptr) (*lo)[dst] = v - h;
        }
}

uint16_t bf16_round_host(float x) {
  // round to nearest even onto 7 explicit mantissa bits; NaN stays NaN
  uint32_t u;
  std::memcpy(&u, &x, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return static_cast<uint16_t>((u >> 16) | ((u & 0xffffu) ? 0x40u : 0u));
  u += 0x7fffu + ((u >> 16) & 1u);
  return static_cast<uint16_t>(u >> 16);
}

float bf16_to_float_host(uint16_t h) {
  const uint32_t u = static_cast<uint32_t>(h) << 16;
  float r;
  std::memcpy(&r, &u, 4);
  return r;
}

void tc_pack_weights_bf16x2(const float* w, int O, int I, int KH, int KW, int k_elems,
                            std::vector<uint16_t>* hi, std::vector<uint16_t>* mid) {
  const int c_blocks = (I + k_elems - 1) / k_elems;
  const size_t cpad = static_cast<size_t>(c_blocks) * k_elems;
  const size_t k_total = static_cast<size_t>(KH) * KW * cpad;
  hi->assign(static_cast<size_t>(O) * k_total, 0);
  mid->assign(hi->size(), 0);
  for (int o = 0; o < O; ++o)
    for (int i = 0; i < I; ++i)
      for (int kh = 0; kh < KH; ++kh)
        for (int kw = 0; kw < KW; ++kw) {
          const float v = w[((static_cast<size_t>(o) * I + i) * KH + kh) * KW + kw];
          const size_t dst = o * k_total + (static_cast<size_t>(kh) * KW + kw) * cpad + i;
          const uint16_t h = bf16_round_host(v);
          (*hi)[dst] = h;
          (*mid)[dst] = bf16_round_host(v - bf16_to_float_host(h));
        }
}

void tc_pack_weights_i8(const int8_t* w, int O, int I, int KH, int KW, int k_elems,
                        std::vector<int8_t>* packed) {
  const int c_blocks = (I + k_elems - 1) / k_elems;
  const size_t cpad = static_cast<size_t>(c_blocks) * k_elems;
  const size_t k_total = static_cast<size_t>(KH) * KW * cpad;
  packed->assign(static_cast<size_t>(O) * k_total, 0);
  for (int o = 0; o < O; ++o)
    for (int i = 0; i < I; ++i)
      for (int kh = 0; kh < KH; ++kh)
        for (int kw = 0; kw < KW; ++kw)
          (*packed)[o * k_total + (static_cast<size_t>(kh) * KW + kw) * cpad + i] =
              w[((static_cast<size_t>(o) * I + i) * KH + kh) * KW + kw];
}

// ------------------------------------------------------------------------------ stem kernel
std::string tc_plan_stem(TcStemLaunch* L, const TcStemConv& c, const TcEpilogue& e, int sm_count) {
  load_driver_entry_points();
  if (!g_driver_error.empty()) return g_driver_error;
  TcStemParams& p = L->p;
  const int N = c.out_channels;
  if (c.row_bytes % 128 != 0 || c.row_bytes / 128 > 256) return "padded input rows must be multiples of 128 bytes";
  if (c.OW > kTcBlockM || c.OW < 1) return "an output row must fit one 128-row tile";
  if (N % 16 != 0 || N > 128) return "output channels must be a multiple of 16, at most 128";
  if (c.KH < 1 || c.KH > 16) return "filter height out of range";
  if (e.res0 != nullptr) return "the stem kernel takes no residual";
  const bool i8 = c.kind == GEMM_I8;
  if (c.kind != GEMM_BF16X3 && !i8) return "the stem kernel takes bf16-pair or int8 operands";
  const bool i8_out = e.out_mode == OUT_I8;
  if (e.out_mode != OUT_F32 && !(e.out_mode == OUT_BF16X2 && !i8) && !(i8_out && i8))
    return "output format not handled by the stem kernel";
  const bool bf16_out = e.out_mode == OUT_BF16X2;
  if (e.ldo != N || (reinterpret_cast<uintptr_t>(e.out0) & 15) != 0 || (reinterpret_cast<uintptr_t>(e.out1) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(e.outq) & 15) != 0)
    return "the stem kernel writes dense, 16-byte aligned rows";
  const int planes = i8 ? 1 : 2;
  L->kind = c.kind;
  if ((c.OW - 1) * 16 + 64 > c.row_bytes) return "padded rows are shorter than the last window";
  p.tiles = c.images * c.OH;
  p.OH = c.OH;
  p.OW = c.OW;
  p.KH = c.KH;
  p.stride_h = c.stride_h;
  p.pad_t = c.pad_t;
  p.N = N;
  p.M = c.images * c.OH * c.OW;
  p.row_bytes = c.row_bytes;
  // the last filter row's windows of tile rows up to 127 reach 127*16 + 64 bytes into (and past) it
  p.a_plane_bytes = ((c.KH - 1) * c.row_bytes + (kTcBlockM - 1) * 16 + 64 + 1023) / 1024 * 1024;
  p.a_plane_bytes = std::max(p.a_plane_bytes, (c.KH * c.row_bytes + 1023) / 1024 * 1024);
  p.b_slot = (N * 64 + 1023) / 1024 * 1024;
  p.bias = e.bias;
  p.scale = e.scale;
  p.out_scale = e.out_scale;
  p.out_mode = e.out_mode;
  p.act = e.act;
  p.act_a = e.act_a;
  p.act_b = e.act_b;
  p.status = e.status;
  p.out0 = e.out0;
  p.out1 = e.out1;
  p.outq = e.outq;
  if (!direct_rows(c.kind, e, N, &p.wide)) return "the stem kernel writes rows of 16-byte pieces";
  const int budget = kTcSmemBudget;
  const int weights = c.KH * planes * p.b_slot;
  const int stage = planes * p.a_plane_bytes;
  // (a stage holds a whole tile's input: two are a double buffer)
  p.stages = std::min(kStemMaxStages, (budget - weights - kDrainBytes) / stage);
  if (p.stages < 2) return "shared memory cannot hold the weights and two row stages";
  // the epilogue of a 64-channel row takes longer than its 42 MMAs: two epilogue groups on alternate tiles
  p.epi_groups = p.tiles < 2 * sm_count ? 1 : 2;
  // four accumulators of 64 columns where they fit, and then a second MMA-issuing warp for alternate tiles
  p.accs = N <= 64 ? 4 : 2;
  p.issuers = p.accs == 4 && env_int("NCNN_B200_STEM_ISSUERS", 2) >= 2 ? 2 : 1;
  L->smem_bytes = weights + p.stages * stage + kDrainBytes + 1024;
  L->smem_bytes = std::max(L->smem_bytes, 120 * 1024);  // one CTA per SM: each allocates tensor memory
  L->grid = std::min(p.tiles, sm_count);
  // input planes: [images][H][row_bytes / 128][64 bf16], KH whole rows per copy, dense in shared memory
  auto rows_map = [&](CUtensorMap* map, const void* base) -> std::string {
    const cuuint64_t line = i8 ? 128 : 64;  // elements per 128-byte line
    const cuuint64_t dims[4] = {line, static_cast<cuuint64_t>(c.row_bytes / 128), static_cast<cuuint64_t>(c.H),
                                static_cast<cuuint64_t>(c.images)};
    const cuuint64_t strides[3] = {128, static_cast<cuuint64_t>(c.row_bytes),
                                   static_cast<cuuint64_t>(c.row_bytes) * c.H};
    const cuuint32_t box[4] = {static_cast<cuuint32_t>(line), static_cast<cuuint32_t>(c.row_bytes / 128),
                               static_cast<cuuint32_t>(c.KH), 1};
    const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
    const CUresult r = g_encode_tiled(map, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4,
                                      const_cast<void*>(base), dims, strides, box, elem_strides,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return "cuTensorMapEncodeTiled failed for the stem input rows with code " + std::to_string(static_cast<int>(r));
    return {};
  };
  std::string err = rows_map(&L->map_a0, c.in0);
  if (err.empty() && !i8) err = rows_map(&L->map_a1, c.in1);
  if (!err.empty()) return err;
  const uint64_t window = i8 ? 64 : 32;  // elements of one 64-byte window
  const uint64_t k_total = static_cast<uint64_t>(c.KH) * window;
  err = encode_tiled_2d(&L->map_b0, c.kind, c.w0, k_total, N, k_total * (i8 ? 1 : 2), static_cast<uint32_t>(window), N, 64);
  if (err.empty() && !i8)
    err = encode_tiled_2d(&L->map_b1, c.kind, c.w1, k_total, N, k_total * 2, static_cast<uint32_t>(window), N, 64);
  if (!err.empty()) return err;
  return err;
}

cudaError_t tc_launch_stem(const TcStemLaunch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, kStemThreads, L.smem_bytes, false, stream);
  auto launch = [&](auto kind) {
    constexpr int KIND = decltype(kind)::value;
    return with_form<KIND, false>(L.p.out_mode, false, [&](auto form) {
      if constexpr (decltype(form)::value % 2 == 1) return cudaErrorInvalidValue;  // (a stem has no residual)
      else return launch_opted(tc_stem_kernel<KIND, decltype(form)::value>, kTcSmemBudget + 1024, lc, L.p, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
    });
  };
  const cudaError_t e = L.kind == GEMM_I8 ? launch(std::integral_constant<int, GEMM_I8>{}) : launch(std::integral_constant<int, GEMM_BF16X3>{});
  return e != cudaSuccess ? e : cudaGetLastError();
}

constexpr int kStemPoolMaxSmem = 218 * 1024;  // dynamic shared memory the stem + pooling kernel may ask for

std::string tc_plan_stem_pool(TcStemPoolLaunch* L, const TcStemConv& c, const TcEpilogue& e_in, int pooled_h, int pooled_w, int sm_count) {
  const bool i8 = c.kind == GEMM_I8;
  if (!(c.kind == GEMM_BF16X3 && e_in.out_mode == OUT_BF16X2) && !(i8 && e_in.out_mode == OUT_F32))
    return "the stem + pooling kernel writes bf16 pairs from bf16 pairs, or fp32 from int8";
  const int N = c.out_channels;
  if (N != 32 && N != 64) return "the stem + pooling kernel takes 32 or 64 output channels";
  if (e_in.act != ACT_NONE && e_in.act != ACT_RELU && e_in.act != ACT_CLIP) return "the stem + pooling kernel applies no activation but ReLU and clip";
  if (c.OH != 2 * pooled_h || c.OW != 2 * pooled_w || pooled_h < 1 || pooled_w < 1) return "the pooled extent must be half the convolution's";
  if (e_in.side_count > 1 || (e_in.side_count == 1 && (!i8 || N != 64))) return "one int8 copy of 64 channels at most";
  // the convolution part is planned as for tc_stem_kernel (validation, input and weight maps, operand geometry);
  // the int8 copy belongs to the pooled tensor
  TcEpilogue e = e_in;
  e.side_count = 0;
  TcStemLaunch conv;
  std::string err = tc_plan_stem(&conv, c, e, sm_count);
  if (!err.empty()) return err;
  const int planes = i8 ? 1 : 2;
  TcStemPoolParams& pp = L->pp;
  pp.s = conv.p;
  pp.images = c.images;
  pp.POH = pooled_h;
  pp.POW = pooled_w;
  pp.ring_row_bytes = (c.OW * N * 4 + 1023) / 1024 * 1024;
  pp.side_q = e_in.side_count ? e_in.side_q[0] : nullptr;
  pp.side_scale = e_in.side_count ? e_in.side_scale[0] : 0.0f;
  const int weights = c.KH * planes * conv.p.b_slot;
  const int stage = planes * conv.p.a_plane_bytes;
  const int fixed = weights + pp.ring_row_bytes + 1024;
  pp.row_stages = fixed + 4 * stage <= kStemPoolMaxSmem ? 4 : 2;
  L->smem_bytes = fixed + pp.row_stages * stage;
  if (L->smem_bytes > kStemPoolMaxSmem) return "shared memory cannot hold the weights, two row stages and a result row";
  L->smem_bytes = std::max(L->smem_bytes, 120 * 1024);  // one CTA per SM: each allocates tensor memory
  const long long pooled_rows = static_cast<long long>(c.images) * pooled_h;
  if (pooled_rows * pooled_w > 0x7fffffffll) return "too many pooled pixels for one launch";
  L->grid = static_cast<int>(std::min<long long>(pooled_rows, sm_count));
  L->kind = c.kind;
  L->map_a0 = conv.map_a0;
  L->map_a1 = conv.map_a1;
  L->map_b0 = conv.map_b0;
  L->map_b1 = conv.map_b1;
  return {};
}

cudaError_t tc_launch_stem_pool(const TcStemPoolLaunch& L, cudaStream_t stream) {
  KernelLaunchConfig lc(L.grid, kStemPoolThreads, L.smem_bytes, false, stream);
  const cudaError_t e = L.kind == GEMM_I8 ? launch_opted(tc_stem_pool_kernel<GEMM_I8>, kStemPoolMaxSmem, lc, L.pp, L.map_a0, L.map_a1, L.map_b0, L.map_b1)
                                          : launch_opted(tc_stem_pool_kernel<GEMM_BF16X3>, kStemPoolMaxSmem, lc, L.pp, L.map_a0, L.map_a1, L.map_b0, L.map_b1);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace nb
