// Host-side planning for the tensor-core contraction kernel: encodes the TMA
// tensor maps, picks the tile shape and stage count, and launches.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>

#include "tc_conv_halo.cuh"
#include "tc_conv_i8.cuh"
#include "tc_conv_patch.cuh"
#include "tc_dw_project.cuh"
#include "tc_gemm.cuh"
#include "tc_gemm2.cuh"
#include "tc_stem.cuh"
#include "tc_stem_pool.cuh"

namespace nb {

struct TcLaunch {
  TcGemmParams p{};
  alignas(64) CUtensorMap map_a0{};
  alignas(64) CUtensorMap map_a1{};
  alignas(64) CUtensorMap map_b0{};
  alignas(64) CUtensorMap map_b1{};
  int kind = GEMM_TF32;
  int grid = 0;
  int smem_bytes = 0;
  int cta2 = 0;  // CTAs per worker of tc_gemm2_kernel: 2 = CTA pairs, 1 = single CTAs with split tiles, 0 = tc_gemm_kernel
};

// Activation tensor as TMA sees it for an im2col load, innermost dimension first:
// channels, width, height, images.  For an ordinary NHWC tensor the strides are the
// dense ones; the 7x7 stem uses an overlapping-window view of a channel-padded image.
struct TcIm2colView {
  const void* plane0 = nullptr;
  const void* plane1 = nullptr;  // lo plane (GEMM_TF32X3 only)
  uint64_t C = 0, W = 0, H = 0, N = 0;
  uint64_t stride_w = 0, stride_h = 0, stride_n = 0;  // bytes
  int KH = 1, KW = 1;
  int stride_conv_h = 1, stride_conv_w = 1;
  int pad_t = 0, pad_l = 0;
  int dil_h = 1, dil_w = 1;
  int OH = 0, OW = 0;
};

struct TcEpilogue {
  const float* bias = nullptr;
  const float* scale = nullptr;
  float* out0 = nullptr;
  float* out1 = nullptr;
  int8_t* outq = nullptr;
  const float* res0 = nullptr;
  const float* res1 = nullptr;
  bool res_bf16 = false;  // the residual planes hold bf16 pairs (hi, mid)
  long long ldo = 0;
  int out_mode = OUT_F32;
  int act = ACT_NONE;
  float act_a = 0.0f, act_b = 0.0f;
  float out_scale = 1.0f;
  int* status = nullptr;
  long long* trace = nullptr;
  // int8 copies of an fp32 result, quantised with side_scale[i] (out_mode OUT_F32, channels a multiple of 16)
  int side_count = 0;
  int8_t* side_q[2] = {nullptr, nullptr};
  float side_scale[2] = {0.0f, 0.0f};
  // workspace for tiles split between CTA pairs (tc_gemm2.cuh): partial accumulators and one flag
  // word per CTA, zero before the first launch; without it tiles are never split
  uint32_t* sk_ws = nullptr;
  size_t sk_ws_bytes = 0;
  int* sk_flags = nullptr;
  int sk_flag_count = 0;
};

// bytes of partial-accumulator workspace and flag words that let every layer split tiles
constexpr size_t kTcSplitWorkspaceBytes = 160ull * kTcBlockM * kTc2MaxBlockN * 4;
constexpr int kTcSplitFlagCount = 640;  // two per CTA (one per epilogue group)
// words that are there: k_rows_f32 counts the finished chunks of every 32 columns (conv_f32.cuh)
constexpr int kTcFlagWords = 16384;

// Elements per K block for a kind and a channel count; 0 when the tensor-core
// path cannot address that channel count (rows must be multiples of 16 bytes).
int tc_k_elems(int kind, int channels);
int tc_row_bytes(int kind, int channels);

// bf16-pair convolutions of at least kTcChunkFrom K blocks are summed in chunks of kTcChunkBlocks: where a batch leaves SMs
// idle, the chunks of a tile run side by side, and where it does not, one CTA adds up the same chunks, so that results do
// not depend on the batch.  Both count K blocks of either width: in a row a block of 64 channels of a filter tap costs the
// chain ~0.57 us, one of 32 channels (channel counts that are no multiple of 64) ~0.45.  3x3 layers, whole -> in chunks, us:
//   blocks       7x7, 1 image     16 images       64 images        14x14, 64 images
//   36 of 64     25.5 -> 19.7     25.4 -> 21.4    27.5 -> 28.2     47.7 -> 52.1 (gives up its paired tiles)
//   45           29.0 -> 19.4     29.7 -> 23.5    32.8 -> 33.5     58.4 -> 64.5 (the same)
//   54           33.2 -> 21.0     33.8 -> 25.6    38.4 -> 39.6     86.8 -> 95.2 (both on CTA pairs)
//   63           36.8 -> 21.4     40.6 -> 30.5    44.4 -> 45.8    113.7 -> 121 (whole on pairs, chunks on one CTA)
//   72           41.2 -> 21.4     42.0 -> 33.7    51.2 -> 52.1    142.4 -> 145 (the same; 192 images of 7x7, both on pairs: 83 -> 93)
//   63 of 32     29.0 -> 16.7     29.2 -> 25.0    32.2 -> 32.0     61.5 -> 61.8
//   81           34.5 -> 18.6     35.0 -> 28.8    39.4 -> 39.6     79.8 -> 79.9
// Whole batches lose the same few per cent at every depth, so there is no crossover to draw the line at.  It lies at four
// chunks: one image then takes about half its time, with three two thirds and with two four fifths.
constexpr int kTcChunkBlocks = 18, kTcChunkFrom = 3 * kTcChunkBlocks + 1;

// Convolution: M = view.N*OH*OW pixels, N = out_channels.  `w0`/`w1` are the packed
// weights [out_channels][KH*KW*c_blocks*k_elems] (see tc_pack_weights).
// Returns an empty string on success, else the reason.
std::string tc_plan_conv(TcLaunch* launch, int kind, const TcIm2colView& view, const void* w0,
                         const void* w1, int out_channels, const TcEpilogue& epilogue,
                         int sm_count);
// The two halves of it: whether and how tc_gemm_kernel or tc_gemm2_kernel would run the layer, which other kernels are
// compared with, and the tensor maps, which only the kernel that runs needs.
std::string tc_plan_conv_tiles(TcLaunch* launch, int kind, const TcIm2colView& view, int out_channels, const TcEpilogue& epilogue, int sm_count);
std::string tc_encode_conv(TcLaunch* launch, int kind, const TcIm2colView& view, const void* w0, const void* w1, int out_channels);

// Plain GEMM: A is [M][K] row-major with row stride lda elements (planes a0/a1),
// weights packed [N][Kpad].
std::string tc_plan_gemm(TcLaunch* launch, int kind, const void* a0, const void* a1, long long M,
                         int K, long long lda, const void* w0, const void* w1, int N,
                         const TcEpilogue& epilogue, int sm_count);

cudaError_t tc_launch(const TcLaunch& launch, cudaStream_t stream);

// NCNN_B200_PDL=0 launches every kernel fully serialised behind its predecessor.
bool tc_pdl_enabled();

// Packs [O][I][KH][KW] (ncnn order) weights into [O][KH*KW][c_blocks*k_elems] with
// zero padding, channel innermost.  For fp32 kinds `hi` receives the values
// rounded to tf32 (GEMM_TF32, GEMM_TF32X3) and `lo` the remainders (GEMM_TF32X3).
void tc_pack_weights_f32(int kind, const float* w, int O, int I, int KH, int KW, int k_elems,
                         std::vector<float>* hi, std::vector<float>* lo);
void tc_pack_weights_i8(const int8_t* w, int O, int I, int KH, int KW, int k_elems,
                        std::vector<int8_t>* packed);

// GEMM_BF16X3: two bf16 planes, hi = bf16(w) and mid = bf16(w - hi), same layout.
void tc_pack_weights_bf16x2(const float* w, int O, int I, int KH, int KW, int k_elems,
                            std::vector<uint16_t>* hi, std::vector<uint16_t>* mid);

float tf32_round_host(float x);
uint16_t bf16_round_host(float x);
float bf16_to_float_host(uint16_t h);

// ---- stride-1 convolution with the input patch resident in shared memory (tc_conv_halo.cuh)
struct TcHaloLaunch {
  TcHaloParams p{};
  alignas(64) CUtensorMap map_a0{};
  alignas(64) CUtensorMap map_a1{};
  alignas(64) CUtensorMap map_b0{};
  alignas(64) CUtensorMap map_b1{};
  int kind = GEMM_TF32;
  int grid = 0;
  int smem_bytes = 0;
  int pair = 0;  // 1: two pixel tiles per cluster of two CTAs (grid counts CTAs)
};

struct TcHaloConv {
  const void* in0 = nullptr;  // NHWC activation planes
  const void* in1 = nullptr;
  int images = 0, H = 0, W = 0, C = 0;
  int KH = 1, KW = 1, pad_t = 0, pad_l = 0, OH = 0, OW = 0;
  const void* w0 = nullptr;  // packed like tc_plan_conv's weights
  const void* w1 = nullptr;
  int out_channels = 0;
};

// True when the patch-resident kernel applies and is expected to win: fp32 kind, stride and
// dilation 1, channels in blocks of 32, output rows of 16 bytes, tiles mostly inside the image.
bool tc_halo_applies(int kind, int C, int KH, int KW, int stride_h, int stride_w, int dil_h, int dil_w, int OH,
                     int OW, int out_channels, int out_mode);
// `pair`: plan the form that runs two pixel tiles on a cluster of two CTAs (tiles up to 256 channels wide)
std::string tc_plan_conv_halo(TcHaloLaunch* launch, int kind, const TcHaloConv& conv, const TcEpilogue& epilogue,
                              int sm_count, bool pair = false);
cudaError_t tc_launch_halo(const TcHaloLaunch& launch, cudaStream_t stream);

// ---- convolution of few pixels out of input patches (tc_conv_patch.cuh)
struct TcPatchLaunch {
  TcPatchParams p{};
  alignas(64) CUtensorMap map_a0{};
  alignas(64) CUtensorMap map_a1{};
  alignas(64) CUtensorMap map_b0{};
  alignas(64) CUtensorMap map_b1{};
  int kind = GEMM_BF16X3;
  int grid = 0;
  int smem_bytes = 0;
};
// Plans the convolution of tc_plan_conv's arguments on tc_conv_patch_kernel, in the tile shape that is expected to take
// the least time.  Returns the reason where the kernel does not apply (bf16 pairs, stride 1 or 2, no dilation), or, unless
// `always`, where `gemm`, the same layer's plan on the other kernels, is expected to be about as fast.
std::string tc_plan_conv_patch(TcPatchLaunch* launch, int kind, const TcIm2colView& view, const void* w0, const void* w1,
                               int out_channels, const TcEpilogue& epilogue, int sm_count, const TcLaunch& gemm, bool always);
cudaError_t tc_launch_patch(const TcPatchLaunch& launch, cudaStream_t stream);

// ---- int8 convolution with its filter resident in shared memory (tc_conv_i8.cuh)
struct TcConvI8Launch {
  TcConvI8Params p{};
  alignas(64) CUtensorMap map_a{};
  alignas(64) CUtensorMap map_b{};
  int out_mode = OUT_I8;
  int grid = 0;
  int threads = 0;
  int smem_bytes = 0;
};
// Plans the convolution of tc_plan_conv's arguments on tc_conv_i8_kernel.  Returns the reason where the kernel does not apply
// (stride and dilation 1, more than 32 channels, a filter that fits shared memory), or, unless `always`, where the other
// kernels are expected to be as fast.
std::string tc_plan_conv_i8(TcConvI8Launch* launch, const TcIm2colView& view, const void* w, int out_channels,
                            const TcEpilogue& epilogue, int sm_count, bool always);
cudaError_t tc_launch_conv_i8(const TcConvI8Launch& launch, cudaStream_t stream);

// ---- 3x3 depthwise convolution fused into the following 1x1 convolution (tc_dw_project.cuh)
struct TcDwProjLaunch {
  TcDwProjParams p{};
  alignas(64) CUtensorMap map_x{};   // fp32 depthwise input, patches of 18 x 10 pixels x 32 channels (expand fused in: bf16 hi plane of the block's input)
  alignas(64) CUtensorMap map_x1{};  // expand fused in: bf16 mid plane of the block's input
  alignas(64) CUtensorMap map_e0{};  // expand weights, bf16 hi / mid planes
  alignas(64) CUtensorMap map_e1{};
  alignas(64) CUtensorMap map_b0{};  // projection weights, bf16 hi / mid planes
  alignas(64) CUtensorMap map_b1{};
  int grid = 0;
  int smem_bytes = 0;
  int stride = 1;
  bool expand = false;
};

struct TcDwProjConv {
  const void* x = nullptr;   // NHWC input: plain fp32 of the depthwise layer, or (expand fused in) the bf16 hi plane of the expand layer's
  const void* x1 = nullptr;  // expand fused in: the bf16 mid plane
  int images = 0, H = 0, W = 0, C = 0;  // depthwise output extent, depthwise channels
  int Hin = 0, Win = 0;                 // depthwise input extent
  int stride = 1;
  int pad_t = 1, pad_l = 1;
  // expand layer fused in (ex_w0 != nullptr): 1x1 convolution Cin -> C on bf16 pairs, Cin <= 32
  int Cin = 0;
  const void* ex_w0 = nullptr;        // packed [C][32] bf16 hi / mid
  const void* ex_w1 = nullptr;
  const float* ex_bias = nullptr;     // [C] or null
  int ex_act = ACT_NONE;
  float ex_act_a = 0.0f, ex_act_b = 0.0f;
  const float* dw_weights = nullptr;  // [9][C]
  const float* dw_bias = nullptr;
  int dw_act = ACT_NONE;
  float dw_act_a = 0.0f, dw_act_b = 0.0f;
  const void* w0 = nullptr;  // projection weights packed [N][ceil(C/32)*32] bf16 hi / mid
  const void* w1 = nullptr;
  int out_channels = 0;
};

// True when the fused kernel takes the pair of layers: 3x3, stride 1, dilation 1, output extent equal to the
// input's, channels in fours; projection 1x1 stride 1 with bf16-pair operands.
bool tc_dw_project_applies(int C, int N, int H, int W, int out_mode, bool has_res, bool res_bf16);
// True when the whole inverted-residual block (1x1 expand Cin -> C with at most 32 input channels, 3x3 depthwise of
// stride 1 or 2 with output OH x OW, 1x1 projection C -> N) fits the fused kernel, whatever formats its output and
// residual get.
bool tc_block_applies(int Cin, int C, int N, int OH, int OW, int stride, bool has_res);
// True when such a block has more weights than shared memory keeps and brings them in for every tile.
bool tc_block_streams(int Cin, int C, int N, int stride);
std::string tc_plan_dw_project(TcDwProjLaunch* launch, const TcDwProjConv& conv, const TcEpilogue& epilogue, int sm_count);
cudaError_t tc_launch_dw_project(const TcDwProjLaunch& launch, cudaStream_t stream);

// ---- stem convolution with the input rows resident in shared memory (tc_stem.cuh)
struct TcStemLaunch {
  TcStemParams p{};
  alignas(64) CUtensorMap map_a0{};
  alignas(64) CUtensorMap map_a1{};
  alignas(64) CUtensorMap map_b0{};
  alignas(64) CUtensorMap map_b1{};
  int kind = GEMM_BF16X3;
  int grid = 0;
  int smem_bytes = 0;
};

struct TcStemConv {
  int kind = GEMM_BF16X3;     // GEMM_BF16X3 (4-channel pixels, bf16 hi/mid planes) or GEMM_I8 (8-channel int8 pixels)
  const void* in0 = nullptr;  // [images][H][row_bytes]: padded rows of 8-byte pixels (bf16 hi plane, or int8)
  const void* in1 = nullptr;  // bf16 mid plane
  int images = 0, H = 0;
  int row_bytes = 0;          // bytes of one padded row (a multiple of 128)
  int KH = 1, stride_h = 1, pad_t = 0, OH = 0, OW = 0;
  const void* w0 = nullptr;   // packed [O][KH][32] bf16 hi / mid, or [O][KH][64] int8 (one 64-byte window per filter row)
  const void* w1 = nullptr;
  int out_channels = 0;
};

// ---- stem convolution + 3x3 stride-2 max pooling in one kernel (tc_stem_pool.cuh)
struct TcStemPoolLaunch {
  TcStemPoolParams pp{};
  alignas(64) CUtensorMap map_a0{};
  alignas(64) CUtensorMap map_a1{};
  alignas(64) CUtensorMap map_b0{};
  alignas(64) CUtensorMap map_b1{};
  int grid = 0;
  int smem_bytes = 0;
  int kind = GEMM_BF16X3;
};
// `epilogue` describes the POOLED tensor (dense rows of out_channels: bf16 pairs behind a bf16-pair stem, fp32 with at
// most one int8 copy behind an int8 stem); pooled extent pooled_h x pooled_w = half the convolution's output extent
// (3x3 windows, stride 2, one pixel of padding above and to the left).
std::string tc_plan_stem_pool(TcStemPoolLaunch* launch, const struct TcStemConv& conv, const TcEpilogue& epilogue, int pooled_h,
                              int pooled_w, int sm_count);
cudaError_t tc_launch_stem_pool(const TcStemPoolLaunch& launch, cudaStream_t stream);

// Applies when output pixels are 16 bytes apart in the padded input row (stride 2 x 4 channels x
// bf16), a row of output fits one 128-row tile, and the rows and resident weights fit shared memory.
std::string tc_plan_stem(TcStemLaunch* launch, const TcStemConv& conv, const TcEpilogue& epilogue, int sm_count);
cudaError_t tc_launch_stem(const TcStemLaunch& launch, cudaStream_t stream);

}  // namespace nb
