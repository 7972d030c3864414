// The second half, or the whole, of an inverted-residual block in one kernel:
//   [1x1 "expand" convolution + activation ->] 3x3 depthwise convolution + activation -> 1x1 "projection"
//   convolution (+ bias, residual, activation).
//
// Run one after the other these layers write the widest tensors of the network to HBM and read them back, on
// layers that are bound by HBM either way.  Here the expanded tensor and the depthwise result never leave the
// SM.  A tile is a rectangle of output pixels of one image (16 x 8 at stride 1, 8 x 8 at stride 2: up to 128
// rows of the projection's GEMM); per block of 32 (expanded) channels
//   * the fp32 input patch of the depthwise filter ((TH-1)*stride+3 rows x (TW-1)*stride+3 columns x 32 channels)
//     arrives in shared memory: loaded by TMA (coordinates outside the image read as zero: that is the padding),
//     or, with the expand layer fused in (EXPAND), computed on the tensor cores from the block's input patch
//     (<= 32 channels, bf16 pairs, loaded once per tile): the MMA thread multiplies the patch (two or three
//     128-pixel strips) by the block's 32 weight rows into a TMEM accumulator of the depthwise group, two blocks
//     ahead of the group; the group's warps read it back (tcgen05.ld), add the bias, apply the activation, write
//     zero where the pixel lies outside the image, and store the fp32 patch,
//   * four CUDA-core warps (two such groups take alternate blocks) compute the depthwise results from it with
//     the arithmetic of the stand-alone kernel (bias, nine fmaf in filter order, activation), split each value
//     into its bf16 pair (hi = bf16(x), mid = bf16(x - hi)) and write both planes straight into the K-major,
//     64-byte-swizzled operand tile that tcgen05.mma reads,
//   * one thread issues the projection's MMAs (mid*hi + hi*mid + hi*hi, as tc_gemm_kernel does) against
//     that channel block's weights, which TMA streams through a small ring,
// and the usual epilogue warps drain the accumulator (bias, residual, activation).
// Without EXPAND the operands, their order and the accumulation are those of the two separate kernels, so the
// results are the same bits.  With EXPAND the expand layer's products are the same too; only its bias is added
// after the accumulation instead of by the epilogue of a separate kernel, which is the same fp32 addition.
//
// Warps (640 threads): 0 TMA producer, 1 MMA issuer, 4-11 epilogue (two groups on alternate tiles), 12-19 depthwise; registers
// are split between the roles.  Every wait is bounded and ends in the status word.
//
// What bounds it: the depthwise warps' instructions, which wait on one another (shared memory -> FMA -> clamp -> split ->
// shared memory), ~2 200 clocks per 32 channels of a stride-2 tile for both groups together.  What counts is how few
// instructions a result takes: a thread owns two channels (packed FMAs) and a square of results, every address is a
// constant away from one base, the expand bias is read before the strips instead of between their stores, and tiles are
// walked by adding with carry.  256 images of MobileNetV2, before (four channels x 8 rows a thread) -> now: 112x112x32 stride 1
// 198 -> 159 us, whole blocks 112x112x96 stride 2 440 -> 290, 56x56x144 stride 2 257 -> 184, stride 1 546 -> 289.
// Sixteen depthwise warps with half the results each were no faster than eight of the old form: each warp adds its own
// waits, addresses and clamps.
#pragma once

#include "tc_gemm.cuh"

namespace nb {

constexpr int kDwpThreads = 640;
// registers a thread: at launch, of the issuing warpgroup, of the two epilogue groups and of the two depthwise groups
constexpr int kDwpRegs = 96, kDwpIssueRegs = 56, kDwpDrainRegs = 96, kDwpFilterRegs = 112;
static_assert(kDwpIssueRegs + 2 * kDwpDrainRegs + 2 * kDwpFilterRegs <= 5 * kDwpRegs, "what the launch gives the block");
constexpr int kDwpChannels = 32;  // channels per block: 64-byte bf16 rows
constexpr int kDwpTileW = 8;
constexpr int kDwpMaxStages = 4;
constexpr int kDwpMaxPatches = 4;

// geometry of a tile by stride
__host__ __device__ constexpr int dwp_tile_h(int stride) { return stride == 1 ? 16 : 8; }
__host__ __device__ constexpr int dwp_patch_h(int stride) { return (dwp_tile_h(stride) - 1) * stride + 3; }
__host__ __device__ constexpr int dwp_patch_w(int stride) { return (kDwpTileW - 1) * stride + 3; }
__host__ __device__ constexpr int dwp_patch_pixels(int stride) { return dwp_patch_h(stride) * dwp_patch_w(stride); }
// bytes from one pixel of the fp32 patch to the next: dense where TMA writes it; with the expand layer inside 16 more, which
// spreads the 32 pixels that a warp stores at a time over the banks and leaves every address a constant away from the first
__host__ __device__ constexpr int dwp_patch_pitch(bool expand) { return kDwpChannels * 4 + (expand ? 16 : 0); }
__host__ __device__ constexpr int dwp_patch_bytes(int stride, bool expand) {
  return (dwp_patch_pixels(stride) * dwp_patch_pitch(expand) + 1023) / 1024 * 1024;
}
// columns of the tile that a depthwise thread computes (times four rows)
__host__ __device__ constexpr int dwp_cols(int stride) { return stride == 1 ? 4 : 2; }
// epilogue warps that have rows to drain: 32 rows each, two groups
__host__ __device__ constexpr int dwp_drain_warps(int stride) { return 2 * dwp_tile_h(stride) * kDwpTileW / 32; }
// one bf16 plane of the operand tile: the rows a tile has, 64 bytes each (the MMA reads 128 rows: past a
// stride-2 tile's 64 it reads what follows in shared memory, into accumulator rows that are never stored)
__host__ __device__ constexpr int dwp_a_plane_bytes(int stride) { return dwp_tile_h(stride) * kDwpTileW * 64; }

struct TcDwProjParams {
  int images, H, W, C;  // depthwise OUTPUT extent, channels of the depthwise layer
  int Hin, Win;         // depthwise input extent (= H, W at stride 1)
  int N;                // projection output channels
  int tiles_y, tiles_x, tiles_n, block_n;
  int c_blocks;         // blocks of 32 channels (the last one may be partly past C: zero-filled)
  int pad_t, pad_l;
  int stages;           // weight ring depth
  int patch_bufs;       // input patch ring depth, 2 or 4 (even: a slot then always serves the same depthwise group)
  int b_bytes;          // one plane of a weight stage, rounded to 1 KB
  int wide;             // rows of result and residual are multiples of 32 bytes, 32-byte aligned
  const float* dw_weights;  // [9][C], tap-major
  const float* dw_bias;     // [C] or null
  int dw_act;
  float dw_act_a, dw_act_b;
  // expand layer (EXPAND): x is [image][Hin][Win][Cin] as bf16 hi / mid planes, weights packed [C][32] bf16 hi / mid
  int Cin;
  int x_row_bytes;          // operand rows of the input patch and of the expand weights: 64 bytes (32 channels), or 32
                            // (16 channels) when the block's input has no more: two patch buffers then fit where one did
  int x_plane_bytes;        // one bf16 plane of an input patch buffer, rounded to 1 KB
  int x_bufs;               // input patch buffers: 2, or 1 when two do not fit
  int ex_ksteps;            // K steps of 16 input channels the expand MMAs run: ceil(Cin / 16)
  const float* ex_bias;     // [C] or null
  int ex_act;
  float ex_act_a, ex_act_b;
  const float* bias;        // projection bias [N] or null
  int res_mode, out_mode, act;
  float act_a, act_b;
  float* out0;
  float* out1;
  const float* res0;
  const float* res1;
  int* status;
};

// (KIND: the projection's arithmetic; bf16 pairs are the only form built)
template <int KIND, int STRIDE, bool EXPAND, int EPI>
__global__ void __launch_bounds__(kDwpThreads, 1)
tc_dw_project_kernel(const __grid_constant__ TcDwProjParams p, const __grid_constant__ CUtensorMap map_x,
                     const __grid_constant__ CUtensorMap map_x1, const __grid_constant__ CUtensorMap map_e0,
                     const __grid_constant__ CUtensorMap map_e1,
                     const __grid_constant__ CUtensorMap map_b0, const __grid_constant__ CUtensorMap map_b1) {
  using namespace ptx;
  constexpr int TH = dwp_tile_h(STRIDE), TW = kDwpTileW;
  constexpr int PH = dwp_patch_h(STRIDE), PW = dwp_patch_w(STRIDE), NPX = PH * PW;
  constexpr uint32_t kPatchBytes = dwp_patch_bytes(STRIDE, EXPAND), kPitch = dwp_patch_pitch(EXPAND);
  constexpr uint32_t kAPlaneBytes = dwp_a_plane_bytes(STRIDE);
  constexpr int MT = (NPX + 127) / 128;        // EXPAND: 128-pixel strips of the patch = MMAs of M = 128
  constexpr uint32_t kExWeightBytes = 2048u;   // EXPAND: one plane of a block's expand weights, 32 rows x 64 bytes
  grid_dependency_trigger();  // the next kernel of the stream may begin its preamble

  extern __shared__ uint8_t dwp_smem_raw[];
  __shared__ __align__(8) uint64_t patch_full[kDwpMaxPatches], patch_empty[kDwpMaxPatches];
  __shared__ __align__(8) uint64_t x_full[2], x_empty[2];
  __shared__ __align__(8) uint64_t e_full[2], e_empty[2];
  __shared__ __align__(8) uint64_t a_full[2], a_empty[2];
  __shared__ __align__(8) uint64_t b_full[kDwpMaxStages], b_empty[kDwpMaxStages];
  __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // the same in all lanes, and known to be
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(dwp_smem_raw) + 1023u) & ~1023u;
  const int P = EXPAND ? 2 : p.patch_bufs;  // EXPAND: one patch per depthwise group, filled by the group itself
  const uint32_t x_base = smem_base;                                      // EXPAND: input patches, hi then mid plane
  const uint32_t x_plane = static_cast<uint32_t>(p.x_plane_bytes);
  const int XB = EXPAND ? p.x_bufs : 1;
  const uint32_t patch_base = x_base + (EXPAND ? static_cast<uint32_t>(XB) * 2u * x_plane : 0u);  // ring of fp32 patches
  const uint32_t a_base = patch_base + static_cast<uint32_t>(P) * kPatchBytes;  // two operand tiles (hi, mid planes)
  const uint32_t a_stage_bytes = 2u * kAPlaneBytes;
  const uint32_t b_base = a_base + 2u * a_stage_bytes;                    // weight ring (hi, mid planes)
  const uint32_t b_bytes = static_cast<uint32_t>(p.b_bytes);
  const uint32_t b_stage_bytes = 2u * b_bytes + (EXPAND ? 2u * kExWeightBytes : 0u);  // (+ the block's expand weights)
  const int S = p.stages;
  // the depthwise filter and bias of every channel, [10][c_blocks * 32] fp32 (taps 0..8, then the bias; zero past C)
  const uint32_t drain = b_base + static_cast<uint32_t>(S) * b_stage_bytes;  // one block per epilogue warp
  const uint32_t table = drain + static_cast<uint32_t>(dwp_drain_warps(STRIDE)) * kDrainWarpBytes;
  const int c_pad = p.c_blocks * kDwpChannels;
  // EXPAND: the expand layer's bias [c_pad] (zero past C)
  const uint32_t ex_table = table + static_cast<uint32_t>(10 * c_pad) * 4u;
  // TMEM columns: the projection's two accumulators, then one expand accumulator (MT strips x 32 columns) per group
  const uint32_t acc_stride = p.block_n > 128 ? 256u : 128u;
  const uint32_t e_col0 = 2u * acc_stride;
  const int tiles_per_image = p.tiles_y * p.tiles_x;
  const int total_tiles = p.images * tiles_per_image * p.tiles_n;
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < kDwpMaxPatches; ++i) {
      mbar_init(smem_u32(&patch_full[i]), 1);
      mbar_init(smem_u32(&patch_empty[i]), 4);  // one arrival per warp of the depthwise group that read it
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&x_full[i]), 1);
      mbar_init(smem_u32(&x_empty[i]), 1);  // the commit after the tile's last expand MMA
      mbar_init(smem_u32(&e_full[i]), 1);
      mbar_init(smem_u32(&e_empty[i]), 4);  // the four warps of the group that read the accumulator
      mbar_init(smem_u32(&a_full[i]), 4);
      mbar_init(smem_u32(&a_empty[i]), 1);
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 4);
    }
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&b_full[i]), 1);
      mbar_init(smem_u32(&b_empty[i]), 1);
    }
    fence_mbar_init();
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_b0);
    prefetch_tensormap(&map_b1);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), kTcTmemCols);
    tmem_relinquish();
  }
  // (constants of the layers, not results of the kernel before: they may be read ahead of the dependency wait)
  for (int i = static_cast<int>(threadIdx.x); i < 10 * c_pad; i += kDwpThreads) {
    const int k = i / c_pad, c = i - k * c_pad;
    float v = 0.0f;
    if (c < p.C) v = k < 9 ? __ldg(p.dw_weights + static_cast<size_t>(k) * p.C + c) : (p.dw_bias != nullptr ? __ldg(p.dw_bias + c) : 0.0f);
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(table + static_cast<uint32_t>(i) * 4u), "f"(v) : "memory");
  }
  if (EXPAND) {
    for (int c = static_cast<int>(threadIdx.x); c < c_pad; c += kDwpThreads) {
      const float v = (c < p.C && p.ex_bias != nullptr) ? __ldg(p.ex_bias + c) : 0.0f;
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(ex_table + static_cast<uint32_t>(c) * 4u), "f"(v) : "memory");
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  if (warp != 0) grid_dependency_wait();  // (the producer waits once its first copies of weights are under way)

  // The CTA's tiles: blockIdx.x + k * gridDim.x, column tiles of one pixel tile next to each other, so CTAs working side by
  // side share the patch in L2.  A walk takes every step-th of them by adding with carry: divisions in each role and tile
  // were a third of a one-block tile's instructions.
  struct Walk {
    int n, x, y, img, dn, dx, dy, dimg;
  };
  auto walk_from = [&](int tile, int step) {
    Walk w;
    w.n = tile % p.tiles_n, tile /= p.tiles_n;
    w.x = tile % p.tiles_x, tile /= p.tiles_x;
    w.y = tile % p.tiles_y, w.img = tile / p.tiles_y;
    w.dn = step % p.tiles_n, step /= p.tiles_n;
    w.dx = step % p.tiles_x, step /= p.tiles_x;
    w.dy = step % p.tiles_y, w.dimg = step / p.tiles_y;
    return w;
  };
  auto walk_on = [&](Walk& w) {
    w.n += w.dn, w.x += w.dx, w.y += w.dy, w.img += w.dimg;
    if (w.n >= p.tiles_n) w.n -= p.tiles_n, ++w.x;
    if (w.x >= p.tiles_x) w.x -= p.tiles_x, ++w.y;
    if (w.y >= p.tiles_y) w.y -= p.tiles_y, ++w.img;
  };

  if (warp < 4) {
    reg_dealloc<kDwpIssueRegs>();
    if (warp == 0) {
      // ------------------------------------------------------------ producer
      // per channel block the fp32 patch (EXPAND: per tile both planes of the input patch), the two planes of the block's
      // projection weights and (EXPAND) of its expand weights; one elected thread (tc_gemm.cuh says why)
      if (elect_one()) {
        const uint32_t patch_tx = static_cast<uint32_t>(NPX * kDwpChannels * 4);
        const uint32_t x_tx = 2u * static_cast<uint32_t>(NPX) * static_cast<uint32_t>(p.x_row_bytes);
        const uint32_t b_tx = 2u * static_cast<uint32_t>(p.block_n) * 64u + (EXPAND ? 2u * 32u * static_cast<uint32_t>(p.x_row_bytes) : 0u);
        int s = 0, pb = 0;
        uint32_t ph = 0, p_ph = 0;
        long long patches = 0, weights = 0, tiles_done = 0, x_issued = 0;
        bool ok = true;
        // a block's weights into ring stage `st`
        auto load_weights = [&](int st, int cb, int n0) {
          const uint32_t fb = smem_u32(&b_full[st]);
          mbar_arrive_expect_tx(fb, b_tx);
          const uint32_t stage = b_base + static_cast<uint32_t>(st) * b_stage_bytes;
          tma_load_2d(stage, &map_b0, fb, cb * kDwpChannels, n0);
          tma_load_2d(stage + b_bytes, &map_b1, fb, cb * kDwpChannels, n0);
          if (EXPAND) {
            tma_load_2d(stage + 2u * b_bytes, &map_e0, fb, 0, cb * kDwpChannels);
            tma_load_2d(stage + 2u * b_bytes + kExWeightBytes, &map_e1, fb, 0, cb * kDwpChannels);
          }
          ++weights;
        };
        // no kernel writes weights: those of the first tile's first blocks come in while the kernel before this one runs
        const int ahead = static_cast<int>(blockIdx.x) < total_tiles ? min(S, p.c_blocks) : 0;
        Walk w = walk_from(static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
        Walk xw = w;  // EXPAND: the tile whose input patch is requested next
        for (int cb = 0; cb < ahead; ++cb) load_weights(cb, cb, w.n * p.block_n);
        grid_dependency_wait();
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++tiles_done, walk_on(w)) {
          const int img = w.img, oy0 = w.y * TH, ox0 = w.x * TW, n0 = w.n * p.block_n;
          if (EXPAND) {
            // With two buffers the patch of the NEXT tile is requested here (the first tile's before the loop): its
            // buffer was released by the tile before this one, so the wait cannot hold up this tile's weight copies.
            // With one buffer the patch of THIS tile is requested, once the previous tile's expand MMAs have read theirs.
            const long long first = XB == 2 ? (tiles_done == 0 ? 0 : tiles_done + 1) : tiles_done;
            const long long last = XB == 2 ? tiles_done + 1 : tiles_done;
            for (long long tl = first; tl <= last && ok; ++tl) {
              const int t2 = static_cast<int>(blockIdx.x) + static_cast<int>(tl) * static_cast<int>(gridDim.x);
              if (t2 >= total_tiles) break;
              const int img2 = xw.img, oy2 = xw.y * TH, ox2 = xw.x * TW;
              walk_on(xw);
              const int xb = static_cast<int>(tl % XB);
              const uint32_t x_ph = static_cast<uint32_t>((tl / XB) & 1);
              if (!mbar_wait_bounded(smem_u32(&x_empty[xb]), x_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
                ok = false;
                break;
              }
              const uint32_t dst = x_base + static_cast<uint32_t>(xb) * 2u * x_plane;
              mbar_arrive_expect_tx(smem_u32(&x_full[xb]), x_tx);
              tma_load_4d(dst, &map_x, smem_u32(&x_full[xb]), 0, ox2 * STRIDE - p.pad_l, oy2 * STRIDE - p.pad_t, img2);
              tma_load_4d(dst + x_plane, &map_x1, smem_u32(&x_full[xb]), 0, ox2 * STRIDE - p.pad_l, oy2 * STRIDE - p.pad_t, img2);
              ++x_issued;
            }
            if (!ok) break;
          }
          for (int cb = 0; cb < p.c_blocks && ok; ++cb) {
            if (!EXPAND) {
              if (!mbar_wait_bounded(smem_u32(&patch_empty[pb]), p_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
                ok = false;
                break;
              }
              mbar_arrive_expect_tx(smem_u32(&patch_full[pb]), patch_tx);
              tma_load_4d(patch_base + static_cast<uint32_t>(pb) * kPatchBytes, &map_x, smem_u32(&patch_full[pb]), cb * kDwpChannels,
                          ox0 * STRIDE - p.pad_l, oy0 * STRIDE - p.pad_t, img);
              ++patches;
              if (++pb == P) {
                pb = 0;
                p_ph ^= 1u;
              }
            }
            if (tiles_done > 0 || cb >= ahead) {
              if (!mbar_wait_bounded(smem_u32(&b_empty[s]), ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
                ok = false;
                break;
              }
              load_weights(s, cb, n0);
            }
            if (++s == S) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        {
          if (!ok) {
            if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
          }
          if (*abort_ptr != 0) {
            // copies issued by this warp may still be landing: wait (bounded) for the last ones
            int zero = 0;
            for (long long i = weights > S ? weights - S : 0; i < weights; ++i)
              mbar_wait_bounded(smem_u32(&b_full[i % S]), static_cast<uint32_t>((i / S) & 1), &zero, 200000000ull);
            for (long long i = patches > P ? patches - P : 0; i < patches; ++i)
              mbar_wait_bounded(smem_u32(&patch_full[i % P]), static_cast<uint32_t>((i / P) & 1), &zero, 200000000ull);
            for (long long i = x_issued > XB ? x_issued - XB : 0; i < x_issued; ++i)
              mbar_wait_bounded(smem_u32(&x_full[i % XB]), static_cast<uint32_t>((i / XB) & 1), &zero, 200000000ull);
          }
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------- MMA issuer
      if (elect_one()) {
        const uint32_t idesc = instr_desc(1u, 1u, kTcBlockM, static_cast<uint32_t>(p.block_n));
        const uint32_t idesc_ex = instr_desc(1u, 1u, kTcBlockM, 32u);
        const uint64_t fixed = smem_desc_kmajor(0u, 64u);  // 64-byte rows, 64-byte swizzle
        const uint64_t fixed_x = smem_desc_kmajor(0u, EXPAND ? static_cast<uint32_t>(p.x_row_bytes) : 64u);
        const uint64_t a_plane_units = kAPlaneBytes >> 4;
        const uint64_t b_units = b_bytes >> 4;
        const int c_blocks = p.c_blocks;
        const int my_tiles = blockIdx.x < static_cast<unsigned>(total_tiles) ? (total_tiles - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;
        bool ok = true;
        // EXPAND: the expand layer of the next item (tile and channel block, in order) into the TMEM accumulator of the
        // group that takes the item: the patch strips (A, 128 pixels x 32 channels each) times the block's 32 weight
        // rows (B), three products per K step.  Issued two items ahead of the projection of the same group.
        int e_tiles = 0, e_cb = 0, xb = 0, st = 0, g = 0;
        uint32_t x_ph = 0, st_ph = 0, g_ph = 0;
        auto issue_expand = [&]() -> bool {
          if (e_tiles == my_tiles) return true;  // (the last items have no successors)
          if (e_cb == 0 && !mbar_wait_bounded(smem_u32(&x_full[xb]), x_ph, abort_ptr, kTcWaitLimitNs)) return false;
          if (!mbar_wait_bounded(smem_u32(&b_full[st]), st_ph, abort_ptr, kTcWaitLimitNs)) return false;
          if (!mbar_wait_bounded(smem_u32(&e_empty[g]), g_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) return false;
          tc_fence_after_sync();
          const uint32_t xa = x_base + static_cast<uint32_t>(xb) * 2u * x_plane;
          const uint32_t wb = b_base + static_cast<uint32_t>(st) * b_stage_bytes + 2u * b_bytes;
          const uint64_t w0 = fixed_x + ((wb & 0x3ffffu) >> 4);
          const uint64_t w_units = kExWeightBytes >> 4;
          const uint64_t x_units = x_plane >> 4;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const uint32_t d = tmem_base + e_col0 + static_cast<uint32_t>(g * MT + mt) * 32u;
            const uint64_t a0 = fixed_x + (((xa + static_cast<uint32_t>(mt) * 128u * static_cast<uint32_t>(p.x_row_bytes)) & 0x3ffffu) >> 4);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              if (k >= p.ex_ksteps) break;  // (16 input channels: the second half of the 64-byte rows is zero padding)
              const uint64_t ka = a0 + 2u * k, kb = w0 + 2u * k;
              mma_f16(d, ka + x_units, kb, idesc_ex, k ? 1u : 0u);  // mid * hi
              mma_f16(d, ka, kb + w_units, idesc_ex, 1u);            // hi * mid
              mma_f16(d, ka, kb, idesc_ex, 1u);                      // hi * hi
            }
          }
          tc_commit(smem_u32(&e_full[g]));
          g ^= 1;
          if (g == 0) g_ph ^= 1u;
          if (++st == S) {
            st = 0;
            st_ph ^= 1u;
          }
          if (++e_cb == c_blocks) {
            tc_commit(smem_u32(&x_empty[xb]));  // the tile's input patch has been read
            e_cb = 0;
            ++e_tiles;
            if (++xb == XB) {
              xb = 0;
              x_ph ^= 1u;
            }
          }
          return true;
        };
        if (EXPAND) ok = issue_expand() && issue_expand();
        int s = 0, as = 0, acc = 0;
        uint32_t ph = 0, a_ph = 0, acc_ph = 0;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
          if (!mbar_wait_bounded(smem_u32(&tempty_bar[acc]), acc_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc) * acc_stride;
          uint32_t accumulate = 0u;
          for (int cb = 0; cb < c_blocks; ++cb) {
            if (EXPAND && !issue_expand()) {
              ok = false;
              break;
            }
            // (EXPAND: the stage's copies were awaited when its expand MMAs were issued)
            if (!mbar_wait_bounded(smem_u32(&a_full[as]), a_ph, abort_ptr, kTcWaitLimitNs) ||
                (!EXPAND && !mbar_wait_bounded(smem_u32(&b_full[s]), ph, abort_ptr, kTcWaitLimitNs))) {
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint64_t a0 = fixed + (((a_base + static_cast<uint32_t>(as) * a_stage_bytes) & 0x3ffffu) >> 4);
            const uint64_t b0 = fixed + (((b_base + static_cast<uint32_t>(s) * b_stage_bytes) & 0x3ffffu) >> 4);
#pragma unroll
            for (int k = 0; k < 2; ++k) {  // two K steps of 16 channels (32 bytes = 2 units) per block
              const uint64_t ka = a0 + 2u * k;
              const uint64_t kb = b0 + 2u * k;
              mma_f16(d_tmem, ka + a_plane_units, kb, idesc, accumulate);  // mid * hi
              mma_f16(d_tmem, ka, kb + b_units, idesc, 1u);                // hi * mid
              mma_f16(d_tmem, ka, kb, idesc, 1u);                          // hi * hi
              accumulate = 1u;
            }
            tc_commit(smem_u32(&a_empty[as]));
            tc_commit(smem_u32(&b_empty[s]));
            as ^= 1;
            if (as == 0) a_ph ^= 1u;
            if (++s == S) {
              s = 0;
              ph ^= 1u;
            }
          }
          if (!ok) break;
          tc_commit(smem_u32(&tfull_bar[acc]));
          acc ^= 1;
          if (acc == 0) acc_ph ^= 1u;
        }
        if (!ok) {
          if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_MMA);
        }
      }
    }  // (warps 2 and 3 have no role: registers are split between whole warpgroups)
  } else if (warp < 12) {
    // ------------------------------------------------------------ epilogue (warps 4-11)
    // two groups of four warps on alternate tiles, an accumulator each
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;  // accumulator row = pixel (row / 8, row % 8) of the tile
    const TcDwProjParams lp = p;
    TcDirect d{};
    d.res_mode = p.res_mode;
    d.act = p.act;
    d.act_a = p.act_a;
    d.act_b = p.act_b;
    d.wide = p.wide;
    const int acc = (warp - 4) >> 2;
    const bool has_rows = quarter * 32 < TH * TW;
    d.stage = drain + static_cast<uint32_t>(acc * (dwp_drain_warps(STRIDE) / 2) + quarter) * kDrainWarpBytes;
    uint32_t acc_ph = 0;
    bool ok = true;
    Walk w = walk_from(static_cast<int>(blockIdx.x + acc * gridDim.x), static_cast<int>(2 * gridDim.x));
    for (int tile = blockIdx.x + acc * gridDim.x; tile < total_tiles && ok; tile += 2 * gridDim.x, walk_on(w)) {
      const int img = w.img, oy0 = w.y * TH, ox0 = w.x * TW, n0 = w.n * p.block_n;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc) * acc_stride;
      // (of a stride-2 tile only the first 64 rows are pixels)
      const int oy = oy0 + (row >> 3), ox = ox0 + (row & 7);
      const bool inside = row < TH * TW && oy < lp.H && ox < lp.W;
      const long long at = ((static_cast<long long>(img) * lp.H + oy) * lp.W + ox) * lp.N + n0;
      const int es = lp.out_mode == OUT_BF16X2 ? 2 : 4, rs = lp.res_mode == RES_BF16X2 ? 2 : 4;
      // (a warp's rows are four rows of eight pixels)
      const long long warp_at = at - (static_cast<long long>(lane >> 3) * lp.W + (lane & 7)) * lp.N;
      d.o0 = reinterpret_cast<uint8_t*>(lp.out0) + warp_at * es;
      d.o1 = reinterpret_cast<uint8_t*>(lp.out1) + warp_at * es;
      d.pitch = static_cast<long long>(lp.N) * es;
      d.pitch8 = d.pitch * lp.W;
      d.rows = TH * TW - 32 * quarter;
      d.xs = lp.W - ox0;
      d.ys = lp.H - (oy0 + 4 * quarter);
      d.r0 = reinterpret_cast<const uint8_t*>(lp.res0) + at * rs;
      d.r1 = reinterpret_cast<const uint8_t*>(lp.res1) + at * rs;
      d.bias = lp.bias != nullptr ? lp.bias + n0 : nullptr;
      TcOperands<KIND, EPI % 2 == 1> ops;
      if (has_rows) ops.fetch(d, 0, lp.N - n0, inside);
      ok = __all_sync(0xffffffffu,
                      mbar_wait_bounded(smem_u32(&tfull_bar[acc]), acc_ph, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      if (has_rows) tc_drain<KIND, EPI, false, false>(d, t_row, lp.block_n, lp.N - n0, inside, ops);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      acc_ph ^= 1u;
    }
    if (!ok && lane == 0) {
      if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_EPILOGUE);
    }
  } else {
    // ------------------------------------------------------------ depthwise (warps 12-19, 256 threads)
    // Two groups of four warps take alternate channel blocks (group g: blocks g, g+2, ... of the CTA's sequence,
    // so group g always fills operand tile g): while one group waits for its patch or for its operand tile to be
    // free, the other computes.  In a group a thread owns two channels (packed FMAs) and a square of COLS x 4 results:
    // 36 values read for 16 results, 45 for 8 at stride 2.
    reg_alloc<kDwpFilterRegs>();
    constexpr int COLS = dwp_cols(STRIDE);
    constexpr int R = 4;                         // result rows per thread
    constexpr int IR = (R - 1) * STRIDE + 3;     // input rows they need
    constexpr int IC = (COLS - 1) * STRIDE + 3;  // input columns
    const int t = static_cast<int>(threadIdx.x) - 384;
    const int group = t >> 7;
    const int pair = t & 15;                                // channels 2*pair and 2*pair+1 of the block
    const int col0 = ((t >> 4) % (TW / COLS)) * COLS;       // first of the thread's columns of the tile
    const int row0 = (((t & 127) >> 4) / (TW / COLS)) * R;  // first of the thread's rows
    bool ok = true;
    // none / ReLU / clip as one clamp: fminf(fmaxf(y, lo), hi) returns y itself between the bounds
    const float act_lo = p.dw_act == ACT_RELU ? 0.0f : (p.dw_act == ACT_CLIP ? p.dw_act_a : -INFINITY);
    const float act_hi = p.dw_act == ACT_CLIP ? p.dw_act_b : INFINITY;
    const float ex_lo = p.ex_act == ACT_RELU ? 0.0f : (p.ex_act == ACT_CLIP ? p.ex_act_a : -INFINITY);
    const float ex_hi = p.ex_act == ACT_CLIP ? p.ex_act_b : INFINITY;
    const uint32_t x_first = static_cast<uint32_t>((row0 * PW + col0) * STRIDE) * kPitch + static_cast<uint32_t>(pair) * 8u;
    // Operand row = pixel (row, column) of the tile; 64-byte rows with the 64-byte swizzle: the 16-byte chunk j of row m
    // lives at m*64 + ((j ^ ((m >> 1) & 3)) * 16).  Rows of one parity share the lower or the upper half of the banks, so
    // the two halves of a warp, which own columns of one parity, store the columns of a pair in opposite order.
    const bool swap = (lane & 16) != 0;
    uint32_t a_at[COLS];  // where the thread's first row goes, as the c-th store
#pragma unroll
    for (int c = 0; c < COLS; ++c)
      a_at[c] = a_base + static_cast<uint32_t>(group) * a_stage_bytes +
                stage_chunk_offset(row0 * TW + col0 + (swap ? c ^ 1 : c), pair >> 2) + static_cast<uint32_t>((pair & 3) * 4);
    uint32_t item = 0;  // position in the CTA's sequence of (tile, channel block)
    const uint32_t patch_shift = P == 4 ? 2u : 1u;  // P is 2 or 4
    Walk w = walk_from(static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, walk_on(w)) {
      const int oy0 = w.y * TH, ox0 = w.x * TW;
      for (int cb = 0; cb < p.c_blocks; ++cb, ++item) {
        if ((item & 1u) != static_cast<uint32_t>(group)) continue;
        const uint32_t use_ph = (item >> 1) & 1u;  // phase of what the group uses once per item
        const uint32_t pb = EXPAND ? static_cast<uint32_t>(group) : item & static_cast<uint32_t>(P - 1);
        const uint32_t patch = patch_base + pb * kPatchBytes;
        if (EXPAND) {
          // ---- the expand layer's accumulator of this block (MT strips of 128 patch pixels x 32 channels in
          // TMEM) -> bias, activation, zero outside the image -> the group's fp32 patch.  A warp reads the 32
          // lanes of its TMEM quarter: one pixel per thread and strip, 16 channels at a time.
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&e_full[group]), use_ph, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
          if (!ok) break;
          tc_fence_after_sync();
          const int q = warp & 3;  // the TMEM lanes this warp may read: 32 q .. 32 q + 31
          const uint32_t bias_at = ex_table + static_cast<uint32_t>(cb * kDwpChannels) * 4u;
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + e_col0 + static_cast<uint32_t>(group * MT) * 32u;
          const int strips = (NPX - q * 32 + 127) / 128;  // of them, those that reach into the patch
          // (all biases first: a load between two stores would wait for its turn in every group of four channels)
          uint64_t eb[16];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(eb[2 * j]), "=l"(eb[2 * j + 1]) : "r"(bias_at + 16u * j));
#pragma unroll 1  // (one copy of the strip's code: the kernel's roles already compete for the instruction cache)
          for (int mt = 0; mt < strips; ++mt) {
            const int px = mt * 128 + q * 32 + lane;
            // (both halves are loaded and awaited in one pass of the loop: a value carried from the load in one pass to the
            // wait in the next may be moved to another register before it has arrived)
            uint32_t v[2][16];
            tmem_ld16(taddr + static_cast<uint32_t>(mt) * 32u, v[0]);
            tmem_ld16(taddr + static_cast<uint32_t>(mt) * 32u + 16u, v[1]);
            const int pr = px / PW, pc = px - pr * PW;
            const int iy = oy0 * STRIDE - p.pad_t + pr, ix = ox0 * STRIDE - p.pad_l + pc;
            // outside the image the depthwise filter sees its zero padding, not act(bias)
            const bool inside = iy >= 0 && iy < p.Hin && ix >= 0 && ix < p.Win;
            const float lo = inside ? ex_lo : 0.0f, hi = inside ? ex_hi : 0.0f;
            const uint32_t rowat = patch + static_cast<uint32_t>(px) * kPitch;
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t y[16];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                uint64_t u;
                f32x2_add(u, f32x2_make(v[h][2 * j], v[h][2 * j + 1]), eb[8 * h + j]);
                const float2 f = f32x2_get(u);
                y[2 * j] = __float_as_uint(fminf(fmaxf(f.x, lo), hi));
                y[2 * j + 1] = __float_as_uint(fminf(fmaxf(f.y, lo), hi));
              }
              if (px < NPX) {
#pragma unroll
                for (int j = 0; j < 4; ++j) sts_16b(rowat + static_cast<uint32_t>(16 * h + 4 * j) * 4u, y + 4 * j);
              }
            }
          }
          // the accumulator has been read: the expand MMAs of the group's next block may overwrite it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&e_empty[group]));
          named_barrier_sync(3 + group, 128);  // the group's patch is complete
        }
        const uint32_t tc = table + static_cast<uint32_t>(cb * kDwpChannels + pair * 2) * 4u;  // the thread's channels
        uint64_t tap[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) tap[k] = lds_b64(tc + static_cast<uint32_t>(k * c_pad) * 4u);
        const uint64_t bias = lds_b64(tc + static_cast<uint32_t>(9 * c_pad) * 4u);
        // The group's operand tile, filled two blocks ago, must have been consumed by its MMAs, and the patch be there.  (One
        // vote behind each wait: it brings the warp together, which a lane-0 arrival may have split.  With both waits in
        // one vote, lanes of a split warp passed the second one before its phase was complete.)
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&a_empty[group]), use_ph ^ 1u, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
        if (!ok) break;
        if (!EXPAND) {
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&patch_full[pb]), (item >> patch_shift) & 1u, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
          if (!ok) break;
        }
        uint64_t acc[R][COLS];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < COLS; ++c) acc[r][c] = bias;
        // input row i of the thread's window feeds result row r with filter row kh = i - r*STRIDE
#pragma unroll
        for (int i = 0; i < IR; ++i) {
          uint64_t x[IC];
#pragma unroll
          for (int j = 0; j < IC; ++j) x[j] = lds_b64(patch + x_first + static_cast<uint32_t>(i * PW + j) * kPitch);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int kh = i - r * STRIDE;
            if (kh < 0 || kh > 2) continue;
#pragma unroll
            for (int kw = 0; kw < 3; ++kw)
#pragma unroll
              for (int c = 0; c < COLS; ++c) f32x2_fma(acc[r][c], x[c * STRIDE + kw], tap[kh * 3 + kw]);
          }
        }
        // the patch has been read: it may be refilled (by the producer, or by this group's next expand step)
        if (EXPAND) {
          named_barrier_sync(5 + group, 128);
        } else {
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&patch_empty[pb]));
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          uint32_t hi[COLS], mid[COLS];
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            const float2 y = f32x2_get(acc[r][c]);
            split_bf16x2(fminf(fmaxf(y.x, act_lo), act_hi), fminf(fmaxf(y.y, act_lo), act_hi), hi[c], mid[c]);
          }
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            const uint32_t at = a_at[c] + static_cast<uint32_t>(r * TW) * 64u;  // (eight rows further: the same chunk)
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(swap ? hi[c ^ 1] : hi[c]) : "memory");
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + kAPlaneBytes), "r"(swap ? mid[c ^ 1] : mid[c]) : "memory");
          }
        }
        fence_proxy_async_smem();  // the tensor core reads what these stores wrote
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&a_full[group]));
        __syncwarp();
      }
    }
    if (!ok && lane == 0) {
      if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_EPILOGUE);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, kTcTmemCols);
}

}  // namespace nb
