// What the two forms of tc_dw_project_kernel share: tile geometry, parameters, the walk over tiles, the epilogue.
#pragma once

#include "tc_gemm.cuh"

namespace nb {

constexpr int kDwpChannels = 32;  // channels per block: 64-byte bf16 rows
constexpr int kDwpTileW = 8;

// geometry of a tile by stride
__host__ __device__ constexpr int dwp_tile_h(int stride) { return stride == 1 ? 16 : 8; }
__host__ __device__ constexpr int dwp_patch_h(int stride) { return (dwp_tile_h(stride) - 1) * stride + 3; }
__host__ __device__ constexpr int dwp_patch_w(int stride) { return (kDwpTileW - 1) * stride + 3; }
__host__ __device__ constexpr int dwp_patch_pixels(int stride) { return dwp_patch_h(stride) * dwp_patch_w(stride); }

struct TcDwProjParams {
  int images, H, W, C;  // depthwise OUTPUT extent, channels of the depthwise layer
  int Hin, Win;         // depthwise input extent (= H, W at stride 1)
  int N;                // projection output channels
  int tiles_y, tiles_x, tiles_n, block_n;
  int c_blocks;         // blocks of 32 channels (the last one may be partly past C: zero-filled)
  int pad_t, pad_l;
  int stages;           // weight ring depth; whole blocks: 0 where all weights stay
  int drain_groups;     // groups of four epilogue warps in the pair: 2, or 1
  int patch_bufs;       // input patch ring depth, 2 or 4 (even: a slot then always serves the same depthwise group)
  int b_bytes;          // one plane of a weight stage, rounded to 1 KB
  int wide;             // rows of result and residual are multiples of 32 bytes, 32-byte aligned
  const float* dw_weights;  // [9][C], tap-major
  const float* dw_bias;     // [C] or null
  int dw_act;
  float dw_act_a, dw_act_b;
  // expand layer inside (tc_block.cuh): x is [image][Hin][Win][input channels] as bf16 hi / mid planes, weights packed [C][32] bf16 hi / mid
  int x_row_bytes;          // operand rows of the input patch and of the expand weights: 64 bytes (32 channels), or 32
                            // (16 channels) when the block's input has no more: two patch buffers then fit where one did
  int x_plane_bytes;        // one bf16 plane of an input patch buffer, rounded to 1 KB
  int x_bufs;               // input patch buffers: 2, or 1 when two do not fit
  int accs;                 // accumulators of the projection: 2, or 1 when a second does not fit beside the expanded pixels
  int e_bufs;               // TMEM buffers of each half's expanded pixels: 2, or 1
  int a_slots;              // operand tiles: 8, or 4
  int ex_ksteps;            // K steps of 16 input channels the expand MMAs run
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

// None / ReLU / clip as one clamp, fminf(fmaxf(y, lo), hi).  Without an activation both bounds are NaN: the other operand comes
// through whatever it is, a NaN too (which bounds of infinities would turn into one of them).
struct DwpClamp {
  float lo, hi;
  __device__ __forceinline__ DwpClamp(int act, float a, float b) {
    const float any = __int_as_float(0x7fffffff);
    lo = act == ACT_NONE ? any : (act == ACT_CLIP ? a : 0.0f);
    hi = act == ACT_NONE ? any : (act == ACT_CLIP ? b : INFINITY);
  }
  __device__ __forceinline__ float operator()(float y) const { return fminf(fmaxf(y, lo), hi); }
};

// The CTA's tiles: blockIdx.x + k * gridDim.x, column tiles of one pixel tile next to each other, so CTAs working side by
// side share the patch in L2.  A walk takes every step-th of them by adding with carry: divisions in each role and tile
// were a third of a one-block tile's instructions.
struct DwpWalk {
  int n, x, y, img, dn, dx, dy, dimg;
  __device__ __forceinline__ DwpWalk(const TcDwProjParams& p, int tile, int step) {
    n = tile % p.tiles_n;
    tile /= p.tiles_n;
    x = tile % p.tiles_x;
    tile /= p.tiles_x;
    y = tile % p.tiles_y;
    img = tile / p.tiles_y;
    dn = step % p.tiles_n;
    step /= p.tiles_n;
    dx = step % p.tiles_x;
    step /= p.tiles_x;
    dy = step % p.tiles_y;
    dimg = step / p.tiles_y;
  }
  __device__ __forceinline__ void on(const TcDwProjParams& p) {
    n += dn;
    x += dx;
    y += dy;
    img += dimg;
    if (n >= p.tiles_n) n -= p.tiles_n, ++x;
    if (x >= p.tiles_x) x -= p.tiles_x, ++y;
    if (y >= p.tiles_y) y -= p.tiles_y, ++img;
  }
};

// Four epilogue warps (`quarter`: the TMEM lanes of this one) drain the projection's accumulators.  Two such groups take
// alternate tiles, an accumulator each; one takes p.accs accumulators in turn.  `drain`: kDrainWarpBytes for each warp of the
// group that has rows.
template <int KIND, int STRIDE, int EPI>
__device__ __forceinline__ void dwp_epilogue(const TcDwProjParams& p, int groups, int group, int quarter, uint32_t drain, uint32_t tmem_base,
                                             uint32_t acc_stride, int total_tiles, uint64_t* tfull_bar, uint64_t* tempty_bar,
                                             volatile int* abort_ptr) {
  using namespace ptx;
  constexpr int TH = dwp_tile_h(STRIDE), TW = kDwpTileW;
  const int lane = threadIdx.x & 31;
  const int row = quarter * 32 + lane;  // accumulator row = pixel (row / 8, row % 8) of the tile
  const TcDwProjParams lp = p;
  TcDirect d{};
  d.res_mode = p.res_mode;
  d.act = p.act;
  d.act_a = p.act_a;
  d.act_b = p.act_b;
  d.wide = p.wide;
  const bool has_rows = quarter * 32 < TH * TW;  // (of a stride-2 tile only the first 64 rows are pixels)
  d.stage = drain + static_cast<uint32_t>(quarter) * kDrainWarpBytes;
  int acc = group;
  uint32_t acc_ph = 0;
  bool ok = true;
  DwpWalk w(p, static_cast<int>(blockIdx.x + group * gridDim.x), static_cast<int>(groups * gridDim.x));
  for (int tile = blockIdx.x + group * gridDim.x; tile < total_tiles && ok; tile += groups * gridDim.x, w.on(p)) {
    const int oy0 = w.y * TH, ox0 = w.x * TW, n0 = w.n * p.block_n;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc) * acc_stride;
    const int oy = oy0 + (row >> 3), ox = ox0 + (row & 7);
    const bool inside = row < TH * TW && oy < lp.H && ox < lp.W;
    const long long at = ((static_cast<long long>(w.img) * lp.H + oy) * lp.W + ox) * lp.N + n0;
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
    if (groups == 1 && lp.accs == 2) acc ^= 1;
    if (groups == 2 || acc == 0) acc_ph ^= 1u;
  }
  if (!ok && lane == 0) {
    if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_EPILOGUE);
  }
}

}  // namespace nb
