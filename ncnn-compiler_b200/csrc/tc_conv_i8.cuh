// int8 convolution with the whole filter and the input patches resident in shared memory.
//
// An int8 K block is short: 64 channels of a tap are two MMAs over 12 KB, and tc_gemm_kernel, which brings 128 pixel rows
// and the weights of every tap into a ring (im2col TMA), spends ~5 600 clocks on a tile of 128 x 64 results whose MMAs take
// ~860.  A filter of 64 -> 64 channels is 36 KB.  Here a CTA loads the weights of its column block once and keeps them; a
// tile is a 16 x 8 rectangle of output pixels whose input patch (18 x 10 pixels for a 3x3 filter) arrives once per channel
// block by tiled TMA (out-of-range coordinates read as zero: that is the padding), and every tap multiplies out of it
// through a descriptor that starts (kh * patch_w + kw) rows further and steps one patch row between 8-row groups.
//
// 64 -> 64 channels on 56x56, 256 images: 121 -> 53 us by events (~45 without them; 16 us of bytes), with an fp32 residual and
// an int8 copy 160 -> 116 (70 us of bytes); ResNet-18, 256 images 1 417 -> 1 175 us, 64 images 458 -> 404.
// What bounds it now is the epilogue's instructions (4 400 a tile and SM, issued in half of all clocks; the tensor pipe is busy
// for 40 %): groups of four warps take tiles in turn, each with accumulators of its own (their number is
// a multiple of the groups', so that an accumulator always belongs to one group, which meets its barrier's phases in order).
//
// int32 sums are exact, so the results are the bits of every other kernel and the planner chooses by time alone.
//
// Warps: 0 weights, then patches; 1 MMA issuer; 2 and up epilogue (tc_epilogue.cuh).  All waits are bounded.
#pragma once

#include "tc_gemm.cuh"

namespace nb {

constexpr int kI8TileH = 16;
constexpr int kI8TileW = 8;
constexpr int kI8MaxGroups = 3;
constexpr int kI8Threads = 64 + 128 * kI8MaxGroups;
constexpr int kI8MaxPatches = 8;
constexpr int kI8MaxAccs = 8;

struct TcConvI8Params {
  int images, OH, OW, N;
  int tiles_y, tiles_x, tiles_n, block_n;
  int c_blocks, k_elems, row_bytes, KH, KW;
  int pad_t, pad_l;
  int patch_h, patch_w;
  int patch_bytes;   // one patch of one channel block, rounded to 1 KB
  int b_bytes;       // weights of one tap and channel block, rounded to 1 KB
  int patches;       // depth of the patch ring
  int groups;        // epilogue groups
  int accs, acc_cols;
  int drain_bytes;   // shared memory of one epilogue warp: staged rows, then its int8 copies
  int wide, far_res; // see TcDirect; far_res: the residual has left L2 and is asked for one tile ahead
  const float* bias;
  const float* scale;
  float* out0;
  int8_t* outq;
  const float* res0;
  long long ldo;
  int res_mode, act;
  float act_a, act_b, out_scale;
  int side_count;
  int8_t* side_q0;
  int8_t* side_q1;
  float side_scale0, side_scale1;
  int* status;
};

template <int EPI, bool SIDE>
__global__ void __launch_bounds__(kI8Threads, 1)
tc_conv_i8_kernel(const __grid_constant__ TcConvI8Params p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b) {
  using namespace ptx;
  grid_dependency_trigger();  // the next kernel of the stream may begin its preamble
  extern __shared__ uint8_t i8_smem_raw[];
  __shared__ __align__(8) uint64_t b_full;
  __shared__ __align__(8) uint64_t a_full[kI8MaxPatches], a_empty[kI8MaxPatches];
  __shared__ __align__(8) uint64_t tfull_bar[kI8MaxAccs], tempty_bar[kI8MaxAccs];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // the same in all lanes, and known to be
  const int lane = threadIdx.x & 31;
  const uint32_t weights = (smem_u32(i8_smem_raw) + 1023u) & ~1023u;
  const uint32_t b_bytes = static_cast<uint32_t>(p.b_bytes), patch_bytes = static_cast<uint32_t>(p.patch_bytes);
  const int taps = p.KH * p.KW;
  const uint32_t ring = weights + static_cast<uint32_t>(taps * p.c_blocks) * b_bytes;
  const uint32_t drain = ring + static_cast<uint32_t>(p.patches) * patch_bytes;
  // a CTA stays with one column block (whose weights it holds); neighbours share their patches in L2
  const int n0 = (static_cast<int>(blockIdx.x) % p.tiles_n) * p.block_n;
  const int first = static_cast<int>(blockIdx.x) / p.tiles_n, step = static_cast<int>(gridDim.x) / p.tiles_n;
  const int tiles = p.images * p.tiles_y * p.tiles_x;
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&b_full), 1);
    for (int i = 0; i < p.patches; ++i) {
      mbar_init(smem_u32(&a_full[i]), 1);
      mbar_init(smem_u32(&a_empty[i]), 1);
    }
    for (int i = 0; i < p.accs; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 4);
    }
    fence_mbar_init();
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), kTcTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  // (host tests of the time-out path: see tc_gemm.cuh)
  const int test_stall = p.status[1];
  const uint64_t wait_limit = test_stall ? 2000000ull : kTcWaitLimitNs;
  if (warp != 0) grid_dependency_wait();

  auto decode = [&](int t, int* img, int* oy0, int* ox0) {
    const int tx = t % p.tiles_x;
    t /= p.tiles_x;
    *img = t / p.tiles_y;
    *oy0 = (t - *img * p.tiles_y) * kI8TileH;
    *ox0 = tx * kI8TileW;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ copies (one elected thread: tc_gemm.cuh says why)
    if (elect_one()) {
      // (no kernel writes weights: they come while the kernel before this one runs)
      const uint32_t wb = smem_u32(&b_full);
      mbar_arrive_expect_tx(wb, static_cast<uint32_t>(taps * p.c_blocks * p.block_n * p.row_bytes));
      uint32_t dst = weights;
      for (int cb = 0; cb < p.c_blocks; ++cb)
        for (int tap = 0; tap < taps; ++tap, dst += b_bytes) tma_load_2d(dst, &map_b, wb, (tap * p.c_blocks + cb) * p.k_elems, n0);
      grid_dependency_wait();
      const uint32_t tx = static_cast<uint32_t>(p.patch_h * p.patch_w * p.row_bytes);
      int ab = 0;
      uint32_t ph = 0;
      long long issued = 0;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step) {
        int img, oy0, ox0;
        decode(tile, &img, &oy0, &ox0);
        for (int cb = 0; cb < p.c_blocks; ++cb) {
          if (!mbar_wait_bounded(smem_u32(&a_empty[ab]), ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          if (!test_stall || issued > 0) {  // (a test's first patch is never armed: the waits for it run out)
            const uint32_t fb = smem_u32(&a_full[ab]);
            mbar_arrive_expect_tx(fb, tx);
            tma_load_4d(ring + static_cast<uint32_t>(ab) * patch_bytes, &map_a, fb, cb * p.k_elems, ox0 - p.pad_l, oy0 - p.pad_t, img);
          }
          ++issued;
          if (++ab == p.patches) {
            ab = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      if (*abort_ptr != 0) {
        // copies may still be landing: wait (bounded) for the weights and the last patches
        int zero = 0;
        mbar_wait_bounded(wb, 0u, &zero, 200000000ull);
        for (long long i = issued > p.patches ? issued - p.patches : 0; i < issued; ++i)
          mbar_wait_bounded(smem_u32(&a_full[i % p.patches]), static_cast<uint32_t>((i / p.patches) & 1), &zero, test_stall ? 2000000ull : 200000000ull);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (elect_one()) {
      const uint32_t idesc = instr_desc(2u, 1u, kTcBlockM, static_cast<uint32_t>(p.block_n));
      const uint64_t b_fixed = smem_desc_kmajor(0u, static_cast<uint32_t>(p.row_bytes));
      // A: the same rows and swizzle, 8-row groups (rows of the tile) one patch row apart; TMA and the MMA unit both
      // swizzle by absolute shared-memory address, so a descriptor may start at any row
      const uint64_t a_fixed = (b_fixed & ~(0x3fffull << 32)) | (static_cast<uint64_t>((p.patch_w * p.row_bytes) >> 4) << 32);
      const uint64_t b_first = b_fixed + ((weights & 0x3ffffu) >> 4);
      const uint64_t b_step = b_bytes >> 4, row_units = static_cast<uint64_t>(p.row_bytes >> 4);
      const uint64_t down = static_cast<uint64_t>(p.patch_w) * row_units;
      const int KH = p.KH, KW = p.KW, c_blocks = p.c_blocks;
      int ab = 0, acc = 0;
      uint32_t a_ph = 0, acc_ph = 0;
      // the next patch is here / the next accumulator is free (asked before a commit: see tc_gemm_common.cuh)
      bool ok = mbar_wait_bounded(smem_u32(&b_full), 0u, abort_ptr, wait_limit), a_seen = false, empty_seen = false;
      auto run = [&](auto steps, auto three) {
        for (int tile = first; tile < tiles && ok; tile += step) {
          if (!empty_seen && !mbar_wait_bounded(smem_u32(&tempty_bar[acc]), acc_ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * p.acc_cols);
          const int next_acc = acc + 1 == p.accs ? 0 : acc + 1;
          const uint32_t next_acc_ph = next_acc == 0 ? acc_ph ^ 1u : acc_ph;
          uint32_t accumulate = 0u;
          uint64_t b = b_first;
          for (int cb = 0; cb < c_blocks; ++cb) {
            if (!a_seen && !mbar_wait_bounded(smem_u32(&a_full[ab]), a_ph, abort_ptr, wait_limit)) {
              ok = false;
              break;
            }
            tc_fence_after_sync();
            uint64_t a_row = a_fixed + (((ring + static_cast<uint32_t>(ab) * patch_bytes) & 0x3ffffu) >> 4);
            if constexpr (decltype(three)::value) {
              // 3x3 filters, unrolled: the instructions between narrow MMAs are what the tensor pipe waits for
              constexpr uint64_t unit = 2 * decltype(steps)::value;  // of a row
#pragma unroll
              for (int tap = 0; tap < 9; ++tap, b += b_step) {
                tc_k_steps<GEMM_I8, false, decltype(steps)::value, false>(d_tmem, a_row + (tap / 3 * (kI8TileW + 2) + tap % 3) * unit, 0, b, 0, idesc, accumulate, 0);
                accumulate = 1u;
              }
            } else {
              for (int kh = 0; kh < KH; ++kh, a_row += down) {
                uint64_t a = a_row;
                for (int kw = 0; kw < KW; ++kw, a += row_units, b += b_step) {
                  tc_k_steps<GEMM_I8, false, decltype(steps)::value, false>(d_tmem, a, 0, b, 0, idesc, accumulate, 0);
                  accumulate = 1u;
                }
              }
            }
            const int next_ab = ab + 1 == p.patches ? 0 : ab + 1;
            const uint32_t next_ph = next_ab == 0 ? a_ph ^ 1u : a_ph;
            a_seen = mbar_test_wait(smem_u32(&a_full[next_ab]), next_ph);
            if (cb + 1 == c_blocks) empty_seen = mbar_test_wait(smem_u32(&tempty_bar[next_acc]), next_acc_ph ^ 1u);
            tc_commit(smem_u32(&a_empty[ab]));
            ab = next_ab;
            a_ph = next_ph;
          }
          if (!ok) break;
          tc_commit(smem_u32(&tfull_bar[acc]));
          acc = next_acc;
          acc_ph = next_acc_ph;
        }
      };
      const bool three = KH == 3 && KW == 3;
      if (p.row_bytes == 128 && three) run(std::integral_constant<int, 4>{}, std::true_type{});
      else if (p.row_bytes == 128) run(std::integral_constant<int, 4>{}, std::false_type{});
      else if (three) run(std::integral_constant<int, 2>{}, std::true_type{});
      else run(std::integral_constant<int, 2>{}, std::false_type{});
      if (!ok && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_MMA);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    constexpr int es = EPI / 2 == OUT_I8 ? 1 : 4;
    const int quarter = warp & 3;
    const int group = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;  // accumulator row = pixel (row / 8, row % 8) of the tile
    const TcConvI8Params lp = p;
    TcDirect d{};
    d.res_mode = p.res_mode;
    d.act = p.act;
    d.act_a = p.act_a;
    d.act_b = p.act_b;
    d.out_scale = p.out_scale;
    d.wide = p.wide;
    d.rows = 32;
    d.pitch = p.ldo * es;
    d.pitch8 = d.pitch * p.OW;
    d.stage = drain + static_cast<uint32_t>((warp - 2) * p.drain_bytes);
    d.bias = p.bias != nullptr ? p.bias + n0 : nullptr;
    d.scale = p.scale + n0;
    if (SIDE) {
      d.side_count = p.side_count;
      d.side_pitch = p.ldo;
      d.side_pitch8 = p.ldo * p.OW;
      d.side_stage = d.stage + kDrainWarpBytes;
      d.side_scale0 = p.side_scale0;
      d.side_scale1 = p.side_scale1;
    }
    uint8_t* const out = EPI / 2 == OUT_I8 ? reinterpret_cast<uint8_t*>(p.outq) : reinterpret_cast<uint8_t*>(p.out0);
    const int left = p.N - n0;
    int acc = group;
    uint32_t acc_ph = 0;
    bool ok = true;
    for (int tile = first + group * step; tile < tiles && ok; tile += lp.groups * step) {
      int img, oy0, ox0;
      decode(tile, &img, &oy0, &ox0);
      const int oy = oy0 + (row >> 3), ox = ox0 + (row & 7);
      const bool inside = oy < lp.OH && ox < lp.OW;
      // (a warp's rows are four rows of eight pixels)
      const long long warp_at = ((static_cast<long long>(img) * lp.OH + oy0 + 4 * quarter) * lp.OW + ox0) * lp.ldo + n0;
      d.o0 = out + warp_at * es;
      d.xs = lp.OW - ox0;
      d.ys = lp.OH - (oy0 + 4 * quarter);
      if (SIDE) {
        d.side_q0 = reinterpret_cast<uint8_t*>(lp.side_q0) + warp_at;
        d.side_q1 = reinterpret_cast<uint8_t*>(lp.side_q1) + warp_at;
      }
      if (EPI % 2 == 1)
        d.r0 = reinterpret_cast<const uint8_t*>(lp.res0 + ((static_cast<long long>(img) * lp.OH + oy) * lp.OW + ox) * lp.ldo + n0);
      TcOperands<GEMM_I8, EPI % 2 == 1> ops;
      ops.fetch(d, 0, left, inside);
      if (EPI % 2 == 1 && lp.far_res && tile + lp.groups * step < tiles) {
        int img2, oy2, ox2;
        decode(tile + lp.groups * step, &img2, &oy2, &ox2);
        oy2 += row >> 3;
        ox2 += row & 7;
        const uint8_t* r = reinterpret_cast<const uint8_t*>(lp.res0 + ((static_cast<long long>(img2) * lp.OH + oy2) * lp.OW + ox2) * lp.ldo + n0);
        if (oy2 < lp.OH && ox2 < lp.OW)
          for (int b = 0; b < 4 * min(lp.block_n, left); b += 128) prefetch_l2(r + b);
      }
      // the vote keeps the warp together: tcgen05.ld needs all 32 lanes
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&tfull_bar[acc]), acc_ph, abort_ptr, wait_limit) ? 1 : 0) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      tc_drain<GEMM_I8, EPI, SIDE, false>(d, tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * lp.acc_cols),
                                          lp.block_n, left, inside, ops);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      acc += lp.groups;
      if (acc >= lp.accs) {
        acc = group;
        acc_ph ^= 1u;
      }
    }
    if (!ok && lane == 0 && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_EPILOGUE);
  }

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, kTcTmemCols);
}

}  // namespace nb
