// Convolution of few pixels: small tiles multiplied straight out of an input patch in shared memory.
//
// A batch of one or a few images has too few 128-row tiles for 148 SMs, and what such a call then waits for is one
// tile's serial chain of K blocks.  In tc_gemm_kernel a block of 64 channels costs that chain ~900 clocks: the copies
// bring 256 pixel rows (two planes) per filter tap into the SM at ~3 clocks a row, while twelve narrow MMAs need 480.
// Here both shrink:
//   * a tile is 8 x 8 output pixels (M = 64; MMAs read 128 bytes of operands a clock: 24 clocks at 32 columns against 40
//     at M = 128), or 16 x 8 where that fills the SMs better,
//   * per block of channels the input patch under the tile is loaded ONCE by tiled TMA (out-of-range coordinates read as
//     zero: that is the padding) and every tap multiplies out of it through a shifted descriptor, so that a K block
//     brings 22 pixel rows and its weights,
//   * the weights' ring fills before the kernel waits for the one before it,
//   * a group of K blocks (all taps of a channel block where shared memory allows) shares one barrier.
// What bounds it now: the MMAs of the chain (12 x 24 clocks per 64 channels) and ~400 clocks between groups, ~0.75 us until
// the first patch has arrived and 0.5 us of epilogue.  256 channels on 14x14, one image: a K block 900 -> 330 clocks, the
// launch 25.5 -> 17.4 us by events; ResNet-18, one image 329 -> 275 us.
// Stride 2: the patch is loaded as two, its even and its odd columns (TMA traversal strides), because the rows of a
// descriptor's 8-row group are neighbours in shared memory; patch rows are skipped by the group stride.
//
// K runs over channel blocks, then taps, as in every convolution kernel here, and MMAs of any M add up a row's products
// alike, so the results are the bits of tc_gemm_kernel, sums in chunks included (TcGemmParams::chunks): the planner
// chooses by time alone.
//
// Warps: 0 patches, 1 MMA issuer, 2-5 epilogue (tc_epilogue.cuh), 6 weights.  All waits are bounded.
#pragma once

#include "tc_gemm.cuh"

namespace nb {

constexpr int kPatchThreads = 224;
constexpr int kPatchTileW = 8;
constexpr int kPatchMaxBufs = 4;

struct TcPatchParams {
  int images, OH, OW, N;
  int tile_h;                       // rows of a tile: 8 (M = 64) or 16 (M = 128)
  int tiles_y, tiles_x, tiles_n, block_n;
  int c_blocks, k_elems, row_bytes, taps, KW, k_blocks;
  int stride, pad_t, pad_l;         // input pixels between the tile origins of neighbouring output pixels
  int group, group_rows;            // K blocks of a group: the taps of group_rows filter rows on one channel block
  int groups;                       // of the whole contraction
  int patch_groups;                 // groups on one patch
  int subs;                         // arrays of a patch and plane: 1, or even and odd columns
  int patch_w, patch_h;             // pixels of one of them
  int row_step;                     // patch rows between output rows
  int sub_bytes;                    // one of them, rounded to 1 KB
  int step_even, step_odd;          // bytes from the operand rows of a group's block 0, 2, .. (1, 3, ..) to those of the next
  int patch_bufs, b_bytes, stages;  // rings: patches, weights (b_bytes: one plane of one block; a stage holds a group)
  int tmem_cols, acc_cols;
  int chunks, chunk_groups, split_k;
  uint32_t* sk_ws;
  int* sk_flags;
  int wide;
  const float* bias;
  float* out0;
  float* out1;
  const float* res0;
  const float* res1;
  long long ldo;
  int res_mode, out_mode, act;
  float act_a, act_b;
  int* status;
};

template <int KIND, int EPI>
__global__ void __launch_bounds__(kPatchThreads, 2)
tc_conv_patch_kernel(const __grid_constant__ TcPatchParams p, const __grid_constant__ CUtensorMap map_a0,
                     const __grid_constant__ CUtensorMap map_a1, const __grid_constant__ CUtensorMap map_b0,
                     const __grid_constant__ CUtensorMap map_b1) {
  using namespace ptx;
  constexpr int PLANES = tc_planes(KIND);
  extern __shared__ uint8_t patch_smem_raw[];
  __shared__ __align__(8) uint64_t a_full[kPatchMaxBufs], a_empty[kPatchMaxBufs];
  __shared__ __align__(8) uint64_t b_full[kTcMaxStages], b_empty[kTcMaxStages];
  __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // the same in all lanes, and known to be
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(patch_smem_raw) + 1023u) & ~1023u;
  const uint32_t sub_bytes = static_cast<uint32_t>(p.sub_bytes);
  const uint32_t plane_bytes = static_cast<uint32_t>(p.subs) * sub_bytes;
  const uint32_t buf_bytes = PLANES * plane_bytes;
  const uint32_t b_bytes = static_cast<uint32_t>(p.b_bytes);
  const uint32_t stage_bytes = static_cast<uint32_t>(p.group) * PLANES * b_bytes;
  const uint32_t b_ring = smem_base + static_cast<uint32_t>(p.patch_bufs) * buf_bytes;
  const uint32_t drain = b_ring + static_cast<uint32_t>(p.stages) * stage_bytes;
  const int S = p.stages, P = p.patch_bufs;
  const int chunks = p.chunks;
  const bool split_k = p.split_k != 0;
  const int tiles = p.images * p.tiles_y * p.tiles_x * p.tiles_n;
  const int units = tiles * (split_k ? chunks : 1);
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < P; ++i) {
      mbar_init(smem_u32(&a_full[i]), 1);
      mbar_init(smem_u32(&a_empty[i]), 1);
    }
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&b_full[i]), 1);
      mbar_init(smem_u32(&b_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 4);
    }
    fence_mbar_init();
    prefetch_tensormap(&map_a0);
    prefetch_tensormap(&map_b0);
    if (PLANES == 2) {
      prefetch_tensormap(&map_a1);
      prefetch_tensormap(&map_b1);
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // Only now may the next kernel come in: its CTAs may share an SM with this one (tensor memory of two CTAs of this kernel
  // fits an SM, and others leave no room in shared memory), and must not take what this one has yet to allocate.
  grid_dependency_trigger();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  // (host tests of the time-out path: see tc_gemm.cuh)
  const int test_stall = p.status[1];
  const uint64_t wait_limit = test_stall ? 2000000ull : kTcWaitLimitNs;
  if (warp != 0 && warp != 6) grid_dependency_wait();

  const int PG = p.patch_groups;

  // unit -> tile position and groups; column blocks of one pixel tile are neighbours, so that they share its patch in L2
  struct Unit {
    int tile, img, oy0, ox0, n0, g0, g1;
  };
  auto decode = [&](int unit) {
    Unit u;
    u.tile = split_k ? unit / chunks : unit;
    u.g0 = split_k ? (unit - u.tile * chunks) * p.chunk_groups : 0;
    u.g1 = split_k ? min(u.g0 + p.chunk_groups, p.groups) : p.groups;
    int t = u.tile / p.tiles_n;
    u.n0 = (u.tile - t * p.tiles_n) * p.block_n;
    const int tx = t % p.tiles_x;
    t /= p.tiles_x;
    u.img = t / p.tiles_y;
    u.oy0 = (t - u.img * p.tiles_y) * p.tile_h;
    u.ox0 = tx * kPatchTileW;
    return u;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ patches (one elected thread: tc_gemm.cuh says why)
    if (elect_one()) {
      const uint32_t tx = PLANES * static_cast<uint32_t>(p.subs * p.patch_w * p.patch_h) * static_cast<uint32_t>(p.row_bytes);
      int ab = 0;
      uint32_t ph = 0;
      long long issued = 0;
      bool ok = true, waited = false;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const Unit u = decode(unit);
        const int patch1 = (u.g1 - 1) / PG;
        for (int patch = u.g0 / PG; patch <= patch1; ++patch) {
          if (!waited) {
            grid_dependency_wait();
            waited = true;
          }
          if (!mbar_wait_bounded(smem_u32(&a_empty[ab]), ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          ++issued;
          if (test_stall && issued == 1) continue;  // (never armed: the waits for it run out)
          const uint32_t fb = smem_u32(&a_full[ab]);
          mbar_arrive_expect_tx(fb, tx);
          for (int sub = 0; sub < p.subs; ++sub) {
            const uint32_t dst = smem_base + static_cast<uint32_t>(ab) * buf_bytes + static_cast<uint32_t>(sub) * sub_bytes;
            const int x = u.ox0 * p.stride - p.pad_l + sub, y = u.oy0 * p.stride - p.pad_t;
            tma_load_4d(dst, &map_a0, fb, patch * p.k_elems, x, y, u.img);
            if (PLANES == 2) tma_load_4d(dst + plane_bytes, &map_a1, fb, patch * p.k_elems, x, y, u.img);
          }
          if (++ab == P) {
            ab = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      if (*abort_ptr != 0) {
        // copies may still be landing: wait (bounded) for the last ones
        int zero = 0;
        for (long long i = issued > P ? issued - P : 0; i < issued; ++i)
          mbar_wait_bounded(smem_u32(&a_full[i % P]), static_cast<uint32_t>((i / P) & 1), &zero, test_stall ? 2000000ull : 200000000ull);
      }
    }
  } else if (warp == 6) {
    // ------------------------------------------------------------ weights
    if (elect_one()) {
      const uint32_t tx = PLANES * static_cast<uint32_t>(p.group * p.block_n) * static_cast<uint32_t>(p.row_bytes);
      int s = 0;
      uint32_t ph = 0;
      long long issued = 0;
      bool ok = true, waited = false;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const Unit u = decode(unit);
        for (int g = u.g0; g < u.g1; ++g) {
          // (no kernel writes weights: the ring fills while the kernel before this one runs)
          if (!waited && issued == S) {
            grid_dependency_wait();
            waited = true;
          }
          if (!mbar_wait_bounded(smem_u32(&b_empty[s]), ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          const uint32_t fb = smem_u32(&b_full[s]);
          const int cb = g / PG;
          mbar_arrive_expect_tx(fb, tx);
          uint32_t dst = b_ring + static_cast<uint32_t>(s) * stage_bytes;
          int k = ((g - cb * PG) * p.group * p.c_blocks + cb) * p.k_elems;
          for (int j = 0; j < p.group; ++j, k += p.c_blocks * p.k_elems, dst += PLANES * b_bytes) {
            tma_load_2d(dst, &map_b0, fb, k, u.n0);
            if (PLANES == 2) tma_load_2d(dst + b_bytes, &map_b1, fb, k, u.n0);
          }
          ++issued;
          if (++s == S) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      if (*abort_ptr != 0) {
        int zero = 0;
        for (long long i = issued > S ? issued - S : 0; i < issued; ++i)
          mbar_wait_bounded(smem_u32(&b_full[i % S]), static_cast<uint32_t>((i / S) & 1), &zero, test_stall ? 2000000ull : 200000000ull);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (elect_one()) {
      const uint32_t idesc = instr_desc(1u, KIND == GEMM_BF16X3 ? 1u : 2u, static_cast<uint32_t>(p.tile_h * kPatchTileW),
                                        static_cast<uint32_t>(p.block_n));
      const int k_steps = p.row_bytes / 32;
      const uint64_t b_fixed = smem_desc_kmajor(0u, static_cast<uint32_t>(p.row_bytes));
      // A: the same rows and swizzle, 8-row groups (output rows) row_step patch rows apart; both TMA and the MMA unit
      // swizzle by absolute shared-memory address, so a descriptor may start at any row
      const uint32_t row_group = static_cast<uint32_t>(p.row_step * p.patch_w * p.row_bytes);
      const uint64_t a_fixed = (b_fixed & ~(0x3fffull << 32)) | (static_cast<uint64_t>(row_group >> 4) << 32);
      const uint64_t a_plane = plane_bytes >> 4, b_plane = b_bytes >> 4;
      const int KW = p.KW;
      const uint64_t b_step = PLANES * b_plane;
      const uint64_t row_units = static_cast<uint64_t>(p.patch_w * p.row_bytes) >> 4, part_units = row_units * static_cast<uint64_t>(p.group_rows);
      const uint64_t step_even = static_cast<uint64_t>(static_cast<int64_t>(p.step_even / 16)), step_odd = static_cast<uint64_t>(static_cast<int64_t>(p.step_odd / 16));
      int s = 0, ab = 0, acc = 0;
      uint32_t ph = 0, a_ph = 0, acc_ph = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const Unit u = decode(unit);
        int g1 = u.g0;
        int kh = u.g0 % PG;  // the group's place on its patch
        bool fresh = true;   // the next group is this unit's first on its patch
        while (g1 < u.g1 && ok) {  // one accumulator per chunk
          const int g0 = g1;
          g1 = chunks > 1 ? min(g0 + p.chunk_groups, u.g1) : u.g1;
          if (!mbar_wait_bounded(smem_u32(&tempty_bar[acc]), acc_ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * p.acc_cols);
          uint32_t accumulate = 0u;
          for (int g = g0; g < g1; ++g) {
            if ((fresh && !mbar_wait_bounded(smem_u32(&a_full[ab]), a_ph, abort_ptr, wait_limit)) ||
                !mbar_wait_bounded(smem_u32(&b_full[s]), ph, abort_ptr, wait_limit)) {
              ok = false;
              break;
            }
            tc_fence_after_sync();
            uint64_t a0 = a_fixed + (((smem_base + static_cast<uint32_t>(ab) * buf_bytes) & 0x3ffffu) >> 4) + static_cast<uint64_t>(kh) * part_units;
            uint64_t b0 = b_fixed + (((b_ring + static_cast<uint32_t>(s) * stage_bytes) & 0x3ffffu) >> 4);
            // A group's MMAs in a row: what lies between two groups (barrier reads next to operand reads that fill shared
            // memory's bandwidth, commits, indexes: ~400 clocks) is more than a block's narrow MMAs take, and the queue of
            // issued MMAs is too short to cover it.
            for (int r = 0; r < p.group_rows; ++r) {
              uint64_t a = a0;
              if (k_steps == 4) {
                for (int j = 0; j < KW; ++j) {
                  tc_k_steps<KIND, false, 4, false>(d_tmem, a, a_plane, b0, b_plane, idesc, accumulate, 0);
                  accumulate = 1u;
                  a += j & 1 ? step_odd : step_even;
                  b0 += b_step;
                }
              } else {
                for (int j = 0; j < KW; ++j) {
                  tc_k_steps<KIND, false, 2, false>(d_tmem, a, a_plane, b0, b_plane, idesc, accumulate, 0);
                  accumulate = 1u;
                  a += j & 1 ? step_odd : step_even;
                  b0 += b_step;
                }
              }
              a0 += row_units;
            }
            tc_commit(smem_u32(&b_empty[s]));
            if (++s == S) {
              s = 0;
              ph ^= 1u;
            }
            fresh = ++kh == PG || g + 1 == u.g1;
            if (fresh) {
              tc_commit(smem_u32(&a_empty[ab]));
              if (++ab == P) {
                ab = 0;
                a_ph ^= 1u;
              }
              kh = 0;
            }
          }
          if (!ok) break;
          tc_commit(smem_u32(&tfull_bar[acc]));
          acc ^= 1;
          if (acc == 0) acc_ph ^= 1u;
        }
      }
      if (!ok && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_MMA);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // M = 128: accumulator row r lies in lane r; M = 64: row r in lane 32 * (r / 16) + r % 16, so a warp has 16 rows
    const int quarter = warp & 3;
    const int warp_rows = p.tile_h * kPatchTileW / 4;
    const int row = quarter * warp_rows + lane;
    const TcPatchParams lp = p;
    TcDirect d{};
    d.res_mode = p.res_mode;
    d.act = p.act;
    d.act_a = p.act_a;
    d.act_b = p.act_b;
    d.wide = p.wide;
    d.rows = warp_rows;
    d.chw = static_cast<long long>(p.OH) * p.OW;
    d.stage = drain + static_cast<uint32_t>(quarter) * kDrainWarpBytes;
    constexpr int es = EPI / 2 == OUT_BF16X2 ? 2 : 4;
    d.pitch = p.ldo * es;
    d.pitch8 = d.pitch * p.OW;
    const uint32_t t_quarter = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    int acc = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      const Unit u = decode(unit);
      const int oy = u.oy0 + (row >> 3), ox = u.ox0 + (row & 7);
      const bool inside = lane < warp_rows && oy < lp.OH && ox < lp.OW;
      const int first_row = u.oy0 + ((quarter * warp_rows) >> 3);  // of the warp
      if (EPI / 2 == OUT_CHW) {
        d.o0 = reinterpret_cast<uint8_t*>(lp.out0) +
               ((static_cast<long long>(u.img) * lp.N + u.n0) * d.chw + static_cast<long long>(oy) * lp.OW + ox) * 4;
      } else {
        const long long at = ((static_cast<long long>(u.img) * lp.OH + first_row) * lp.OW + u.ox0) * lp.ldo + u.n0;
        d.o0 = reinterpret_cast<uint8_t*>(lp.out0) + at * es;
        d.o1 = reinterpret_cast<uint8_t*>(lp.out1) + at * es;
      }
      d.xs = lp.OW - u.ox0;
      d.ys = lp.OH - first_row;
      if (EPI % 2 == 1) {
        const int rs = lp.res_mode == RES_BF16X2 ? 2 : 4;
        const long long at = ((static_cast<long long>(u.img) * lp.OH + oy) * lp.OW + ox) * lp.ldo + u.n0;
        d.r0 = reinterpret_cast<const uint8_t*>(lp.res0) + at * rs;
        d.r1 = reinterpret_cast<const uint8_t*>(lp.res1) + at * rs;
      }
      d.bias = lp.bias != nullptr ? lp.bias + u.n0 : nullptr;
      const int left = lp.N - u.n0;
      TcOperands<KIND, EPI % 2 == 1> ops;
      ops.fetch(d, 0, left, inside);
      uint32_t t_row = 0;
      // the vote keeps the warp together: tcgen05.ld needs all 32 lanes
      auto wait_acc = [&] {
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&tfull_bar[acc]), acc_ph, abort_ptr, wait_limit) ? 1 : 0) != 0;
        tc_fence_after_sync();
        t_row = t_quarter + static_cast<uint32_t>(acc * lp.acc_cols);
      };
      auto release_acc = [&] {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
        acc ^= 1;
        if (acc == 0) acc_ph ^= 1u;
      };
      wait_acc();
      if (!ok) break;
      if (chunks > 1 && split_k) {
        // the chunks of a tile run on different CTAs; whichever warp publishes its rows last adds them up (tc_gemm.cuh)
        const size_t slot_words = static_cast<size_t>(kTcBlockM) * lp.block_n;
        uint32_t* const ws = lp.sk_ws + static_cast<size_t>(unit) * slot_words + static_cast<size_t>(quarter * 32 + lane) * 16;
        tc_publish_chunk(t_row, ws, lp.block_n, inside);
        int* const count = lp.sk_flags + u.tile * 4 + quarter;
        __threadfence();
        __syncwarp();
        int before = 0;
        if (lane == 0) before = atomicAdd(count, 1);
        if (__shfl_sync(0xffffffffu, before, 0) != chunks - 1) {
          release_acc();
          continue;
        }
        if (lane == 0) *count = 0;  // for the next launch
        __threadfence();
        tc_gather_chunks<KIND>(ws - static_cast<size_t>(unit - u.tile * chunks) * slot_words, slot_words, chunks, t_row, lp.block_n, inside);
      } else if (chunks > 1) {
        const uint32_t t_sum = t_quarter + static_cast<uint32_t>(2 * lp.acc_cols);
        for (int c = 0; c < chunks && ok; ++c) {
          tc_add_chunk(t_row, t_sum, lp.block_n, c == 0);
          if (c + 1 == chunks) break;
          release_acc();
          wait_acc();
        }
        if (!ok) break;
        t_row = t_sum;
      }
      tc_drain<KIND, EPI, false, false>(d, t_row, lp.block_n, left, inside, ops);
      release_acc();
    }
    if (!ok && lane == 0 && atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_EPILOGUE);
  }

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
}

}  // namespace nb
