// The second half, or the whole, of an inverted-residual block in one kernel:
//   [1x1 "expand" convolution + activation ->] 3x3 depthwise convolution + activation -> 1x1 "projection"
//   convolution (+ bias, residual, activation).
//
// Run one after the other these layers write the widest tensors of the network to HBM and read them back, on
// layers that are bound by HBM either way.  Here the expanded tensor and the depthwise result never leave the
// SM.  The whole block is tc_block.cuh; this is the pair at stride 1.  A tile is a 16 x 8 rectangle of output pixels of one
// image (the 128 rows of the projection's GEMM); per block of 32 channels
//   * the fp32 input patch of the depthwise filter (18 x 10 pixels x 32 channels) arrives in shared memory by TMA
//     (coordinates outside the image read as zero: that is the padding),
//   * four CUDA-core warps (two such groups take alternate blocks) compute the depthwise results from it with
//     the arithmetic of the stand-alone kernel (bias, nine fmaf in filter order, activation), split each value
//     into its bf16 pair (hi = bf16(x), mid = bf16(x - hi)) and write both planes straight into the K-major,
//     64-byte-swizzled operand tile that tcgen05.mma reads,
//   * one thread issues the projection's MMAs (mid*hi + hi*mid + hi*hi, as tc_gemm_kernel does) against
//     that channel block's weights, which TMA streams through a small ring,
// and the usual epilogue warps drain the accumulator (bias, residual, activation).
// The operands, their order and the accumulation are those of the two separate kernels, so the results are the same bits.
//
// Warps (640 threads): 0 TMA producer, 1 MMA issuer, 4-11 epilogue (two groups on alternate tiles, or the first alone), 12-19 depthwise; registers
// are split between the roles.  Every wait is bounded and ends in the status word.
//
// What bounds it: shared memory (~800 of a block's ~1 700 clocks are its own reads and writes, ~250 the MMAs') and the
// instructions of the depthwise warps, which wait on one another (shared memory -> FMA -> clamp -> split -> shared memory).
// What counts is how few a result takes: a thread owns two channels (packed FMAs) and a square of results, every address is a
// constant away from one base, and tiles are walked by adding with carry.  256 images of 112x112x32 -> 16: 198 us with four
// channels x 8 rows a thread -> 159.  Sixteen depthwise warps with half the results each were no faster.
#pragma once

#include "tc_block.cuh"

namespace nb {

constexpr int kDwpThreads = 640;
// registers a thread: at launch (what the compiler gives 640 threads of one block; checked where a launch is planned), of the issuing
// warpgroup, of the two epilogue groups and of the two depthwise groups
constexpr int kDwpRegs = 96, kDwpIssueRegs = 56, kDwpDrainRegs = 96, kDwpFilterRegs = 112;
static_assert(kDwpIssueRegs + 2 * kDwpDrainRegs + 2 * kDwpFilterRegs <= 5 * kDwpRegs, "what the launch gives the block");
constexpr int kDwpMaxStages = 4;
constexpr int kDwpMaxPatches = 4;
constexpr int kDwpPatchBytes = (dwp_patch_pixels(1) * kDwpChannels * 4 + 1023) / 1024 * 1024;
constexpr int kDwpAPlaneBytes = 128 * 64;  // one bf16 plane of the operand tile

template <int KIND, int EPI>
__device__ __forceinline__ void dwp_pair_body(const TcDwProjParams& p, const CUtensorMap& map_x, const CUtensorMap& map_b0, const CUtensorMap& map_b1) {
  using namespace ptx;
  constexpr int TH = dwp_tile_h(1), TW = kDwpTileW;
  constexpr int PW = dwp_patch_w(1), NPX = dwp_patch_pixels(1);
  constexpr uint32_t kPatchBytes = kDwpPatchBytes, kPitch = kDwpChannels * 4;
  constexpr uint32_t kAPlaneBytes = kDwpAPlaneBytes;
  grid_dependency_trigger();  // the next kernel of the stream may begin its preamble

  extern __shared__ uint8_t dwp_smem_raw[];
  __shared__ __align__(8) uint64_t patch_full[kDwpMaxPatches], patch_empty[kDwpMaxPatches];
  __shared__ __align__(8) uint64_t a_full[2], a_empty[2];
  __shared__ __align__(8) uint64_t b_full[kDwpMaxStages], b_empty[kDwpMaxStages];
  __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // the same in all lanes, and known to be
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(dwp_smem_raw) + 1023u) & ~1023u;
  const int P = p.patch_bufs;
  const uint32_t patch_base = smem_base;  // ring of fp32 patches
  const uint32_t a_base = patch_base + static_cast<uint32_t>(P) * kPatchBytes;  // two operand tiles (hi, mid planes)
  const uint32_t a_stage_bytes = 2u * kAPlaneBytes;
  const uint32_t b_base = a_base + 2u * a_stage_bytes;                    // weight ring (hi, mid planes)
  const uint32_t b_bytes = static_cast<uint32_t>(p.b_bytes);
  const uint32_t b_stage_bytes = 2u * b_bytes;
  const int S = p.stages;
  // the depthwise filter and bias of every channel, [10][c_blocks * 32] fp32 (taps 0..8, then the bias; zero past C)
  const uint32_t drain = b_base + static_cast<uint32_t>(S) * b_stage_bytes;  // one block per epilogue warp
  const uint32_t table = drain + static_cast<uint32_t>(4 * p.drain_groups) * kDrainWarpBytes;
  const int c_pad = p.c_blocks * kDwpChannels;
  const uint32_t acc_stride = p.block_n > 128 ? 256u : 128u;  // TMEM columns of an accumulator
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
      mbar_init(smem_u32(&a_full[i]), 4);  // the four warps of the group that filled it
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
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  if (warp != 0) grid_dependency_wait();  // (the producer waits once its first copies of weights are under way)

  if (warp < 4) {
    reg_dealloc<kDwpIssueRegs>();
    if (warp == 0) {
      // ------------------------------------------------------------ producer
      // per channel block the fp32 patch and the two planes of the block's projection weights; one elected thread (tc_gemm.cuh says why)
      if (elect_one()) {
        const uint32_t patch_tx = static_cast<uint32_t>(NPX * kDwpChannels * 4);
        const uint32_t b_tx = 2u * static_cast<uint32_t>(p.block_n) * 64u;
        int s = 0, pb = 0;
        uint32_t ph = 0, p_ph = 0;
        long long patches = 0, weights = 0, tiles_done = 0;
        bool ok = true;
        // a block's weights into ring stage `st`
        auto load_weights = [&](int st, int cb, int n0) {
          const uint32_t fb = smem_u32(&b_full[st]);
          mbar_arrive_expect_tx(fb, b_tx);
          const uint32_t stage = b_base + static_cast<uint32_t>(st) * b_stage_bytes;
          tma_load_2d(stage, &map_b0, fb, cb * kDwpChannels, n0);
          tma_load_2d(stage + b_bytes, &map_b1, fb, cb * kDwpChannels, n0);
          ++weights;
        };
        // no kernel writes weights: those of the first tile's first blocks come in while the kernel before this one runs
        const int ahead = static_cast<int>(blockIdx.x) < total_tiles ? min(S, p.c_blocks) : 0;
        DwpWalk w(p, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
        for (int cb = 0; cb < ahead; ++cb) load_weights(cb, cb, w.n * p.block_n);
        grid_dependency_wait();
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++tiles_done, w.on(p)) {
          const int img = w.img, oy0 = w.y * TH, ox0 = w.x * TW, n0 = w.n * p.block_n;
          for (int cb = 0; cb < p.c_blocks && ok; ++cb) {
            if (!mbar_wait_bounded(smem_u32(&patch_empty[pb]), p_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(smem_u32(&patch_full[pb]), patch_tx);
            tma_load_4d(patch_base + static_cast<uint32_t>(pb) * kPatchBytes, &map_x, smem_u32(&patch_full[pb]), cb * kDwpChannels,
                        ox0 - p.pad_l, oy0 - p.pad_t, img);
            ++patches;
            if (++pb == P) {
              pb = 0;
              p_ph ^= 1u;
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
          }
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------- MMA issuer
      if (elect_one()) {
        const uint32_t idesc = instr_desc(1u, 1u, kTcBlockM, static_cast<uint32_t>(p.block_n));
        const uint64_t fixed = smem_desc_kmajor(0u, 64u);  // 64-byte rows, 64-byte swizzle
        const uint64_t a_plane_units = kAPlaneBytes >> 4;
        const uint64_t b_units = b_bytes >> 4;
        const int c_blocks = p.c_blocks;
        bool ok = true;
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
            if (!mbar_wait_bounded(smem_u32(&a_full[as]), a_ph, abort_ptr, kTcWaitLimitNs) ||
                !mbar_wait_bounded(smem_u32(&b_full[s]), ph, abort_ptr, kTcWaitLimitNs)) {
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
    // two groups of four warps on alternate tiles, an accumulator each; or one, where the second's shared memory is the rings'
    const int group = (warp - 4) >> 2;
    if (group < p.drain_groups)
      dwp_epilogue<KIND, 1, EPI>(p, p.drain_groups, group, warp & 3, drain + static_cast<uint32_t>(group) * 4u * kDrainWarpBytes, tmem_base,
                                 acc_stride, total_tiles, tfull_bar, tempty_bar, abort_ptr);
  } else {
    // ------------------------------------------------------------ depthwise (warps 12-19, 256 threads)
    // Two groups of four warps take alternate channel blocks (group g: blocks g, g+2, ... of the CTA's sequence,
    // so group g always fills operand tile g): while one group waits for its patch or for its operand tile to be
    // free, the other computes.  In a group a thread owns two channels (packed FMAs) and a square of 4 x 4 results:
    // 36 values read for 16 results.
    reg_alloc<kDwpFilterRegs>();
    constexpr int COLS = 4, R = 4;            // columns and rows of results per thread
    constexpr int IR = R + 2, IC = COLS + 2;  // input rows and columns they need
    const int t = static_cast<int>(threadIdx.x) - 384;
    const int group = t >> 7;
    const int pair = t & 15;                                // channels 2*pair and 2*pair+1 of the block
    const int col0 = ((t >> 4) % (TW / COLS)) * COLS;       // first of the thread's columns of the tile
    const int row0 = (((t & 127) >> 4) / (TW / COLS)) * R;  // first of the thread's rows
    bool ok = true;
    const DwpClamp act(p.dw_act, p.dw_act_a, p.dw_act_b);
    const uint32_t x_first = static_cast<uint32_t>(row0 * PW + col0) * kPitch + static_cast<uint32_t>(pair) * 8u;
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
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      for (int cb = 0; cb < p.c_blocks; ++cb, ++item) {
        if ((item & 1u) != static_cast<uint32_t>(group)) continue;
        const uint32_t use_ph = (item >> 1) & 1u;  // phase of what the group uses once per item
        const uint32_t pb = item & static_cast<uint32_t>(P - 1);
        const uint32_t patch = patch_base + pb * kPatchBytes;
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
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&patch_full[pb]), (item >> patch_shift) & 1u, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
        if (!ok) break;
        uint64_t acc[R][COLS];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < COLS; ++c) acc[r][c] = bias;
        // input row i of the thread's window feeds result row r with filter row kh = i - r
#pragma unroll
        for (int i = 0; i < IR; ++i) {
          uint64_t x[IC];
#pragma unroll
          for (int j = 0; j < IC; ++j) x[j] = lds_b64(patch + x_first + static_cast<uint32_t>(i * PW + j) * kPitch);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int kh = i - r;
            if (kh < 0 || kh > 2) continue;
#pragma unroll
            for (int kw = 0; kw < 3; ++kw)
#pragma unroll
              for (int c = 0; c < COLS; ++c) f32x2_fma(acc[r][c], x[c + kw], tap[kh * 3 + kw]);
          }
        }
        // the patch has been read: it may be refilled
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&patch_empty[pb]));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          uint32_t hi[COLS], mid[COLS];
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            const float2 y = f32x2_get(acc[r][c]);
            split_bf16x2(act(y.x), act(y.y), hi[c], mid[c]);
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

// (KIND: the projection's arithmetic; bf16 pairs are the only form built.  EXPAND: the whole block; STREAMED: its weights do not stay.)
template <int KIND, int STRIDE, bool EXPAND, int EPI, bool STREAMED = false>
__global__ void __launch_bounds__(EXPAND ? kBlkThreads : kDwpThreads, 1)
tc_dw_project_kernel(const __grid_constant__ TcDwProjParams p, const __grid_constant__ CUtensorMap map_x,
                     const __grid_constant__ CUtensorMap map_x1, const __grid_constant__ CUtensorMap map_e0,
                     const __grid_constant__ CUtensorMap map_e1,
                     const __grid_constant__ CUtensorMap map_b0, const __grid_constant__ CUtensorMap map_b1) {
  if constexpr (EXPAND) tc_block_body<STRIDE, EPI, STREAMED>(p, map_x, map_x1, map_e0, map_e1, map_b0, map_b1);
  else dwp_pair_body<KIND, EPI>(p, map_x, map_b0, map_b1);
}

}  // namespace nb
