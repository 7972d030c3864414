// A whole inverted-residual block in one kernel: 1x1 "expand" convolution (+ activation) -> 3x3 depthwise convolution
// (+ activation) -> 1x1 projection (+ bias, residual, activation).  The expanded tensor and the depthwise result never
// leave the SM.
//
// The expand layer is multiplied transposed: its weights are the A operand (128 expanded channels = TMEM lanes), the
// pixels of the block's input patch the B operand (N = TMEM columns).  A depthwise thread then owns one channel and finds
// every pixel of it in its own TMEM lane: it takes the patch row by row into registers (bias, activation, zero outside the
// image), keeps the rows that the filter spans, and needs no shared memory for its input.  Its results, eight pixels of a
// channel at a time, are rows of an M-major operand tile (64 pixels of one channel = 128 bytes, 128-byte swizzle) and leave
// as 16-byte stores.
//
// A tile is a rectangle of output pixels of one image (16 x 8 at stride 1, 8 x 8 at stride 2), cut into an upper and a lower
// half; an item is one tile and 32 expanded channels.  Warps w and w + 4 of the eight depthwise warps own the TMEM quarter
// w & 3 and take the upper and lower half of the same item.  Items follow one another through the quarters: item i belongs to
// quarter i & 3 whatever the tile, so blocks of 5 x 32 channels keep four schedulers as busy as blocks of 4 x 32 do.  The
// items of one tile that fill the quarters up to the last are a set: one run of MMAs per half makes all their expanded
// pixels (the A descriptor starts so many rows ahead that every block lands in its quarter; the other lanes hold products
// that nobody reads).
//
// Warps (512 threads): 0 TMA producer (input patches; all weights once), 1 MMA issuer, 4-7 epilogue, 8-15 depthwise.  Every wait is
// bounded and ends in the status word.  Tensor memory holds the projection's accumulators, two, or one of more than 96 columns at
// stride 2, and one or two buffers of each half's expanded pixels.  Where a stride-2 block has too many weights to stay in shared memory (`stages` > 0),
// warp 2 brings a set's expand weights at a time, each block's where its quarter expects it, and warp 3 the projection's through a
// ring of blocks: two more producers, because the expand MMAs run a set ahead of the projection's and with one of them for both,
// or for the patches too, each could wait for what the other has yet to free.
//
// What bounds it: the depthwise warps' instructions (~1 500 for half an item, two warps to a scheduler, about every second
// slot), and for stride 2, whose pixels fill tensor memory once, the wait for the next set's expand MMAs.  With the expanded
// pixels in a shared-memory patch instead (two channels and a square of results to a thread) the kernel was bound by that
// memory, 80 % of its cycles with the MMAs' reads.  256 images, the patch form -> this one: 56x56x144 stride 1 289 -> 240 us,
// stride 2 184 -> 162, 28x28x192 stride 1 105 -> 94, stride 2 66 -> 53, 112x112x96 stride 2 290 -> 299: three blocks that rotate
// through the quarters are 1.5 sets a tile where one would do, and with a single buffer of expanded pixels sets wait for one another.
// Measured without gain: sixteen depthwise warps (279 us where eight take 260: what they share is the clamps' pipe), rows
// loaded one step ahead (a load takes 65 clocks), packed multiply-adds of two columns (275: the odd pairs cost moves),
// every step unrolled (474: the warps wait for instructions).
#pragma once

#include "tc_dw_common.cuh"

namespace nb {

constexpr int kBlkThreads = 512;
constexpr int kBlkMaxSlots = 8;
constexpr int kBlkMaxStages = 8;

// a half of a tile: result rows, input rows, and TMEM columns of its input pixels
__host__ __device__ constexpr int blk_half_rows(int stride) { return dwp_tile_h(stride) / 2; }
__host__ __device__ constexpr int blk_in_rows(int stride) { return (blk_half_rows(stride) - 1) * stride + 3; }
__host__ __device__ constexpr int blk_in_cols(int stride) { return (blk_in_rows(stride) * dwp_patch_w(stride) + 15) / 16 * 16; }
// one plane of an operand tile: 64 pixels x 32 channels are 4 KB
__host__ __device__ constexpr int blk_a_plane_bytes(int stride) { return dwp_tile_h(stride) * kDwpTileW / 64 * 4096; }
// the depthwise filter and bias, then the expand layer's bias
constexpr int kBlkTableRows = 11;

// One half of an item: rows of expanded pixels out of TMEM, depthwise filter, operand tile.  `release` is called once the
// last pixels are in registers.  An input row goes into the sums of all result rows that it feeds and is done with: the sums
// are carried from row to row by multiply-adds that write to another register than they read, and nothing is moved.
template <int STRIDE, class F>
__device__ __forceinline__ void blk_depthwise(uint32_t t_in, uint32_t table, int c_pad, int ch, int iy0, int h_in, uint32_t cols_in,
                                              const DwpClamp& ex_act, const DwpClamp& act, uint32_t a_at, uint32_t chunk0, F&& release) {
  using namespace ptx;
  constexpr int PW = dwp_patch_w(STRIDE), ROWS = blk_half_rows(STRIDE), IN = blk_in_rows(STRIDE);
  constexpr uint32_t kPlane = blk_a_plane_bytes(STRIDE);
  float tap[9];
  const uint32_t at = table + static_cast<uint32_t>(ch) * 4u;
#pragma unroll
  for (int k = 0; k < 9; ++k) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(tap[k]) : "r"(at + static_cast<uint32_t>(k * c_pad) * 4u));
  float bias, ex_bias;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(bias) : "r"(at + static_cast<uint32_t>(9 * c_pad) * 4u));
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(ex_bias) : "r"(at + static_cast<uint32_t>(10 * c_pad) * 4u));
  const uint64_t ex_bias2 = f32x2_make(__float_as_uint(ex_bias), __float_as_uint(ex_bias));
  auto fetch = [&](int row, uint32_t (&v)[PW]) {
    const uint32_t t = t_in + static_cast<uint32_t>(row * PW);
    tmem_ld8(t, v);
    if constexpr (STRIDE == 1) {
      tmem_ld2(t + 8u, v + 8);
    } else {
      tmem_ld8(t + 8u, v + 8);
      tmem_ld1(t + 16u, v + 16);
    }
  };
  // (a row and a column of pixels are the same for the whole warp: these branches do not split it)
  auto finish = [&](int row, uint32_t (&v)[PW]) {
    const int iy = iy0 + row;
    if (iy < 0 || iy >= h_in) {
#pragma unroll
      for (int j = 0; j < PW; ++j) v[j] = 0u;
      return;
    }
#pragma unroll
    for (int j = 0; j + 1 < PW; j += 2) {
      uint64_t u;
      f32x2_add(u, f32x2_make(v[j], v[j + 1]), ex_bias2);
      const float2 f = f32x2_get(u);
      v[j] = __float_as_uint(ex_act(f.x));
      v[j + 1] = __float_as_uint(ex_act(f.y));
    }
    if (PW % 2 == 1) v[PW - 1] = __float_as_uint(ex_act(__fadd_rn(__uint_as_float(v[PW - 1]), ex_bias)));
    if (cols_in != (1u << PW) - 1u) {
#pragma unroll
      for (int j = 0; j < PW; ++j)
        if (!(cols_in >> j & 1u)) v[j] = 0u;
    }
  };
  uint32_t to_chunk = 0;
  auto put = [&](const float (&y)[8]) {
    uint32_t w_hi[4], w_mid[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      split_bf16x2(act(y[2 * c]), act(y[2 * c + 1]), w_hi[c], w_mid[c]);
    // eight pixels of a row are one 16-byte chunk of the channel's 128 bytes, at chunk ^ (channel & 7)
    const uint32_t to = a_at + (chunk0 ^ to_chunk);
    to_chunk += 16u;
    sts_16b(to, w_hi);
    sts_16b(to + kPlane, w_mid);
  };
  if constexpr (STRIDE == 1) {
    float sum_a[8], sum_b[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) sum_a[c] = sum_b[c] = bias;
#pragma unroll 1  // (one copy: warps at different places of longer code wait for instructions)
    for (int t = 0; t < IN; t += 2) {
      uint32_t x[2][PW];
      fetch(t, x[0]);
      fetch(t + 1, x[1]);
      tmem_ld_wait();
      if (t + 2 == IN) release();
      finish(t, x[0]);
      finish(t + 1, x[1]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float out[8];
#pragma unroll
        for (int kw = 0; kw < 3; ++kw)
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float v = __uint_as_float(x[i][c + kw]);
            out[c] = fmaf(v, tap[6 + kw], kw == 0 ? sum_b[c] : out[c]);
            sum_b[c] = fmaf(v, tap[3 + kw], kw == 0 ? sum_a[c] : sum_b[c]);
            sum_a[c] = fmaf(v, tap[kw], kw == 0 ? bias : sum_a[c]);
          }
        if (t > 0) put(out);
      }
    }
  } else {
    float sum_b[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) sum_b[c] = bias;
    uint32_t x[2][PW];
#pragma unroll 1
    for (int r = 0; r <= ROWS; ++r) {
      fetch(2 * r, x[0]);
      if (r < ROWS) fetch(2 * r + 1, x[1]);
      tmem_ld_wait();
      if (r == ROWS) release();
      finish(2 * r, x[0]);
      if (r > 0) {
        float out[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) out[c] = fmaf(__uint_as_float(x[0][2 * c]), tap[6], sum_b[c]);
#pragma unroll
        for (int c = 0; c < 8; ++c) out[c] = fmaf(__uint_as_float(x[0][2 * c + 1]), tap[7], out[c]);
#pragma unroll
        for (int c = 0; c < 8; ++c) out[c] = fmaf(__uint_as_float(x[0][2 * c + 2]), tap[8], out[c]);
        put(out);
      }
      if (r == ROWS) break;
      finish(2 * r + 1, x[1]);
#pragma unroll
      for (int c = 0; c < 8; ++c) sum_b[c] = fmaf(__uint_as_float(x[0][2 * c]), tap[0], bias);
#pragma unroll
      for (int k = 1; k < 6; ++k)
#pragma unroll
        for (int c = 0; c < 8; ++c) sum_b[c] = fmaf(__uint_as_float(x[k / 3][2 * c + k % 3]), tap[k], sum_b[c]);
    }
  }
}

// (STREAMED: weights that do not stay; in the same code the branches cost the issuing thread 2 to 3 % of every stride-2 block)
template <int STRIDE, int EPI, bool STREAMED>
__device__ __forceinline__ void tc_block_body(const TcDwProjParams& p, const CUtensorMap& map_x, const CUtensorMap& map_x1,
                                              const CUtensorMap& map_e0, const CUtensorMap& map_e1, const CUtensorMap& map_b0,
                                              const CUtensorMap& map_b1) {
  using namespace ptx;
  constexpr int TH = dwp_tile_h(STRIDE), TW = kDwpTileW;
  constexpr int PW = dwp_patch_w(STRIDE), NPX = dwp_patch_h(STRIDE) * PW;
  constexpr int HALF = blk_half_rows(STRIDE), COLS = blk_in_cols(STRIDE);
  constexpr uint32_t kAPlane = blk_a_plane_bytes(STRIDE);
  grid_dependency_trigger();  // the next kernel of the stream may begin its preamble

  extern __shared__ uint8_t dwp_smem_raw[];
  __shared__ __align__(8) uint64_t x_full[2], x_empty[2], w_full;  // (w_full, w_empty: all weights, or a set's expand weights)
  __shared__ __align__(8) uint64_t w_empty, b_full[kBlkMaxStages], b_empty[kBlkMaxStages];
  __shared__ __align__(8) uint64_t e_full[4], e_empty[4];  // [half][buffer]
  __shared__ __align__(8) uint64_t a_full[kBlkMaxSlots], a_empty[kBlkMaxSlots];
  __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // the same in all lanes, and known to be
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(dwp_smem_raw) + 1023u) & ~1023u;
  const int c_blocks = p.c_blocks, c_pad = c_blocks * kDwpChannels;
  const uint32_t x_plane = static_cast<uint32_t>(p.x_plane_bytes), x_row = static_cast<uint32_t>(p.x_row_bytes);
  const int XB = p.x_bufs, NB = p.e_bufs;
  const uint32_t slots = static_cast<uint32_t>(p.a_slots);  // 4 or 8
  const uint32_t slot_shift = slots == 8u ? 3u : 2u;
  // input patches (hi, mid planes), expand weights, operand tiles, projection weights, the epilogue's, tables.  (An expand
  // MMA may read up to 96 weight rows ahead of a plane or behind it: the patches lie before, the operand tiles behind.)
  const uint32_t x_base = smem_base;
  const uint32_t e_plane = static_cast<uint32_t>(STREAMED ? 4 * kDwpChannels : c_pad) * x_row;
  const uint32_t e_base = x_base + static_cast<uint32_t>(XB) * 2u * x_plane;
  const uint32_t a_base = e_base + 2u * e_plane;
  const uint32_t b_bytes = static_cast<uint32_t>(p.b_bytes);
  const uint32_t b_base = a_base + slots * 2u * kAPlane;
  const uint32_t drain = b_base + static_cast<uint32_t>(STREAMED ? p.stages : c_blocks) * 2u * b_bytes;
  const uint32_t table = drain + static_cast<uint32_t>(TH * TW / 32) * kDrainWarpBytes;
  // TMEM columns: the projection's accumulators, then the halves' expanded pixels
  const uint32_t acc_stride = static_cast<uint32_t>(p.block_n);
  const uint32_t e_col0 = static_cast<uint32_t>(p.accs) * acc_stride;
  const int total_tiles = p.images * p.tiles_y * p.tiles_x;
  // With one block of channels a tile is one item, and a single buffer lets no second one run beside it: its halves then go to
  // quarters two apart, so that their two warps have a scheduler each (28x28x32 -> 48 at stride 2, 3 281 images: 698 -> 651 us).
  const int apart = c_blocks == 1 ? 2 : 0;
  const uint32_t e_tx = 2u * kDwpChannels * x_row, b_tx = 2u * static_cast<uint32_t>(p.block_n) * 64u;  // a block's weights
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&x_full[i]), 1);
      mbar_init(smem_u32(&x_empty[i]), 1);  // the commit after the tile's last expand MMA
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 4);
    }
    mbar_init(smem_u32(&w_full), 1);
    if constexpr (STREAMED) {
      mbar_init(smem_u32(&w_empty), 1);
      for (int i = 0; i < kBlkMaxStages; ++i) {
        mbar_init(smem_u32(&b_full[i]), 1);
        mbar_init(smem_u32(&b_empty[i]), 1);
      }
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&e_full[i]), 1);
      mbar_init(smem_u32(&e_empty[i]), 4);  // the half's four warps, those without an item in the set too
    }
    for (int i = 0; i < kBlkMaxSlots; ++i) {
      mbar_init(smem_u32(&a_full[i]), 2);  // the two halves
      mbar_init(smem_u32(&a_empty[i]), 1);
    }
    fence_mbar_init();
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_x1);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), kTcTmemCols);
    tmem_relinquish();
  }
  // (constants of the layers, not results of the kernel before: they may be read ahead of the dependency wait; zero past C)
  for (int i = static_cast<int>(threadIdx.x); i < kBlkTableRows * c_pad; i += kBlkThreads) {
    const int k = i / c_pad, c = i - k * c_pad;
    float v = 0.0f;
    if (c < p.C) {
      if (k < 9) v = __ldg(p.dw_weights + static_cast<size_t>(k) * p.C + c);
      else if (k == 9) v = p.dw_bias != nullptr ? __ldg(p.dw_bias + c) : 0.0f;
      else v = p.ex_bias != nullptr ? __ldg(p.ex_bias + c) : 0.0f;
    }
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(table + static_cast<uint32_t>(i) * 4u), "f"(v) : "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  if (warp != 0) grid_dependency_wait();  // (the producer waits once the weights are under way)

  if (warp == 0) {
    // ------------------------------------------------------------ producer (one elected thread: tc_gemm.cuh says why)
    if (elect_one() && static_cast<int>(blockIdx.x) < total_tiles) {
      const uint32_t wb = smem_u32(&w_full);
      if (!STREAMED) mbar_arrive_expect_tx(wb, static_cast<uint32_t>(c_blocks) * (e_tx + b_tx));
      for (int cb = 0; cb < c_blocks && !STREAMED; ++cb) {
        const uint32_t e_at = e_base + static_cast<uint32_t>(cb * kDwpChannels) * x_row;
        tma_load_2d(e_at, &map_e0, wb, 0, cb * kDwpChannels);
        tma_load_2d(e_at + e_plane, &map_e1, wb, 0, cb * kDwpChannels);
        const uint32_t b_at = b_base + static_cast<uint32_t>(cb) * 2u * b_bytes;
        tma_load_2d(b_at, &map_b0, wb, cb * kDwpChannels, 0);
        tma_load_2d(b_at + b_bytes, &map_b1, wb, cb * kDwpChannels, 0);
      }
      grid_dependency_wait();
      const uint32_t x_tx = 2u * static_cast<uint32_t>(NPX) * x_row;
      DwpWalk w(p, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
      int xb = 0;
      uint32_t x_ph = 0;
      long long issued = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, w.on(p)) {
        if (!mbar_wait_bounded(smem_u32(&x_empty[xb]), x_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
          ok = false;
          break;
        }
        const uint32_t fb = smem_u32(&x_full[xb]), dst = x_base + static_cast<uint32_t>(xb) * 2u * x_plane;
        const int ix = w.x * TW * STRIDE - p.pad_l, iy = w.y * TH * STRIDE - p.pad_t;
        mbar_arrive_expect_tx(fb, x_tx);
        tma_load_4d(dst, &map_x, fb, 0, ix, iy, w.img);
        tma_load_4d(dst + x_plane, &map_x1, fb, 0, ix, iy, w.img);
        ++issued;
        if (++xb == XB) {
          xb = 0;
          x_ph ^= 1u;
        }
      }
      if (!ok) {
        if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      }
      if (*abort_ptr != 0) {
        // copies issued by this thread may still be landing: wait (bounded) for the last ones
        int zero = 0;
        if (!STREAMED) mbar_wait_bounded(wb, 0u, &zero, 200000000ull);
        for (long long i = issued > XB ? issued - XB : 0; i < issued; ++i)
          mbar_wait_bounded(smem_u32(&x_full[i % XB]), static_cast<uint32_t>((i / XB) & 1), &zero, 200000000ull);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (elect_one() && static_cast<int>(blockIdx.x) < total_tiles) {
      const uint32_t idesc_e = instr_desc(1u, 1u, kTcBlockM, COLS);
      const uint32_t idesc = instr_desc(1u, 1u, kTcBlockM, static_cast<uint32_t>(p.block_n)) | kInstrAMnMajor;
      const uint64_t fixed_x = smem_desc_kmajor(0u, x_row), fixed_b = smem_desc_kmajor(0u, 64u);
      // (a stride-2 tile has 64 rows: its second 64 are the first once more, into accumulator rows that nobody reads)
      const uint64_t a_first = smem_desc_mnmajor(a_base, STRIDE == 1 ? 4096u : 0u, 1024u);
      const int my_tiles = (total_tiles - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1;
      bool ok = STREAMED || mbar_wait_bounded(smem_u32(&w_full), 0u, abort_ptr, kTcWaitLimitNs);
      // expand: the next set in order
      int e_tiles = 0, e_cb = 0, xb = 0, eb = 0;
      uint32_t e_item = 0, x_ph = 0, e_ph = 0, w_ph = 0;
      auto issue_expand = [&]() -> bool {
        if (e_tiles == my_tiles) return true;  // (the last sets have no successors)
        if (e_cb == 0 && !mbar_wait_bounded(smem_u32(&x_full[xb]), x_ph, abort_ptr, kTcWaitLimitNs)) return false;
        const int q0 = static_cast<int>(e_item & 3u);
        const int count = min(4 - q0, c_blocks - e_cb);
        if (STREAMED && !mbar_wait_bounded(smem_u32(&w_full), w_ph, abort_ptr, kTcWaitLimitNs)) return false;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          // the rows of block e_cb in its quarter: the operand starts so many blocks ahead of it
          const uint32_t wa = STREAMED ? e_base : e_base + static_cast<uint32_t>((e_cb - ((q0 + h * apart) & 3)) * kDwpChannels) * x_row;
          const uint64_t w0 = fixed_x + ((wa & 0x3ffffu) >> 4), w1 = w0 + (e_plane >> 4);
          if (!mbar_wait_bounded(smem_u32(&e_empty[h * 2 + eb]), e_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) return false;
          tc_fence_after_sync();
          const uint32_t xa = x_base + static_cast<uint32_t>(xb) * 2u * x_plane + static_cast<uint32_t>(h * HALF * STRIDE * PW) * x_row;
          const uint64_t x0 = fixed_x + ((xa & 0x3ffffu) >> 4), x1 = x0 + (x_plane >> 4);
          const uint32_t d = tmem_base + e_col0 + static_cast<uint32_t>((h * NB + eb) * COLS);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if (k >= p.ex_ksteps) break;  // (16 input channels: the second half of the 64-byte rows is zero padding)
            mma_f16(d, w0 + 2u * k, x1 + 2u * k, idesc_e, k ? 1u : 0u);  // the input's mid * hi
            mma_f16(d, w1 + 2u * k, x0 + 2u * k, idesc_e, 1u);           // its hi * mid
            mma_f16(d, w0 + 2u * k, x0 + 2u * k, idesc_e, 1u);           // hi * hi
          }
          tc_commit(smem_u32(&e_full[h * 2 + eb]));
        }
        if (STREAMED) {
          tc_commit(smem_u32(&w_empty));
          w_ph ^= 1u;
        }
        if (++eb == NB) {
          eb = 0;
          e_ph ^= 1u;
        }
        e_item += static_cast<uint32_t>(count);
        e_cb += count;
        if (e_cb == c_blocks) {
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
      for (int i = 0; i < NB && ok; ++i) ok = issue_expand();
      int acc = 0, bs = 0;
      uint32_t acc_ph = 0, item = 0, b_ph = 0;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        if (!mbar_wait_bounded(smem_u32(&tempty_bar[acc]), acc_ph ^ 1u, abort_ptr, kTcWaitLimitNs)) {
          ok = false;
          break;
        }
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc) * acc_stride;
        uint32_t accumulate = 0u;
        for (int cb = 0; cb < c_blocks && ok;) {
          const int count = min(4 - static_cast<int>(item & 3u), c_blocks - cb);
          // A set after this one is expanded as soon as this one's pixels have been taken, before its projection (56x56x144,
          // 256 images: 260 -> 240 us).  With an operand tile for each quarter only, the depthwise warps wait for the
          // projection, which then goes first where a second buffer allows (28x28x192: 94 us, 109 the other way).
          const bool expand_first = NB == 1 || slots == 8u;
          if (expand_first) ok = issue_expand();
          for (int i = 0; i < count && ok; ++i, ++item, ++cb) {
            const uint32_t slot = item & (slots - 1u);
            if (!mbar_wait_bounded(smem_u32(&a_full[slot]), (item >> slot_shift) & 1u, abort_ptr, kTcWaitLimitNs) ||
                (STREAMED && !mbar_wait_bounded(smem_u32(&b_full[bs]), b_ph, abort_ptr, kTcWaitLimitNs))) {
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint64_t a0 = a_first + static_cast<uint64_t>(slot * 2u * (kAPlane >> 4));
            const uint64_t b0 = fixed_b + (((b_base + static_cast<uint32_t>(STREAMED ? bs : cb) * 2u * b_bytes) & 0x3ffffu) >> 4);
            const uint64_t b1 = b0 + (b_bytes >> 4);
#pragma unroll
            for (int k = 0; k < 2; ++k) {  // two K steps of 16 channels: 2 KB of A, 32 bytes of a row of B
              const uint64_t ka = a0 + 128u * k, kb = 2u * k;
              mma_f16(d_tmem, ka + (kAPlane >> 4), b0 + kb, idesc, accumulate);  // mid * hi
              mma_f16(d_tmem, ka, b1 + kb, idesc, 1u);                           // hi * mid
              mma_f16(d_tmem, ka, b0 + kb, idesc, 1u);                           // hi * hi
              accumulate = 1u;
            }
            tc_commit(smem_u32(&a_empty[slot]));
            if (STREAMED) {
              tc_commit(smem_u32(&b_empty[bs]));
              if (++bs == p.stages) {
                bs = 0;
                b_ph ^= 1u;
              }
            }
          }
          if (!expand_first && ok) ok = issue_expand();
        }
        if (!ok) break;
        tc_commit(smem_u32(&tfull_bar[acc]));
        if (p.accs == 2) acc ^= 1;
        if (acc == 0) acc_ph ^= 1u;
      }
      if (!ok) {
        if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_MMA);
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ producer of a set's expand weights
    if (STREAMED && elect_one()) {
      const uint32_t full = smem_u32(&w_full);
      uint32_t item = 0, ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x)
        for (int cb = 0; cb < c_blocks;) {
          const int q0 = static_cast<int>(item & 3u);
          const int count = min(4 - q0, c_blocks - cb);
          ok = mbar_wait_bounded(smem_u32(&w_empty), ph ^ 1u, abort_ptr, kTcWaitLimitNs);
          if (!ok) break;
          mbar_arrive_expect_tx(full, static_cast<uint32_t>(count) * e_tx);
          for (int i = 0; i < count; ++i) {
            const uint32_t at = e_base + static_cast<uint32_t>((q0 + i) * kDwpChannels) * x_row;
            tma_load_2d(at, &map_e0, full, 0, (cb + i) * kDwpChannels);
            tma_load_2d(at + e_plane, &map_e1, full, 0, (cb + i) * kDwpChannels);
          }
          ph ^= 1u;
          item += static_cast<uint32_t>(count);
          cb += count;
        }
      if (!ok) {
        if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      }
      int zero = 0;
      if (*abort_ptr != 0 && item > 0) mbar_wait_bounded(full, ph ^ 1u, &zero, 200000000ull);  // the last set's copies may still be landing
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------ producer of the projection's weights, a block to a stage
    if (STREAMED && elect_one()) {
      const int S = p.stages;
      int s = 0;
      uint32_t ph = 0;
      long long issued = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x)
        for (int cb = 0; cb < c_blocks; ++cb) {
          ok = mbar_wait_bounded(smem_u32(&b_empty[s]), ph ^ 1u, abort_ptr, kTcWaitLimitNs);
          if (!ok) break;
          const uint32_t full = smem_u32(&b_full[s]), at = b_base + static_cast<uint32_t>(s) * 2u * b_bytes;
          mbar_arrive_expect_tx(full, b_tx);
          tma_load_2d(at, &map_b0, full, cb * kDwpChannels, 0);
          tma_load_2d(at + b_bytes, &map_b1, full, cb * kDwpChannels, 0);
          ++issued;
          if (++s == S) {
            s = 0;
            ph ^= 1u;
          }
        }
      if (!ok) {
        if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      }
      int zero = 0;
      for (long long i = *abort_ptr != 0 && issued > S ? issued - S : 0; *abort_ptr != 0 && i < issued; ++i)
        mbar_wait_bounded(smem_u32(&b_full[i % S]), static_cast<uint32_t>((i / S) & 1), &zero, 200000000ull);
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------ epilogue
    dwp_epilogue<GEMM_BF16X3, STRIDE, EPI>(p, 1, 0, warp & 3, drain, tmem_base, acc_stride, total_tiles, tfull_bar, tempty_bar, abort_ptr);
  } else {
    // ------------------------------------------------------------ depthwise
    const int q = warp & 3, h = (warp - 8) >> 2;
    const DwpClamp act(p.dw_act, p.dw_act_a, p.dw_act_b), ex_act(p.ex_act, p.ex_act_a, p.ex_act_b);
    // this thread's channel in an operand tile: eight channels to an atom; the half's 64 pixels (stride 2: its half of them)
    const uint32_t a_at = a_base + static_cast<uint32_t>(STRIDE == 1 ? h * 4096 : 0) + static_cast<uint32_t>((lane >> 3) * 1024 + (lane & 7) * 128);
    const uint32_t chunk0 = static_cast<uint32_t>(((lane & 7) ^ (STRIDE == 1 ? 0 : h * 4)) << 4);
    uint32_t item = 0, e_ph = 0;
    int eb = 0;
    bool ok = true;
    DwpWalk w(p, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, w.on(p)) {
      const int iy0 = (w.y * TH + h * HALF) * STRIDE - p.pad_t, ix0 = w.x * TW * STRIDE - p.pad_l;
      // which columns of the patch lie in the image
      const int left = max(0, -ix0), right = min(PW, p.Win - ix0);
      const uint32_t cols_in = right > left ? ((1u << right) - 1u) & ~((1u << left) - 1u) : 0u;
      for (int cb = 0; cb < c_blocks;) {
        const int q0 = static_cast<int>((item + static_cast<uint32_t>(h * apart)) & 3u);
        const int count = min(4 - q0, c_blocks - cb);
        const uint32_t full = smem_u32(&e_full[h * 2 + eb]), empty = smem_u32(&e_empty[h * 2 + eb]);
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(full, e_ph, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
        if (!ok) break;
        auto release = [&]() {
          // the pixels have been read: the expand MMAs of a later set may overwrite them
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(empty);
          __syncwarp();
        };
        if (q < q0 || q >= q0 + count) {
          release();
        } else {
          tc_fence_after_sync();
          const uint32_t mine = item + static_cast<uint32_t>(q - q0);
          const uint32_t slot = mine & (slots - 1u);
          // the operand tile's last user must have consumed it (one vote behind each wait: it brings the warp together)
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&a_empty[slot]), ((mine >> slot_shift) & 1u) ^ 1u, abort_ptr, kTcWaitLimitNs) ? 1 : 0) != 0;
          if (!ok) break;
          const uint32_t t_in = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + e_col0 + static_cast<uint32_t>((h * NB + eb) * COLS);
          blk_depthwise<STRIDE>(t_in, table, c_pad, (cb + q - q0) * kDwpChannels + lane, iy0, p.Hin, cols_in, ex_act, act,
                                a_at + slot * 2u * kAPlane, chunk0, release);
          fence_proxy_async_smem();  // the tensor core reads what these stores wrote
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&a_full[slot]));
          __syncwarp();
        }
        item += static_cast<uint32_t>(count);
        cb += count;
        if (++eb == NB) {
          eb = 0;
          e_ph ^= 1u;
        }
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
