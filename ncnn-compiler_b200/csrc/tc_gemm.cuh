// Tensor-core contraction kernel for sm_100a: out[M,N] = epilogue(A[M,K] * B[N,K]^T).
//
// One kernel serves Convolution (A rows are output pixels gathered from an NHWC
// activation tensor by TMA im2col loads, K runs over filter taps x input
// channels), InnerProduct and Gemm (A is a plain row-major matrix loaded by
// tiled TMA).  B is always the packed weight matrix [N][K], K contiguous.
//
// Pipeline per CTA (persistent, one CTA per SM, 352 threads):
//   warps 0,6  TMA producers (A tiles / B tiles): fill a ring of shared-memory stages
//              (A tile 128 x K-block, B tile block_n x K-block, 128B/64B-swizzled rows)
//   warp 1     MMA issuer: tcgen05.mma from shared memory into one of four TMEM
//              accumulators (128 lanes x block_n fp32/int32 columns), or two pairs of them
//   warps 2-5, 7-10  epilogue: tcgen05.ld of the finished accumulator, then bias, residual,
//              activation, dequantise/requantise, store (tc_epilogue.cuh)
// The epilogue of tile i overlaps the main loops of the tiles after it.
//
// Arithmetic kinds:
//   GEMM_TF32    one kind::tf32 MMA per K step (fast mode, ~1e-3 relative error)
//   GEMM_TF32X3  operands are stored as hi/lo tf32 planes (x = hi + lo exactly);
//                three MMAs lo*hi + hi*lo + hi*hi recover ~fp32 accuracy
//   GEMM_BF16X3  operands are stored as two bf16 planes (x ~ hi + mid, 16 significant bits);
//                three kind::f16 MMAs mid*hi + hi*mid + hi*hi, each at twice the tf32 rate
//                on half the operand bytes, give ~1e-5 relative error
//   GEMM_I8      kind::i8, int32 accumulation, exact
#pragma once

#include "tc_epilogue.cuh"

namespace nb {

// Results of any alignment, element by element (rows that are no multiple of 16 bytes).
// BF16IO: a bf16-pair tensor takes part (as output or residual); kept out of the other
// instantiation so that the int8 and plain fp32 epilogues stay lean.
template <int KIND, bool BF16IO, bool SIDE = false>
__device__ __forceinline__ void tc_epilogue_chunk(const TcGemmParams& p, const uint32_t (&v)[16],
                                                  long long m, int n_first, const float* tile_bias,
                                                  const float* tile_scale) {
  float y[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int n = n_first + j;
    float t;
    if (n < p.N) {
      if (KIND == GEMM_I8) {
        t = __fmul_rn(static_cast<float>(static_cast<int>(v[j])), tile_scale[j]);
      } else {
        t = __uint_as_float(v[j]);
      }
      if (p.bias != nullptr) t = __fadd_rn(t, tile_bias[j]);
    } else {
      t = 0.0f;
    }
    y[j] = t;
  }
  const long long row = m * p.ldo;
  const bool vec4 = (p.ldo % 4 == 0) && (n_first % 4 == 0);
  if (BF16IO && p.res_mode == RES_BF16X2) {
    const uint16_t* r0 = reinterpret_cast<const uint16_t*>(p.res0);
    const uint16_t* r1 = reinterpret_cast<const uint16_t*>(p.res1);
    if ((p.ldo % 8 == 0) && n_first + 15 < p.N) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(r0 + row + n_first + 8 * g));
        const uint4 b = __ldg(reinterpret_cast<const uint4*>(r1 + row + n_first + 8 * g));
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          y[8 * g + 2 * e] = __fadd_rn(y[8 * g + 2 * e], __fadd_rn(bf16_low(aw[e]), bf16_low(bw[e])));
          y[8 * g + 2 * e + 1] = __fadd_rn(y[8 * g + 2 * e + 1], __fadd_rn(bf16_high(aw[e]), bf16_high(bw[e])));
        }
      }
    } else {
      for (int j = 0; j < 16; ++j)
        if (n_first + j < p.N)
          y[j] = __fadd_rn(y[j], __fadd_rn(__uint_as_float(static_cast<uint32_t>(r0[row + n_first + j]) << 16),
                                           __uint_as_float(static_cast<uint32_t>(r1[row + n_first + j]) << 16)));
    }
  } else if (p.res0 != nullptr) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int n = n_first + 4 * g;
      if (vec4 && n + 3 < p.N) {
        float4 r = __ldg(reinterpret_cast<const float4*>(p.res0 + row + n));
        if (p.res1 != nullptr) {
          const float4 l = __ldg(reinterpret_cast<const float4*>(p.res1 + row + n));
          r.x = __fadd_rn(r.x, l.x);
          r.y = __fadd_rn(r.y, l.y);
          r.z = __fadd_rn(r.z, l.z);
          r.w = __fadd_rn(r.w, l.w);
        }
        y[4 * g + 0] = __fadd_rn(y[4 * g + 0], r.x);
        y[4 * g + 1] = __fadd_rn(y[4 * g + 1], r.y);
        y[4 * g + 2] = __fadd_rn(y[4 * g + 2], r.z);
        y[4 * g + 3] = __fadd_rn(y[4 * g + 3], r.w);
      } else {
        for (int e = 0; e < 4; ++e) {
          if (n + e < p.N) {
            float r = __ldg(p.res0 + row + n + e);
            if (p.res1 != nullptr) r = __fadd_rn(r, __ldg(p.res1 + row + n + e));
            y[4 * g + e] = __fadd_rn(y[4 * g + e], r);
          }
        }
      }
    }
  }
  if (p.out_mode == OUT_I8) {
    int q[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      int t = quantize_rha(y[j], p.out_scale);
      if (p.act == ACT_RELU) t = max(t, 0);
      q[j] = t;
    }
    if ((p.ldo % 16 == 0) && (n_first % 16 == 0) && n_first + 15 < p.N) {
      uint32_t w[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        w[g] = (static_cast<uint32_t>(q[4 * g + 0]) & 0xffu) |
               ((static_cast<uint32_t>(q[4 * g + 1]) & 0xffu) << 8) |
               ((static_cast<uint32_t>(q[4 * g + 2]) & 0xffu) << 16) |
               ((static_cast<uint32_t>(q[4 * g + 3]) & 0xffu) << 24);
      }
      *reinterpret_cast<uint4*>(p.outq + row + n_first) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      for (int j = 0; j < 16; ++j)
        if (n_first + j < p.N) p.outq[row + n_first + j] = static_cast<int8_t>(q[j]);
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) y[j] = apply_act(y[j], p.act, p.act_a, p.act_b);
  if (SIDE && p.side_count > 0) {
    tc_store_side_quant(p.side_q0 + m * p.side_ld + n_first, p.side_scale0, y);
    if (p.side_count > 1) tc_store_side_quant(p.side_q1 + m * p.side_ld + n_first, p.side_scale1, y);
  }
  if (BF16IO && p.out_mode == OUT_BF16X2) {
    uint16_t* o0 = reinterpret_cast<uint16_t*>(p.out0);
    uint16_t* o1 = reinterpret_cast<uint16_t*>(p.out1);
    uint32_t hi[8], mid[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) split_bf16x2(y[2 * e], y[2 * e + 1], hi[e], mid[e]);
    if ((p.ldo % 8 == 0) && n_first + 15 < p.N) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        *reinterpret_cast<uint4*>(o0 + row + n_first + 8 * g) =
            make_uint4(hi[4 * g], hi[4 * g + 1], hi[4 * g + 2], hi[4 * g + 3]);
        *reinterpret_cast<uint4*>(o1 + row + n_first + 8 * g) =
            make_uint4(mid[4 * g], mid[4 * g + 1], mid[4 * g + 2], mid[4 * g + 3]);
      }
    } else {
      for (int j = 0; j < 16; ++j) {
        if (n_first + j < p.N) {
          o0[row + n_first + j] = static_cast<uint16_t>(j & 1 ? hi[j >> 1] >> 16 : hi[j >> 1] & 0xffffu);
          o1[row + n_first + j] = static_cast<uint16_t>(j & 1 ? mid[j >> 1] >> 16 : mid[j >> 1] & 0xffffu);
        }
      }
    }
    return;
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int n = n_first + 4 * g;
    float hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float t = y[4 * g + e];
      if (p.out_mode == OUT_F32) {
        hi[e] = t;
        lo[e] = 0.0f;
      } else {
        hi[e] = round_tf32(t);
        lo[e] = __fadd_rn(t, -hi[e]);
      }
    }
    if (vec4 && n + 3 < p.N) {
      *reinterpret_cast<float4*>(p.out0 + row + n) = make_float4(hi[0], hi[1], hi[2], hi[3]);
      if (p.out_mode == OUT_F32_SPLIT)
        *reinterpret_cast<float4*>(p.out1 + row + n) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    } else {
      for (int e = 0; e < 4; ++e) {
        if (n + e < p.N) {
          p.out0[row + n + e] = hi[e];
          if (p.out_mode == OUT_F32_SPLIT) p.out1[row + n + e] = lo[e];
        }
      }
    }
  }
}

// SIDE: the instantiation that also writes int8 copies of its fp32 result (TcGemmParams::side_q); kept out
// of the plain kernel so that layers without such copies run exactly the code they ran before.
template <int KIND, int EPI, bool SIDE = false>
__global__ void __launch_bounds__(kTcThreads, 1)
tc_gemm_kernel(const __grid_constant__ TcGemmParams p, const __grid_constant__ CUtensorMap map_a0,
               const __grid_constant__ CUtensorMap map_a1,
               const __grid_constant__ CUtensorMap map_b0,
               const __grid_constant__ CUtensorMap map_b1) {
  using namespace ptx;
  grid_dependency_trigger();  // the next kernel of the stream may begin its preamble
  constexpr int PLANES = tc_planes(KIND);

  extern __shared__ uint8_t tc_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kTcMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kTcMaxStages];
  __shared__ __align__(8) uint64_t tfull_bar[4];
  __shared__ __align__(8) uint64_t tempty_bar[4];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  // (the shuffle tells the compiler that the warp number is the same in all lanes: see the issuing roles below)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
  const uint32_t slot = static_cast<uint32_t>(kTcBlockM) * p.row_bytes;
  const uint32_t stage_bytes = static_cast<uint32_t>(p.stage_bytes);
  const int AS = p.pair ? 2 : 1;  // A tiles per stage
  const uint32_t b_slot = (stage_bytes / PLANES) - static_cast<uint32_t>(AS) * slot;  // B tile, rounded to 1 KB
  const int S = p.stages;
  // int8 K blocks are small (two MMAs over 12 KB for 64 channels): a stage holds SUB of them, so that the
  // ~450 cycles of arming and releasing a stage are paid once per SUB blocks
  const int SUB = KIND == GEMM_I8 ? (p.sub_blocks > 1 ? p.sub_blocks : 1) : 1;
  const int k_groups = p.k_blocks / SUB;
  const int taps = p.k_blocks / p.c_blocks;  // K runs over channel blocks, then the taps of one (plain matrices: one tap)
  // a unit of work is a tile, or one chunk of its K blocks
  constexpr bool CHUNKS = KIND == GEMM_BF16X3 || KIND == GEMM_I8;  // (int8: on different CTAs only)
  const int chunks = CHUNKS ? p.chunks : 1;
  const bool split_k = CHUNKS && p.split_k != 0;
  const int chunk_groups = chunks > 1 ? p.chunk_blocks : k_groups;  // (such contractions have one K block per stage)
  const int units = p.tiles_m * p.tiles_n * (split_k ? chunks : 1);
  // 512 TMEM columns: four accumulators (of a shallow contraction several tiles are in the pipeline at once), two
  // pairs of them, or three and the running sum of the chunks
  const int accs = chunks > 1 ? 3 : (p.pair ? 2 : 4);
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 2);  // one arrival per producer warp
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&tfull_bar[i]), 1);
      mbar_init(smem_u32(&tempty_bar[i]), 8);  // every epilogue warp
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
    tmem_alloc(smem_u32(&tmem_slot), kTcTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  // Fault injection for the time-out path (host tests only; status[1] is zero in production): the first
  // tile's first stage is never armed, so the MMA issuer's bounded wait on it runs out, every role leaves
  // through the abort path, and the host reads status 7.  The limit shrinks to 2 ms for such a run.  (Read before the
  // wait below, so that no copy waits for it; the host changes the word only while nothing runs.)
  const int test_stall = p.status[1];
  const uint64_t wait_limit = test_stall ? 2000000ull : kTcWaitLimitNs;
  // barriers, tensor memory and descriptors are ready: from here on the kernel touches tensors that the
  // kernel before it in the stream may still be writing.  The producers wait later, see below.
  if (warp != 0 && warp != 6) grid_dependency_wait();

  if (warp == 0 || warp == 6) {
    // ------------------------------------------------------------ producers
    // warp 0 feeds the A tiles, warp 6 the B tiles, each arming the stage for its own bytes (the full barrier
    // counts two arrivals).  The issuing roles (these two and the MMA warp) run in one thread picked by
    // elect.sync under a warp number that is the same in all lanes: TMA and tcgen05 instructions take their
    // operands from uniform registers, and only then can the compiler keep descriptors and coordinates there.
    // Chosen by `lane == 0` instead, every instruction first moves its operands over, one by one: 54 (unrolled)
    // to 148 clocks between narrow MMAs against 40-64, which is the tensor pipe's own pace.
    // No kernel writes weights, so the B producer fills the ring while the kernel before this one still runs, and waits
    // for that kernel before it waits for a stage to come free (whose limit must not count other kernels' time); the A
    // producer has its first coordinates ready when it waits.  With the drain's operands fetched ahead (tc_drain), whole passes:
    // ResNet-18, one image 355 -> 333 us, int8, 256 images 1445 -> 1389; MobileNetV2, one image 325 -> 296.
    const bool is_b = warp == 6;
    if (elect_one()) {
      const uint32_t b_tx = PLANES * static_cast<uint32_t>(p.block_n) * p.row_bytes;
      const uint32_t b_off = static_cast<uint32_t>(PLANES * AS) * slot;
      int s = 0;
      uint32_t ph = 0;
      long long issued = 0;
      bool ok = true, waited = false;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int tile = split_k ? unit / chunks : unit;
        const int kg0 = split_k ? (unit - tile * chunks) * chunk_groups : 0;
        const int kg1 = split_k ? min(kg0 + chunk_groups, k_groups) : k_groups;
        const int m_blk = tile / p.tiles_n;
        const int n_blk = tile - m_blk * p.tiles_n;
        const bool pair_tile = m_blk < p.pair_rows;
        const long long m0 = pair_tile ? static_cast<long long>(m_blk) * (2 * kTcBlockM)
                                       : static_cast<long long>(p.pair_rows) * (2 * kTcBlockM) +
                                             static_cast<long long>(m_blk - p.pair_rows) * kTcBlockM;
        const int halves = pair_tile ? 2 : 1;
        // a second half that starts past the last row repeats the first (its results are never stored)
        const long long m1 = pair_tile && m0 + kTcBlockM < p.M ? m0 + kTcBlockM : m0;
        const uint32_t my_tx = is_b ? b_tx : static_cast<uint32_t>(PLANES * halves * p.a_rows) * p.row_bytes;
        const int n0 = n_blk * p.block_n;
        int img[2] = {0, 0}, h_base[2] = {0, 0}, w_base[2] = {0, 0};
        if (p.a_im2col && !is_b) {
          const unsigned per_img = static_cast<unsigned>(p.OH) * static_cast<unsigned>(p.OW);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (half == 1 && !pair_tile) break;
            const unsigned m = static_cast<unsigned>(half ? m1 : m0);  // (below M, which is an int)
            img[half] = static_cast<int>(m / per_img);
            const int r = static_cast<int>(m - static_cast<unsigned>(img[half]) * per_img);
            const int oh = r / p.OW;
            const int ow = r - oh * p.OW;
            h_base[half] = oh * p.stride_h - p.pad_t;
            w_base[half] = ow * p.stride_w - p.pad_l;
          }
        }
        if (p.trace != nullptr && blockIdx.x == 0 && !is_b) p.trace[(unit / gridDim.x) * 16 + 0] = clock64();
        // the current K block: channel block, tap, and the tap's filter row and column
        int cb = 0, tap = 0, kh = 0, kw = 0;
        if (kg0 > 0) {
          cb = kg0 / taps;
          tap = kg0 - cb * taps;
          kh = tap / p.KW;
          kw = tap - kh * p.KW;
        }
        for (int kg = kg0; kg < kg1; ++kg) {
          const uint32_t fb = smem_u32(&full_bar[s]);
          const bool stall = test_stall && kg == kg0 && unit == static_cast<int>(blockIdx.x);
          if (!waited && (!is_b || issued == S)) {
            grid_dependency_wait();
            waited = true;
          }
          if (!mbar_wait_bounded(smem_u32(&empty_bar[s]), ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          const bool tr = p.trace != nullptr && blockIdx.x == 0 && !is_b && unit == static_cast<int>(gridDim.x) && kg < 32;
          if (tr) p.trace[1024 + kg * 4 + 0] = clock64();
          if (!stall) {
            mbar_arrive_expect_tx(fb, my_tx * static_cast<uint32_t>(SUB));
            for (int sb = 0; sb < SUB; ++sb) {
              const uint32_t dst = smem_base + static_cast<uint32_t>(s * SUB + sb) * stage_bytes;
              if (is_b) {
                const int k = (tap * p.c_blocks + cb) * p.k_elems;
                tma_load_2d(dst + b_off, &map_b0, fb, k, n0);
                if (PLANES == 2) tma_load_2d(dst + b_off + b_slot, &map_b1, fb, k, n0);
              } else {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                  if (half == 1 && !pair_tile) break;
                  const uint32_t at = dst + static_cast<uint32_t>(half * PLANES) * slot;
                  if (p.a_im2col) {
                    const uint16_t dw = static_cast<uint16_t>(kw * p.dil_w), dh = static_cast<uint16_t>(kh * p.dil_h);
                    tma_load_im2col_4d(at, &map_a0, fb, cb * p.k_elems, w_base[half], h_base[half], img[half], dw, dh);
                    if (PLANES == 2)
                      tma_load_im2col_4d(at + slot, &map_a1, fb, cb * p.k_elems, w_base[half], h_base[half], img[half], dw, dh);
                  } else {
                    const int k = cb * p.k_elems;
                    tma_load_2d(at, &map_a0, fb, k, static_cast<int>(half ? m1 : m0));
                    if (PLANES == 2) tma_load_2d(at + slot, &map_a1, fb, k, static_cast<int>(half ? m1 : m0));
                  }
                }
              }
              if (++kw == p.KW) {
                kw = 0;
                ++kh;
              }
              if (++tap == taps) {
                tap = kh = kw = 0;
                ++cb;
              }
            }
          }
          if (tr) p.trace[1024 + kg * 4 + 1] = clock64();
          ++issued;
          if (++s == S) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok) {
        if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_PRODUCER);
      }
      if (*abort_ptr != 0) {
        // Some role gave up.  Copies this warp issued may still be landing in
        // shared memory: wait (bounded) for each of the last S fills to finish.
        int zero = 0;
        const long long first = issued > S ? issued - S : 0;
        for (long long i = first; i < issued; ++i) {
          const int st = static_cast<int>(i % S);
          const uint32_t par = static_cast<uint32_t>((i / S) & 1);
          mbar_wait_bounded(smem_u32(&full_bar[st]), par, &zero, test_stall ? 2000000ull : 200000000ull);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (elect_one()) {
      // formats: kind::i8 s32 <- s8 (2, 1); kind::tf32 f32 <- tf32 (1, 2); kind::f16 f32 <- bf16 (1, 1)
      const uint32_t idesc = KIND == GEMM_I8
                                 ? instr_desc(2u, 1u, kTcBlockM, static_cast<uint32_t>(p.block_n))
                                 : instr_desc(1u, KIND == GEMM_BF16X3 ? 1u : 2u, kTcBlockM,
                                              static_cast<uint32_t>(p.block_n));
      // One thread issues every MMA, so its instruction stream is the critical path:
      // descriptors are formed by adding small constants to values computed once.
      // (the start-address field counts 16-byte units; a K step is 32 bytes = 2 units)
      const int k_steps = p.row_bytes / 32;
      const uint64_t desc_fixed = smem_desc_kmajor(0u, static_cast<uint32_t>(p.row_bytes));
      const uint64_t a_first = desc_fixed + ((smem_base & 0x3ffffu) >> 4);
      const uint64_t stage_units = stage_bytes >> 4;
      const uint64_t slot_units = slot >> 4;
      const uint64_t b_slot_units = b_slot >> 4;
      const uint64_t a1_from_a = static_cast<uint64_t>(PLANES) * slot_units;  // second half's planes
      const uint64_t b_from_a = static_cast<uint64_t>(PLANES * AS) * slot_units;
      const uint32_t acc_stride = p.pair ? 256u : 128u;
      const int pair_rows = p.pair_rows;
      const int tiles_n = p.tiles_n;
      const bool tracing = p.trace != nullptr && blockIdx.x == 0;
      int s = 0;
      uint32_t ph = 0;
      int acc = 0;
      uint32_t acc_ph = 0;
      bool ok = true;
      bool full_seen = false, empty_seen = false;  // the next stage is full / the next accumulator is free (see tc_k_block)
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int tile = split_k ? unit / chunks : unit;
        // the accumulators of this unit: one, or one per chunk of a whole tile
        int kb1 = split_k ? (unit - tile * chunks) * chunk_groups : 0;
        const int kb_end = split_k ? min(kb1 + chunk_groups, k_groups) : k_groups;
        while (kb1 < kb_end && ok) {
          const int kb0 = kb1;
          kb1 = min(kb0 + chunk_groups, kb_end);
          if (!empty_seen && !mbar_wait_bounded(smem_u32(&tempty_bar[acc]), acc_ph ^ 1u, abort_ptr, wait_limit)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          if (tracing) p.trace[(unit / gridDim.x) * 16 + 1] = clock64();
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc) * acc_stride;
          const bool pair = tile / tiles_n < pair_rows;
          uint32_t accumulate = 0u;
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!full_seen && !mbar_wait_bounded(smem_u32(&full_bar[s]), ph, abort_ptr, wait_limit)) {
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const bool tr = tracing && unit == static_cast<int>(gridDim.x) && kb < 32;
            if (tr) p.trace[1024 + kb * 4 + 2] = clock64();
            for (int sb = 0; sb < SUB; ++sb) {
              const uint64_t a0 = a_first + static_cast<uint64_t>(s * SUB + sb) * stage_units;
              const uint64_t b0 = a0 + b_from_a;
              if (pair) tc_k_block<KIND, false, true>(k_steps, d_tmem, a0, slot_units, b0, b_slot_units, idesc, accumulate, a1_from_a);
              else tc_k_block<KIND, false>(k_steps, d_tmem, a0, slot_units, b0, b_slot_units, idesc, accumulate);
              accumulate = 1u;
            }
            const bool last = kb + 1 == kb1;
            const int next_s = s + 1 == S ? 0 : s + 1;
            const uint32_t next_ph = s + 1 == S ? ph ^ 1u : ph;
            full_seen = mbar_test_wait(smem_u32(&full_bar[next_s]), next_ph);
            if (last) empty_seen = mbar_test_wait(smem_u32(&tempty_bar[acc + 1 == accs ? 0 : acc + 1]), acc + 1 == accs ? acc_ph : acc_ph ^ 1u);
            tc_commit(smem_u32(&empty_bar[s]));
            if (tr) p.trace[1024 + kb * 4 + 3] = clock64();
            s = next_s;
            ph = next_ph;
          }
          if (!ok) break;
          tc_commit(smem_u32(&tfull_bar[acc]));
          if (tracing) p.trace[(unit / gridDim.x) * 16 + 2] = clock64();
          if (++acc == accs) {
            acc = 0;
            acc_ph ^= 1u;
          }
        }
      }
      if (!ok) {
        if (atomicCAS(const_cast<int*>(abort_ptr), 0, 1) == 0) atomicCAS(p.status, 0, TC_TIMEOUT_MMA);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Two groups of four warps (2-5 and 7-10; a warp reads the quarter of the TMEM lanes that its number selects)
    // drain every tile together: each takes half of a tile's columns, or one half of a paired tile's rows.
    const int group = warp >= 7 ? 1 : 0;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int half_cols = ((p.block_n / 2) + 15) & ~15;
    int acc = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    const TcGemmParams lp = p;  // a register copy (a reference to the kernel parameter makes every access a generic load)
    TcDirect d{};
    d.res_mode = p.res_mode;
    d.act = p.act;
    d.act_a = p.act_a;
    d.act_b = p.act_b;
    d.out_scale = p.out_scale;
    d.wide = p.wide;
    d.chw = static_cast<long long>(p.OH) * p.OW;
    constexpr int es = EPI / 2 == OUT_I8 ? 1 : (EPI / 2 == OUT_BF16X2 ? 2 : 4);
    uint8_t* const out0 = EPI / 2 == OUT_I8 ? reinterpret_cast<uint8_t*>(p.outq) : reinterpret_cast<uint8_t*>(p.out0);
    uint8_t* const out1 = reinterpret_cast<uint8_t*>(p.out1);
    d.pitch = p.ldo * es;
    d.pitch8 = 8 * d.pitch;
    d.xs = 8;
    d.ys = 4;
    d.stage = smem_base + static_cast<uint32_t>(S * SUB) * stage_bytes + static_cast<uint32_t>(group * 4 + quarter) * kDrainWarpBytes;
    if (SIDE) {
      d.side_count = p.side_count;
      d.side_pitch = p.side_ld;
      d.side_pitch8 = 8 * p.side_ld;
      d.side_stage = smem_base + static_cast<uint32_t>(S * SUB) * stage_bytes + 8u * kDrainWarpBytes +
                     static_cast<uint32_t>(group * 4 + quarter) * 2u * kDrainSideBytes;
      d.side_scale0 = p.side_scale0;
      d.side_scale1 = p.side_scale1;
    }
    const bool tracing = p.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 64;
    // this thread's row and columns of a tile: rows of one half of a pair, or half of the columns
    struct Share {
      long long m;
      int n_first, c_first, cols;
      bool pair;
    };
    // An int8 layer's fp32 residual that has left L2 since it was written (126 MB) starts on its way back one tile ahead;
    // the drain itself asks one step ahead only.  56x56x64, 256 images: 169 -> 156 us.  (28x28x128, which is still in L2,
    // went from 84 to 88, and bf16-pair layers with long main loops gained nothing.)
    const bool far_residual = KIND == GEMM_I8 && EPI != kEpiAny && EPI % 2 == 1 && lp.res_mode == RES_F32 &&
                              static_cast<long long>(lp.M) * lp.ldo * 4 > (126ll << 20);
    auto share = [&](int tile) {
      const int m_blk = tile / p.tiles_n;
      Share w;
      w.pair = m_blk < p.pair_rows;
      const long long m_tile = w.pair ? static_cast<long long>(m_blk) * (2 * kTcBlockM)
                                      : static_cast<long long>(p.pair_rows) * (2 * kTcBlockM) +
                                            static_cast<long long>(m_blk - p.pair_rows) * kTcBlockM;
      w.m = m_tile + (w.pair && group ? kTcBlockM : 0) + row;
      w.c_first = !w.pair && group ? half_cols : 0;
      w.cols = w.pair ? p.block_n : (group ? p.block_n - half_cols : half_cols);
      w.n_first = (tile - m_blk * p.tiles_n) * p.block_n + w.c_first;
      return w;
    };
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      const int tile = split_k ? unit / chunks : unit;
      const Share here = share(tile);
      const bool pair_tile = here.pair;
      const long long m = here.m;
      const int c_first = here.c_first, cols = here.cols, n_first = here.n_first;
      const bool valid = m < lp.M;
      TcOperands<KIND, EPI != kEpiAny && EPI % 2 == 1> ops;  // (residual, bias, scale: on their way before the accumulator is waited for)
      if constexpr (EPI != kEpiAny) {
        if (EPI / 2 == OUT_CHW) {
          const unsigned px = static_cast<unsigned>(d.chw);
          const unsigned img = static_cast<unsigned>(m) / px;
          d.o0 = out0 + ((static_cast<long long>(img) * lp.N + n_first) * d.chw + (static_cast<unsigned>(m) - img * px)) * 4;
        } else {
          const long long at = (m - lane) * d.pitch + static_cast<long long>(n_first) * es;  // (the warp's first row)
          d.o0 = out0 + at;
          d.o1 = out1 + at;
          const long long rows_left = lp.M - (m - lane);
          d.rows = rows_left > 32 ? 32 : static_cast<int>(rows_left);
        }
        if (EPI % 2 == 1) {
          const int rs = lp.res_mode == RES_BF16X2 ? 2 : 4;
          d.r0 = reinterpret_cast<const uint8_t*>(lp.res0) + (m * lp.ldo + n_first) * rs;
          d.r1 = reinterpret_cast<const uint8_t*>(lp.res1) + (m * lp.ldo + n_first) * rs;
        }
        d.bias = lp.bias != nullptr ? lp.bias + n_first : nullptr;
        d.scale = lp.scale + n_first;
        if (SIDE) {
          const long long side_at = (m - lane) * lp.side_ld + n_first;
          d.side_q0 = reinterpret_cast<uint8_t*>(lp.side_q0) + side_at;
          d.side_q1 = reinterpret_cast<uint8_t*>(lp.side_q1) + side_at;
        }
        ops.fetch(d, 0, cols > 0 ? lp.N - n_first : 0, valid);
      }
      if (far_residual && unit + static_cast<int>(gridDim.x) < units) {
        const Share next = share(unit + static_cast<int>(gridDim.x));
        const long long bytes = 4ll * min(next.cols, lp.N - next.n_first);
        const uint8_t* r0 = reinterpret_cast<const uint8_t*>(lp.res0 + next.m * lp.ldo + next.n_first);
        if (next.m < lp.M)
          for (long long b = 0; b < bytes; b += 128) prefetch_l2(r0 + b);
      }
      if (tracing) p.trace[(unit / gridDim.x) * 16 + 3] = clock64();
      // the vote keeps the warp together: tcgen05.ld below needs all 32 lanes
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&tfull_bar[acc]), acc_ph, abort_ptr, wait_limit) ? 1 : 0) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      if (tracing) p.trace[(unit / gridDim.x) * 16 + 4] = clock64();
      uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                       static_cast<uint32_t>(acc) * (p.pair ? 256u : 128u) + (pair_tile && group ? 128u : 0u) + static_cast<uint32_t>(c_first);
      if (CHUNKS && chunks > 1) {
        const uint32_t t_first = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(c_first);
        const uint32_t t_sum = t_first + 384u;
        uint32_t* const ws = lp.sk_ws + static_cast<size_t>(unit) * kTcBlockM * lp.block_n +
                             static_cast<size_t>(c_first) * kTcBlockM + static_cast<size_t>(row) * 16;
        for (int c = split_k ? chunks - 1 : 0; c < chunks; ++c) {  // (split: this unit's chunk alone)
          if (c > 0 && !split_k) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&tfull_bar[acc]), acc_ph, abort_ptr, wait_limit) ? 1 : 0) != 0;
            if (!ok) break;
            tc_fence_after_sync();
            t_row = t_first + static_cast<uint32_t>(acc) * 128u;
          }
          if (split_k) tc_publish_chunk(t_row, ws, cols, valid);
          else if (KIND == GEMM_BF16X3) tc_add_chunk(t_row, t_sum, cols, c == 0);
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
          if (++acc == accs) {
            acc = 0;
            acc_ph ^= 1u;
          }
        }
        if (!ok) break;
        if (split_k) {
          // whichever warp publishes these rows and columns last of the tile's chunks adds them up
          int* const count = lp.sk_flags + tile * 8 + group * 4 + quarter;
          __threadfence();
          __syncwarp();
          int before = 0;
          if (lane == 0) before = atomicAdd(count, 1);
          if (__shfl_sync(0xffffffffu, before, 0) != chunks - 1) continue;
          if (lane == 0) *count = 0;  // for the next launch
          __threadfence();
          const size_t slot_words = static_cast<size_t>(kTcBlockM) * lp.block_n;
          tc_gather_chunks<KIND>(ws - static_cast<size_t>(unit - tile * chunks) * slot_words, slot_words, chunks, t_sum, cols, valid);
        }
        t_row = t_sum;
      }
      if constexpr (EPI != kEpiAny) {
        tc_drain<KIND, EPI, SIDE, false>(d, t_row, cols, lp.N - n_first, valid, ops);
      } else {
        const bool bf16_io = lp.out_mode == OUT_BF16X2 || lp.res_mode == RES_BF16X2;
        for (int c0 = 0; c0 < cols; c0 += 16) {
          uint32_t v[16];
          tmem_ld16(t_row + static_cast<uint32_t>(c0), v);
          tmem_ld_wait();
          const int n = n_first + c0;
          if (valid && n < lp.N) {
            if (SIDE && lp.side_count > 0) tc_epilogue_chunk<KIND, true, true>(lp, v, m, n, lp.bias + n, lp.scale + n);
            else if (bf16_io) tc_epilogue_chunk<KIND, true>(lp, v, m, n, lp.bias + n, lp.scale + n);
            else tc_epilogue_chunk<KIND, false>(lp, v, m, n, lp.bias + n, lp.scale + n);
          }
        }
      }
      if (tracing) p.trace[(unit / gridDim.x) * 16 + 5] = clock64();
      if (CHUNKS && chunks > 1) continue;  // (the accumulators were handed back above)
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      if (++acc == accs) {
        acc = 0;
        acc_ph ^= 1u;
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
