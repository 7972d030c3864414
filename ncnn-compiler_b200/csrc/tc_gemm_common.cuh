// Kinds, formats, parameters and small device functions shared by the tensor-core contraction kernels.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "ptx_sm100.cuh"

namespace nb {

enum : int { GEMM_TF32 = 0, GEMM_TF32X3 = 1, GEMM_I8 = 2, GEMM_BF16X3 = 3 };

__host__ __device__ constexpr int tc_planes(int kind) { return kind == GEMM_TF32X3 || kind == GEMM_BF16X3 ? 2 : 1; }
__host__ __device__ constexpr int tc_elem_bytes(int kind) { return kind == GEMM_I8 ? 1 : (kind == GEMM_BF16X3 ? 2 : 4); }
// ACT_SIGMOID..ACT_SCALE follow the reference's separate activation ops:
//   SIGMOID      1/(1+exp(-clamp(x, +-88.376...)))            (ConvertSigmoid, NCNNToTosa.cpp:2991-3021)
//   SWISH        x * 1/(1+exp(-x))                            (ConvertSwish, :3702-3720)
//   HARDSIGMOID  clamp(x*alpha + beta, 0, 1), HARDSWISH x * that (ConvertHardActivation, :3023-3072)
//   TANH         tanh(x)                                      (ConvertTanH, :3722-3736)
//   SCALE        x * a                                        (ConvertDropout, :2047-2070)
//   SQUARE       x * x                                        (ConvertUnary, :5225-5252)
enum : int {
  ACT_NONE = 0, ACT_RELU = 1, ACT_LEAKY = 2, ACT_CLIP = 3, ACT_SIGMOID = 4, ACT_SWISH = 5, ACT_HARDSIGMOID = 6,
  ACT_HARDSWISH = 7, ACT_TANH = 8, ACT_SCALE = 9, ACT_SQUARE = 10, ACT_GELU = 11
};
// OUT_F32        plain fp32
// OUT_F32_SPLIT  two fp32 planes: hi = value rounded to tf32, lo = value - hi
// OUT_I8         int8 after requantisation with out_scale
// OUT_F32_TF32   fp32 rounded to tf32 (fast mode keeps operands unbiased)
// OUT_BF16X2     two bf16 planes: hi = bf16(value), mid = bf16(value - hi)
// OUT_CHW        plain fp32 in the caller's [image][channel][pixel] order (a graph output)
enum : int { OUT_F32 = 0, OUT_F32_SPLIT = 1, OUT_I8 = 2, OUT_F32_TF32 = 3, OUT_BF16X2 = 4, OUT_CHW = 5 };
// format of the optional residual operand of the epilogue
enum : int { RES_NONE = 0, RES_F32 = 1, RES_SPLIT = 2, RES_BF16X2 = 3 };

enum : int {
  TC_OK = 0,
  TC_TIMEOUT_PRODUCER = 1,
  TC_TIMEOUT_MMA = 2,
  TC_TIMEOUT_EPILOGUE = 3,
};

constexpr int kTcThreads = 352;  // warps: 0 A producer, 1 MMA issuer, 2-5 and 7-10 two epilogue groups, 6 B producer
constexpr int kTcBlockM = 128;
constexpr int kTcMaxStages = 8;
constexpr uint32_t kTcTmemCols = 512;           // four accumulators of up to 128 columns, or two pairs of them
constexpr uint64_t kTcWaitLimitNs = 2000000000ull;  // a wait longer than 2 s is a bug

struct TcGemmParams {
  int M, N;
  int tiles_m, tiles_n, block_n;
  int k_blocks;   // K iterations per tile = taps * c_blocks
  int c_blocks;   // channel blocks per filter tap (K blocks for a plain GEMM)
  int half_blocks;  // tc_gemm2_kernel: K blocks are halves of the usual size, c_blocks and k_blocks count halves
  int k_elems;    // elements per K block
  int row_bytes;  // bytes per shared-memory operand row: 128 or 64
  int stages;
  int a_rows;       // rows of A that a copy brings: 128, or what a single tile of fewer rows has (a multiple of 8)
  int stage_bytes;  // bytes of one ring stage: planes * (A tile + B tile rounded to 1 KB)
  int a_im2col;  // A addressing: 0 plain matrix (tiled TMA), 1 im2col TMA
  int OH, OW, KW;
  int stride_h, stride_w, pad_t, pad_l, dil_h, dil_w;
  // epilogue
  const float* bias;   // [N] or null
  const float* scale;  // [N] int8 dequantisation factor 1/(s_w*s_in), GEMM_I8 only
  float* out0;
  float* out1;
  int8_t* outq;
  const float* res0;  // optional residual (same layout as the output), plane hi
  const float* res1;  // optional residual plane lo
  int res_mode;       // RES_*
  long long ldo;      // output row stride in elements
  int out_mode;
  int act;
  float act_a, act_b;  // leaky slope / clip bounds
  float out_scale;     // requantisation scale (OUT_I8)
  int* status;         // device words: [0] stays 0 unless a bounded wait gave up; [1] non-zero injects a stalled
                       // stage into tc_gemm_kernel (host tests of the time-out path), zero in production
  int direct;          // results leave through tc_drain (rows of 16-byte pieces); 0: element by element
  int wide;            // rows of result and residual are multiples of 32 bytes, 32-byte aligned
  // 1: tiles may be two 128-row halves that share one B tile per K block: the A halves sit side by
  // side in a stage and accumulate into neighbouring column ranges.  The first pair_rows tile rows
  // are such pairs (256 rows each), the remaining tiles_m - pair_rows tile rows are single tiles:
  // whole waves of pairs, then a last wave that is not coarser than it has to be.
  int pair;
  int pair_rows;
  int sub_blocks;  // int8: K blocks per ring stage (one barrier hand-shake for several small copies); 1 elsewhere
  long long* trace;    // optional (bring-up): per-role clock stamps of CTA 0, 8 values per tile
  // CTA pairs (tc_gemm2.cuh): tiles are 256 rows, tiles_m counts those.
  // streamk = 1: every pair gets an equal share of all (tile, K block) units, so a tile may be split
  // between neighbouring pairs; the pair that holds a tile's last K block adds the others' partial
  // accumulators (exchanged through sk_ws) and runs the epilogue.
  int streamk;
  // Quantised copies of an fp32 result for the int8 contractions that read it next (up to two, each with
  // its consumer's input scale): written by the epilogue next to the fp32 tensor, so no Quantize pass
  // re-reads it.  Q(.) is the reference's (NCNNToTosa.cpp:356-385) applied to the value that is stored.
  int side_count;
  int8_t* side_q0;
  int8_t* side_q1;
  float side_scale0, side_scale1;
  long long side_ld;   // row stride of the int8 copies in elements
  // The K blocks are summed in `chunks` groups of chunk_blocks each and the groups' sums added in order: deep bf16-pair
  // convolutions (set_chunks: by the layer alone, so that every batch size rounds the same), and InnerProducts of few rows
  // (split_rows).  split_k = 1: the chunks of a tile run on different CTAs (tc_gemm_kernel).
  int chunks, chunk_blocks, split_k;
  uint32_t* sk_ws;     // one slot of 128 x block_n accumulator words per CTA
  int* sk_flags;       // one word per CTA: 1 while its slot holds a partial that nobody has consumed
};

// ---- issuing MMAs
// One thread issues all MMAs of a CTA, and two things decide whether the tensor pipe stays busy:
//   * the instructions between MMAs: a K block's steps are unrolled completely (tc_k_block), with descriptors that
//     differ by constants; a loop over the steps costs 53 clocks for each narrow MMA instead of 43;
//   * barrier reads after a commit: they return only when the MMAs before that commit are done (measured: ~290 clocks
//     of an idle pipe per K block).  So the barrier that the NEXT K block or tile waits for is tested between a
//     block's MMAs and its commit (mbar_test_wait), and read again only if it was not complete then.
// Together: 7x7x512 -> 512 (72 K blocks) 39.6 -> 29.0 us for one image, 90 -> 67 us for 128.
template <int KIND, bool CTA_PAIR>
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  if (CTA_PAIR) {
    if (KIND == GEMM_I8) ptx::mma_i8_pair(d, a, b, idesc, accumulate);
    else if (KIND == GEMM_BF16X3) ptx::mma_f16_pair(d, a, b, idesc, accumulate);
    else ptx::mma_tf32_pair(d, a, b, idesc, accumulate);
  } else {
    if (KIND == GEMM_I8) ptx::mma_i8(d, a, b, idesc, accumulate);
    else if (KIND == GEMM_BF16X3) ptx::mma_f16(d, a, b, idesc, accumulate);
    else ptx::mma_tf32(d, a, b, idesc, accumulate);
  }
}
// one K step (32 bytes of every operand row): the product, or the three of operands split into two planes
// (`a_plane`, `b_plane`: from the high plane to the low one, in 16-byte units)
template <int KIND, bool CTA_PAIR>
__device__ __forceinline__ void tc_k_step(uint32_t d, uint64_t a, uint64_t a_plane, uint64_t b, uint64_t b_plane, uint32_t idesc,
                                          uint32_t accumulate) {
  if (tc_planes(KIND) == 2) {
    tc_mma<KIND, CTA_PAIR>(d, a + a_plane, b, idesc, accumulate);  // low * high
    tc_mma<KIND, CTA_PAIR>(d, a, b + b_plane, idesc, 1u);          // high * low
    tc_mma<KIND, CTA_PAIR>(d, a, b, idesc, 1u);                    // high * high
  } else {
    tc_mma<KIND, CTA_PAIR>(d, a, b, idesc, accumulate);
  }
}
// the K steps of one block of 128-, 64- or 32-byte operand rows; `accumulate` is 0 for a tile's first block.
// HALVES: the same B block also against a second A tile (`a_half` further), into the columns 128 further.
template <int KIND, bool CTA_PAIR, int STEPS, bool HALVES>
__device__ __forceinline__ void tc_k_steps(uint32_t d, uint64_t a, uint64_t a_plane, uint64_t b, uint64_t b_plane, uint32_t idesc,
                                           uint32_t accumulate, uint64_t a_half) {
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {  // (a step is 32 bytes, 2 units)
    tc_k_step<KIND, CTA_PAIR>(d, a + 2u * k, a_plane, b + 2u * k, b_plane, idesc, k == 0 ? accumulate : 1u);
    if (HALVES) tc_k_step<KIND, CTA_PAIR>(d + 128u, a + a_half + 2u * k, a_plane, b + 2u * k, b_plane, idesc, k == 0 ? accumulate : 1u);
  }
}
template <int KIND, bool CTA_PAIR, bool HALVES = false>
__device__ __forceinline__ void tc_k_block(int steps, uint32_t d, uint64_t a, uint64_t a_plane, uint64_t b, uint64_t b_plane,
                                           uint32_t idesc, uint32_t accumulate, uint64_t a_half = 0) {
  if (steps == 4) tc_k_steps<KIND, CTA_PAIR, 4, HALVES>(d, a, a_plane, b, b_plane, idesc, accumulate, a_half);
  else if (steps == 2) tc_k_steps<KIND, CTA_PAIR, 2, HALVES>(d, a, a_plane, b, b_plane, idesc, accumulate, a_half);
  else tc_k_steps<KIND, CTA_PAIR, 1, HALVES>(d, a, a_plane, b, b_plane, idesc, accumulate, a_half);
}

// ---- sums in chunks (see TcGemmParams::chunks)
// Adds the accumulator of one chunk to the running sum of this warp's 32 rows, both in tensor memory (an epilogue thread
// has no registers for the sums of a whole tile); `first`: starts the sum.  Every lane of the warp must call it.
__device__ __forceinline__ void tc_add_chunk(uint32_t t_acc, uint32_t t_sum, int cols, bool first) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 16) {
    uint32_t v[16], s[16];
    ptx::tmem_ld16(t_acc + static_cast<uint32_t>(c), v);
    if (!first) ptx::tmem_ld16(t_sum + static_cast<uint32_t>(c), s);
    ptx::tmem_ld_wait();
    if (!first)
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__fadd_rn(__uint_as_float(s[j]), __uint_as_float(v[j])));
    ptx::tmem_st16(t_sum + static_cast<uint32_t>(c), v);
  }
  ptx::tmem_st_wait();
}
// The same sum of chunks that different CTAs computed.  `ws` is this thread's row in the slot of a chunk
// ([16-column group][row][16] words); the slots of a tile's chunks follow each other.
// (`valid`: the row exists; every lane of the warp must call it)
__device__ __forceinline__ void tc_publish_chunk(uint32_t t_acc, uint32_t* ws, int cols, bool valid) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 16) {
    uint32_t v[16];
    ptx::tmem_ld16(t_acc + static_cast<uint32_t>(c), v);
    ptx::tmem_ld_wait();
    if (!valid) continue;
    uint4* d = reinterpret_cast<uint4*>(ws + static_cast<size_t>(c) * 128);
#pragma unroll
    for (int q = 0; q < 4; ++q) __stcg(d + q, make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
  }
}
template <int KIND>
__device__ __forceinline__ void tc_gather_chunks(const uint32_t* ws, size_t slot_words, int chunks, uint32_t t_sum, int cols, bool valid) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 16) {
    uint32_t v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = 0u;
    if (valid) {
#pragma unroll 4
      for (int k = 0; k < chunks; ++k) {
        const uint4* s = reinterpret_cast<const uint4*>(ws + static_cast<size_t>(k) * slot_words + static_cast<size_t>(c) * 128);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 f = __ldcg(s + q);
          const uint32_t w[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (KIND == GEMM_I8) v[4 * q + j] += w[j];
            else v[4 * q + j] = k == 0 ? w[j] : __float_as_uint(__fadd_rn(__uint_as_float(v[4 * q + j]), __uint_as_float(w[j])));
          }
        }
      }
    }
    ptx::tmem_st16(t_sum + static_cast<uint32_t>(c), v);
  }
  ptx::tmem_st_wait();
}

// round-half-away-from-zero exactly as the reference evaluates it in fp32:
// floor(v + 0.5f) for v >= 0, ceil(v - 0.5f) otherwise, then clamp to [-127, 127].  Both are the sum of v and a half of
// its own sign, cut off towards zero; the clamp's bounds are whole numbers, so it may come before the cut.
__device__ __forceinline__ int quantize_rha(float x, float s) {
  const float v = __fmul_rn(x, s);
  const float t = __fadd_rn(v, copysignf(0.5f, v));
  return __float2int_rz(fmaxf(fminf(t, 127.0f), -127.0f));
}
// four quantised values as four bytes, the first lowest
__device__ __forceinline__ uint32_t pack_i8x4(int a, int b, int c, int d) {
  uint32_t hi, r;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
  return r;
}
__device__ __forceinline__ uint32_t quantize4(float a, float b, float c, float d, float s) {
  return pack_i8x4(quantize_rha(a, s), quantize_rha(b, s), quantize_rha(c, s), quantize_rha(d, s));
}
// The same with a clamp at zero in place of -127 (a fused ReLU, or values and a scale that are not negative): what is negative
// ends as zero however it is rounded, and cutting off a fraction is an addition, 2^23 plus the value rounded towards zero,
// whose low bits are the whole part.  Conversions to int run at an eighth of the rate of additions.
// (The form with a sign takes more instructions than it saves: 56x56x64 with an int8 copy 128 -> 141 us.)
__device__ __forceinline__ uint32_t quantize4_at_zero(float a, float b, float c, float d, float s) {
  auto bits = [s](float x) {
    return __float_as_uint(__fadd_rz(fmaxf(fminf(__fadd_rn(__fmul_rn(x, s), 0.5f), 127.0f), 0.0f), 8388608.0f));
  };
  return __byte_perm(__byte_perm(bits(a), bits(b), 0x0040), __byte_perm(bits(c), bits(d), 0x0040), 0x5410);
}

__device__ __forceinline__ float round_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// two floats -> two bf16 (round to nearest even), `a` in the low half
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float bf16_low(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_high(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
// hi = bf16(x), mid = bf16(x - hi) for two values at once
__device__ __forceinline__ void split_bf16x2(float a, float b, uint32_t& hi, uint32_t& mid) {
  hi = pack_bf16x2(a, b);
  mid = pack_bf16x2(__fadd_rn(a, -bf16_low(hi)), __fadd_rn(b, -bf16_high(hi)));
}

// two fp32 values in one register pair
__device__ __forceinline__ void f32x2_fma(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t f32x2_fma3(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ void f32x2_add(uint64_t& d, uint64_t a, uint64_t b) {
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t f32x2_make(uint32_t lo, uint32_t hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ float2 f32x2_get(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t lds_b64(uint32_t at) {
  uint64_t v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(at));
  return v;
}

// The activations a network seldom uses live in one function that is called, not inlined: an epilogue applies its
// activation to 16 or 32 values in a row, and a copy of every branch per value made the loops large enough to
// stall on instruction fetch (a 3x3 depthwise block spent 5000 cycles there instead of 400).
static __device__ __noinline__ float apply_act_rare(float y, int act, float a, float b) {
  if (act == ACT_SIGMOID) {
    const float c = fminf(fmaxf(y, -88.3762626647949f), 88.3762626647949f);
    return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-c)));
  }
  if (act == ACT_SWISH) return __fmul_rn(y, __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-y))));
  if (act == ACT_HARDSIGMOID || act == ACT_HARDSWISH) {
    const float gate = fminf(fmaxf(__fadd_rn(__fmul_rn(y, a), b), 0.0f), 1.0f);
    return act == ACT_HARDSWISH ? __fmul_rn(y, gate) : gate;
  }
  if (act == ACT_TANH) return tanhf(y);
  if (act == ACT_SCALE) return __fmul_rn(y, a);
  if (act == ACT_SQUARE) return __fmul_rn(y, y);
  // (x * erfc(x * -1/sqrt(2))) * 0.5, the order of ConvertGELU (NCNNToTosa.cpp:4670-4738)
  if (act == ACT_GELU) return __fmul_rn(__fmul_rn(y, erfcf(__fmul_rn(y, -0.7071067811865476f))), 0.5f);
  return y;
}

__device__ __forceinline__ float apply_act(float y, int act, float a, float b) {
  if (act == ACT_NONE) return y;
  if (act == ACT_RELU) return fmaxf(y, 0.0f);
  if (act == ACT_CLIP) return fminf(fmaxf(y, a), b);
  if (act == ACT_LEAKY) return y >= 0.0f ? y : __fmul_rn(y, a);
  return apply_act_rare(y, act, a, b);
}

// 16 fp32 results of one row -> 16 int8 with the reference's rounding, one 16-byte store
__device__ __forceinline__ void tc_store_side_quant(int8_t* q, float scale, const float (&y)[16]) {
  uint32_t w[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) w[g] = quantize4(y[4 * g], y[4 * g + 1], y[4 * g + 2], y[4 * g + 3], scale);
  *reinterpret_cast<uint4*>(q) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Operand rows of 64 bytes with the 64-byte TMA swizzle: the 16-byte chunk j of row r lives at
// r*64 + ((j ^ ((r >> 1) & 3)) * 16).
__device__ __forceinline__ uint32_t stage_chunk_offset(int row, int j) {
  return static_cast<uint32_t>(row * 64 + ((j ^ ((row >> 1) & 3)) << 4));
}

}  // namespace nb
