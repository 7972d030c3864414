// Epilogue of the tensor-core kernels: accumulator columns -> bias, residual, activation, output format -> HBM.
//
// A thread owns one accumulator row (one output pixel) and takes it 16 columns at a time from tensor memory; the TMEM
// load and the residual loads of the next 16 columns are in flight while the current ones are worked on.  Every 128
// bytes of finished rows go through 4 KB of shared memory that belong to the warp alone and leave as stores of whole
// 128-byte lines (a thread storing its own row touches 32 lines per instruction: layers that are bound by their
// result ran 30-45 % slower that way).  A warp meets no barrier and waits for no other warp.
//
// What bounds it: instruction latency, because an epilogue warp has its scheduler almost to itself.  The form before
// this one staged chunks of 128 rows, met at a barrier per chunk and had one thread issue the TMA stores of all:
// 3 900 cycles for a 128 x 64 tile of bf16 pairs, 7 500 with a residual.
#pragma once

#include "tc_gemm_common.cuh"

namespace nb {

constexpr int kDrainWarpBytes = 4096;  // shared memory of one epilogue warp
constexpr int kDrainSideBytes = 2048;  // and of each int8 copy

// What one warp needs to finish its 32 rows.
struct TcDirect {
  // result planes at row 0 of the warp, first column of this drain (OUT_I8: int8; OUT_CHW: this thread's own pixel,
  // fp32, columns `chw` elements apart); row r lies (r / 8) * pitch8 + (r % 8) * pitch bytes further
  uint8_t* o0;
  uint8_t* o1;
  long long pitch, pitch8;
  int rows, xs, ys;     // row r exists when r < rows, r % 8 < xs and r / 8 < ys
  uint32_t stage;       // this warp's shared memory (16-byte aligned)
  const uint8_t* r0;    // residual planes at this thread's row, or null
  const uint8_t* r1;
  const float* bias;    // at the first column, or null
  const float* scale;   // GEMM_I8
  int res_mode;
  int act;
  float act_a, act_b, out_scale;
  int wide;             // residual rows are multiples of 32 bytes and 32-byte aligned: full-sector loads
  long long chw;        // OUT_CHW: elements between channels
  int side_count;       // int8 copies of an fp32 result
  uint8_t* side_q0;     // at row 0 of the warp
  uint8_t* side_q1;
  long long side_pitch, side_pitch8;
  uint32_t side_stage;  // kDrainSideBytes of the warp's own per copy
  float side_scale0, side_scale1;
  // partial accumulators of other CTAs to add first (split tiles): slots fix_stride words apart, [16-column group][row][16]
  const uint32_t* fix_ws;
  long long fix_stride;
  int fix_count;
};

__device__ __forceinline__ void ldg_32b(const void* p, uint32_t* w) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(p)
               : "memory");
}

// BYTES bytes of a row (32 or 64), of which the first `have` bytes exist (a multiple of 16)
template <int BYTES>
__device__ __forceinline__ void tc_row_load(const uint8_t* p, uint32_t* w, int have, int wide) {
#pragma unroll
  for (int h = 0; h < BYTES / 32; ++h) {
    if (wide && have >= 32 * h + 32) {
      ldg_32b(p + 32 * h, w + 8 * h);
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (have >= 32 * h + 16 * q + 16) v = *reinterpret_cast<const uint4*>(p + 32 * h + 16 * q);
        w[8 * h + 4 * q] = v.x;
        w[8 * h + 4 * q + 1] = v.y;
        w[8 * h + 4 * q + 2] = v.z;
        w[8 * h + 4 * q + 3] = v.w;
      }
    }
  }
}

// the activations an epilogue seldom meets, out of line: 16 inlined copies of them would sit in every drain loop
static __device__ __noinline__ void tc_act_many(float* y, int act, float a, float b) {
#pragma unroll 1
  for (int j = 0; j < 16; ++j) y[j] = apply_act(y[j], act, a, b);
}

__device__ __forceinline__ void sts_16b(uint32_t at, const uint32_t* w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}
// 16 fp32 results -> 16 int8 with the reference's rounding; `positive`: neither results nor scale are below zero
__device__ __forceinline__ void tc_stage_side_quant(uint32_t at, float scale, bool positive, const float (&y)[16]) {
  uint32_t w[4];
  if (positive) {
#pragma unroll
    for (int g = 0; g < 4; ++g) w[g] = quantize4_at_zero(y[4 * g], y[4 * g + 1], y[4 * g + 2], y[4 * g + 3], scale);
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g) w[g] = quantize4(y[4 * g], y[4 * g + 1], y[4 * g + 2], y[4 * g + 3], scale);
  }
  sts_16b(at, w);
}
__device__ __forceinline__ uint4 lds_16b(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}

// Where this lane's stores of a flush go: piece `lane % CHUNKS` of rows lane / CHUNKS + i * (32 / CHUNKS).  Worked out
// once per drain: byte offset of the first row, and which rows exist.
template <int CHUNKS>
struct TcFlushLane {
  long long first;
  uint32_t rows;  // bit i: row i of this lane exists
  __device__ __forceinline__ void init(const TcDirect& d, long long pitch, long long pitch8) {
    const int r0 = static_cast<int>(threadIdx.x & 31) / CHUNKS;
    first = (r0 >> 3) * pitch8 + (r0 & 7) * pitch;
    rows = (1u << CHUNKS) - 1u;
    if (d.rows >= 32 && d.xs >= 8 && d.ys >= 4) return;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int r = r0 + i * (32 / CHUNKS);
      if (!(r < d.rows && (r & 7) < d.xs && (r >> 3) < d.ys)) rows &= ~(1u << i);
    }
  }
};

// The warp's 32 staged rows of 128 bytes (CHUNKS = 8 pieces of 16 bytes; int8: 64 bytes, 4 pieces) to the result.  Piece
// j of row r sits at piece j ^ (r & 7) of its row (64-byte rows: j ^ ((r >> 1) & 3)), so that both the row-wise writes
// and these line-wise reads meet every bank once.  The first `n0` bytes of a row belong to plane 0 at p0, the rest to
// plane 1 at p1 (two planes: n0 = 64); `have` bytes of each plane's part exist.
template <int CHUNKS>
__device__ __forceinline__ void tc_flush(uint32_t stage, long long pitch, long long pitch8, const TcFlushLane<CHUNKS>& fl, uint8_t* p0,
                                         uint8_t* p1, int n0, int have) {
  __syncwarp();
  const int lane = threadIdx.x & 31;
  const int piece = lane % CHUNKS, r0 = lane / CHUNKS;
  const int at = piece * 16;
  const bool second = at >= n0;
  uint8_t* const p = (second ? p1 + (at - n0) : p0 + at) + fl.first;
  const uint32_t rows = (second ? at - n0 : at) < have ? fl.rows : 0u;
  uint4 v[CHUNKS];
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    const int r = r0 + i * (32 / CHUNKS);
    const int swz = CHUNKS == 8 ? piece ^ (r & 7) : piece ^ ((r >> 1) & 3);
    v[i] = lds_16b(stage + static_cast<uint32_t>(r * CHUNKS * 16 + swz * 16));
  }
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    // CHUNKS = 8: rows r0 + 4 i; CHUNKS = 4: rows r0 + 8 i
    const long long off = CHUNKS == 8 ? (i >> 1) * pitch8 + (i & 1) * 4 * pitch : i * pitch8;
    if (rows & (1u << i)) *reinterpret_cast<uint4*>(p + off) = v[i];
  }
  __syncwarp();
}

// 16 per-column constants (zeros behind the end)
__device__ __forceinline__ void tc_load16(const float* p, int have, float (&b)[16]) {
  if (p == nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j) b[j] = 0.0f;
  } else if (have >= 16) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(p) + q);
      b[4 * q] = t.x, b[4 * q + 1] = t.y, b[4 * q + 2] = t.z, b[4 * q + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) b[j] = j < have ? __ldg(p + j) : 0.0f;
  }
}

// What 16 columns of a row meet besides their accumulator: bias, dequantisation factor and residual.
template <int KIND, bool RES>
struct TcOperands {
  static constexpr int RW = !RES ? 1 : (KIND == GEMM_TF32X3 ? 32 : 16);  // residual words: 16 fp32, 8 + 8 of a bf16 pair, or 16 + 16 of a split pair
  uint32_t r[RW];
  float bias[16], scale[16];
  // those of columns c to c + 15, of which `have` exist (none: nothing is read)
  __device__ __forceinline__ void fetch(const TcDirect& d, int c, int have, bool valid) {
    tc_load16(d.bias != nullptr ? d.bias + c : nullptr, have, bias);
    if (KIND == GEMM_I8) tc_load16(d.scale + c, have, scale);
    if (!RES) return;
    if (!valid) {
#pragma unroll
      for (int j = 0; j < RW; ++j) r[j] = 0u;
    } else if (d.res_mode == RES_BF16X2) {
      tc_row_load<32>(d.r0 + 2 * c, r, 2 * have, d.wide);
      tc_row_load<32>(d.r1 + 2 * c, r + (RES ? 8 : 0), 2 * have, d.wide);
    } else {
      tc_row_load<64>(d.r0 + 4 * c, r, 4 * have, d.wide);
      if (KIND == GEMM_TF32X3 && d.res_mode == RES_SPLIT) tc_row_load<64>(d.r1 + 4 * c, r + (RW == 32 ? 16 : 0), 4 * have, d.wide);
    }
  }
};

template <int KIND, int OUT, bool RES, bool SIDE, bool FIX>
__device__ __forceinline__ void tc_drain_as(const TcDirect& d, uint32_t t_row, int cols, int left, bool valid, TcOperands<KIND, RES>& ops) {
  using namespace ptx;
  constexpr int RW = TcOperands<KIND, RES>::RW;
  const int row = threadIdx.x & 31;
  const uint32_t stage_row = d.stage + static_cast<uint32_t>(row) * 128u;
  TcFlushLane<OUT == OUT_I8 ? 4 : 8> fl;
  if (OUT != OUT_CHW) fl.init(d, d.pitch, d.pitch8);
  TcFlushLane<4> side_fl;
  if (SIDE) side_fl.init(d, d.side_pitch, d.side_pitch8);
  uint32_t nxt[16];
  uint32_t(&r)[RW] = ops.r;
  float(&bias)[16] = ops.bias, (&scale)[16] = ops.scale;
  tmem_ld16(t_row, nxt);
#pragma unroll 1
  for (int c = 0; c < cols; c += 16) {
    const int have = left - c;  // columns from here on
    const bool more = c + 16 < cols;
    float y[16];
    tmem_ld_wait();
    if (FIX && d.fix_count > 0 && valid) {
      const uint32_t* src = d.fix_ws + static_cast<size_t>(c >> 4) * 128 * 16;
      uint32_t sum[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) sum[j] = 0u;
      for (int i = 0; i < d.fix_count; ++i) {
        // (written by other SMs during this launch: read from L2, never through L1)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 a = __ldcg(reinterpret_cast<const uint4*>(src) + q);
          const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (KIND == GEMM_I8) sum[4 * q + e] += w[e];
            else sum[4 * q + e] = __float_as_uint(__fadd_rn(__uint_as_float(sum[4 * q + e]), __uint_as_float(w[e])));
          }
        }
        src += d.fix_stride;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (KIND == GEMM_I8) nxt[j] += sum[j];
        else nxt[j] = __float_as_uint(__fadd_rn(__uint_as_float(nxt[j]), __uint_as_float(sum[j])));
      }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float t = KIND == GEMM_I8 ? __fmul_rn(static_cast<float>(static_cast<int>(nxt[j])), scale[j]) : __uint_as_float(nxt[j]);
      y[j] = __fadd_rn(t, bias[j]);
    }
    if (RES) {
      if (d.res_mode == RES_BF16X2) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          y[2 * e] = __fadd_rn(y[2 * e], __fadd_rn(bf16_low(r[e % RW]), bf16_low(r[(8 + e) % RW])));
          y[2 * e + 1] = __fadd_rn(y[2 * e + 1], __fadd_rn(bf16_high(r[e % RW]), bf16_high(r[(8 + e) % RW])));
        }
      } else {
        const bool split = KIND == GEMM_TF32X3 && d.res_mode == RES_SPLIT;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float t = __uint_as_float(r[j % RW]);
          if (split) t = __fadd_rn(t, __uint_as_float(r[(16 + j) % RW]));
          y[j] = __fadd_rn(y[j], t);
        }
      }
    }
    if (more) {
      // the next 16 columns' operands are on their way while these are finished and stored
      tmem_ld16(t_row + static_cast<uint32_t>(c + 16), nxt);
      ops.fetch(d, c + 16, have - 16, valid);
    }
    if (OUT == OUT_I8) {
      // requantise, clamp at zero for a fused ReLU (the order of the reference's int8 path)
      uint32_t w[4];
      if (d.act == ACT_RELU) {
#pragma unroll
        for (int g = 0; g < 4; ++g) w[g] = quantize4_at_zero(y[4 * g], y[4 * g + 1], y[4 * g + 2], y[4 * g + 3], d.out_scale);
      } else {
#pragma unroll
        for (int g = 0; g < 4; ++g) w[g] = quantize4(y[4 * g], y[4 * g + 1], y[4 * g + 2], y[4 * g + 3], d.out_scale);
      }
      const int piece = (c >> 4) & 3;
      sts_16b(d.stage + static_cast<uint32_t>(row * 64 + ((piece ^ ((row >> 1) & 3)) << 4)), w);
      if (piece == 3 || !more) {
        const int c64 = c & ~63;
        if constexpr (OUT == OUT_I8) tc_flush<4>(d.stage, d.pitch, d.pitch8, fl, d.o0 + c64, nullptr, 64, min(left - c64, c - c64 + 16));
      }
      continue;
    }
    if (d.act == ACT_RELU) {
#pragma unroll
      for (int j = 0; j < 16; ++j) y[j] = fmaxf(y[j], 0.0f);
    } else if (d.act == ACT_CLIP) {
#pragma unroll
      for (int j = 0; j < 16; ++j) y[j] = fminf(fmaxf(y[j], d.act_a), d.act_b);
    } else if (d.act != ACT_NONE) {
      float t[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) t[j] = y[j];
      tc_act_many(t, d.act, d.act_a, d.act_b);
#pragma unroll
      for (int j = 0; j < 16; ++j) y[j] = t[j];
    }
    if (SIDE) {
      // int8 copies, 64 columns to a flush
      const int piece = (c >> 4) & 3, c64 = c & ~63;
      const uint32_t at = d.side_stage + static_cast<uint32_t>(row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
      tc_stage_side_quant(at, d.side_scale0, d.act == ACT_RELU && d.side_scale0 >= 0.0f, y);
      if (d.side_count > 1) tc_stage_side_quant(at + kDrainSideBytes, d.side_scale1, d.act == ACT_RELU && d.side_scale1 >= 0.0f, y);
      if (piece == 3 || !more) {
        const int n = min(left - c64, c - c64 + 16);
        tc_flush<4>(d.side_stage, d.side_pitch, d.side_pitch8, side_fl, d.side_q0 + c64, nullptr, 64, n);
        if (d.side_count > 1)
          tc_flush<4>(d.side_stage + kDrainSideBytes, d.side_pitch, d.side_pitch8, side_fl, d.side_q1 + c64, nullptr, 64, n);
      }
    }
    if (OUT == OUT_CHW) {
      // neighbouring lanes are neighbouring pixels: every store is 128 consecutive bytes of a channel plane
      float* o = reinterpret_cast<float*>(d.o0) + c * d.chw;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < have && valid) o[j * d.chw] = y[j];
      continue;
    }
    const int h = (c >> 4) & 1;  // which half of a 32-column step
    const int c32 = c & ~31;
    const bool full = h == 1 || !more;
    const int step_cols = min(left - c32, c - c32 + 16);  // columns staged when the step is complete
    auto put = [&](int piece, const uint32_t* w) { sts_16b(stage_row + static_cast<uint32_t>((piece ^ (row & 7)) << 4), w); };
    if constexpr (OUT == OUT_BF16X2) {
      uint32_t hi[8], mid[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) split_bf16x2(y[2 * e], y[2 * e + 1], hi[e], mid[e]);
      put(2 * h, hi);
      put(2 * h + 1, hi + 4);
      put(4 + 2 * h, mid);
      put(4 + 2 * h + 1, mid + 4);
      if (full) tc_flush<8>(d.stage, d.pitch, d.pitch8, fl, d.o0 + 2 * c32, d.o1 + 2 * c32, 64, 2 * step_cols);
    } else if constexpr (OUT == OUT_F32_SPLIT) {
      uint32_t w[16], lo[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float hi = round_tf32(y[j]);
        w[j] = __float_as_uint(hi);
        lo[j] = __float_as_uint(__fadd_rn(y[j], -hi));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        put(q, w + 4 * q);
        put(4 + q, lo + 4 * q);
      }
      tc_flush<8>(d.stage, d.pitch, d.pitch8, fl, d.o0 + 4 * c, d.o1 + 4 * c, 64, 4 * min(have, 16));
    } else if constexpr (OUT == OUT_F32 || OUT == OUT_F32_TF32) {
      uint32_t w[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) w[j] = __float_as_uint(OUT == OUT_F32_TF32 ? round_tf32(y[j]) : y[j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) put(4 * h + q, w + 4 * q);
      if (full) tc_flush<8>(d.stage, d.pitch, d.pitch8, fl, d.o0 + 4 * c32, nullptr, 128, 4 * step_cols);
    }
  }
}

// The epilogue a kernel is compiled with: an output format, with or without a residual.  One kernel per form: a kernel
// with all of them behind run-time branches spends its tiles on instruction fetch (24 -> 144 channels, 64 images of 112 x 112:
// 233 us with ten forms in one kernel, 198 with eight, 176 with one).
constexpr int epi_form(int out_mode, bool res) { return out_mode * 2 + (res ? 1 : 0); }
constexpr int kEpiAny = -1;  // element by element, any format and alignment

// Drains `cols` accumulator columns (a multiple of 16) of this warp's 32 rows, of which `left` exist in the result (a
// multiple of the 16-byte piece of every format involved).  `valid`: this thread's row exists.  Every lane of the warp
// must call it.  SIDE: int8 copies may take part; FIX: partial accumulators may.  `ops`: the first 16 columns' operands,
// which a caller fetches before it waits for the accumulator (a tile alone in the pipeline otherwise pays their way from
// L2 or HBM after its last product).
template <int KIND, int EPI, bool SIDE, bool FIX>
__device__ __forceinline__ void tc_drain(const TcDirect& d, uint32_t t_row, int cols, int left, bool valid, TcOperands<KIND, EPI % 2 == 1>& ops) {
  if (cols > left) cols = (left + 15) & ~15;
  if (cols <= 0) return;
  tc_drain_as<KIND, EPI / 2, EPI % 2 == 1, SIDE, FIX>(d, t_row, cols, left, valid, ops);
}
template <int KIND, int EPI, bool SIDE, bool FIX>
__device__ __forceinline__ void tc_drain(const TcDirect& d, uint32_t t_row, int cols, int left, bool valid) {
  TcOperands<KIND, EPI % 2 == 1> ops;
  ops.fetch(d, 0, left, valid);
  tc_drain<KIND, EPI, SIDE, FIX>(d, t_row, cols, left, valid, ops);
}

}  // namespace nb
