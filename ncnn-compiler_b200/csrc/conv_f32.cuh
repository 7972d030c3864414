// fp32 convolution and InnerProduct / Gemm on the CUDA cores: every product and sum an fp32 fused multiply-add.
// Serves the CUDA-core accuracy mode and the fp32 layers whose channel counts the tensor-core path cannot address.
//
// out[m][o] = epilogue(sum_k A[m][k] * W[k][o]), A gathered from the channel-last activations (k = filter tap x
// channel), W stored in pairs of k ([K/2][O][2], f32_weight_at).  A block computes BM x 64 results with 8 x 8 per
// thread (8 warps on an SM); K advances in steps of 16 through a ring of cp.async stages, so that global latency is
// hidden by the two steps in flight.
//
// What bounds it: the FMA pipe (128 fp32 lanes per SM, 74 TFLOP/s at 1965 MHz).  The inner loop uses packed
// fma.rn.f32x2, which runs at the same rate with half the issue slots.  A pair is the even and the odd k of one result
// (two running sums, added at the end of a chunk): both operands then come out of shared memory as the pairs they are.
// Pairs of results instead need every A value twice, and those moves hold the pipe at three quarters of its rate.
// A stays in [row][k] order (16 + 4 floats a row, so that the rows a warp reads fall into different banks) and needs no
// transposition on the way in.
// ResNet-18, 8 images (29 GFLOP): 8.94 ms (3.3 TFLOP/s) with one thread per result -> 1.09 ms (27 TFLOP/s).
//
// Sums: K is cut into chunks of at most kF32Chunk elements, each summed in order and the chunk sums added in order.
// The cut depends on the layer alone.  Where there are too few tiles to fill the GPU, a tile's chunks go to different
// blocks and the last one to finish adds them up in the same order: the same bits for every batch size.  Chunks of 256:
// one ResNet-18 image takes 0.46 ms (0.60 with chunks of 512), eight 1.09 (1.05).
#pragma once

#include "kernels.cuh"

namespace nb {

constexpr int kF32Chunk = 256;
constexpr int kF32Bk = 16;
constexpr int kF32Bn = 64;
constexpr int kF32Stages = 3;
constexpr int kF32Ak = kF32Bk + 4;  // row pitch of A in shared memory

struct F32ConvParams {
  ConvGeom g;              // (InnerProduct: H = W = OH = OW = KH = KW = 1, C = K, images = M)
  const float* weights;    // [K/2][O][2], K = KH*KW*C rounded up to even (zero weight)
  ConvEpilogue e;          // e.bias is added to the finished sum
  int K, chunks, chunk_k;  // chunk_k: elements per chunk, a multiple of kF32Bk
  int split;               // 1: blockIdx.y is the chunk
  int tiles_n;
  int vec_a, vec_b, vec_o; // 16-byte pieces: C a multiple of 4, O of 2, O of 4 (and the arrays aligned)
  int plain;               // fp32 out, fp32 residual or none, O a multiple of 4, activation none / ReLU / clip:
  float clamp_lo, clamp_hi;  // the bounds of that activation
  float* partials;         // split: [tile][chunk][BM][64]
  int* counters;           // split: one per tile, zero between launches
};

// chunks of a contraction of K elements and elements per chunk
inline void f32_chunks(int K, int* chunks, int* chunk_k) {
  const int c = (K + kF32Chunk - 1) / kF32Chunk;
  *chunk_k = ((K + c - 1) / c + kF32Bk - 1) / kF32Bk * kF32Bk;
  *chunks = (K + *chunk_k - 1) / *chunk_k;
}

__device__ __forceinline__ void cp_async_4(uint32_t smem_dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_dst), "l"(src), "r"(src_bytes) : "memory");
}

template <int BM>
static __global__ void __launch_bounds__(BM, 256 / BM) k_conv_f32(const float* __restrict__ x, ActRef out, const F32ConvParams p) {
  ptx::grid_begin();
  constexpr int NT = BM;  // 8 x 8 results per thread
  constexpr int TX = kF32Bn / 8;
  constexpr int TY = NT / TX;  // thread (ty, tx): rows ty + TY * i, columns 16 * j + 2 * tx + {0, 1}
  constexpr int A_STAGE = BM * kF32Ak, B_STAGE = kF32Bk * kF32Bn;
  constexpr int A_ROWS = BM * 4 / NT;           // 16-byte pieces of A per thread and step
  constexpr int B_PIECES = B_STAGE / 4 / NT;
  extern __shared__ __align__(16) float f32_smem[];
  __shared__ int3 row_at[BM];  // single-element loads: first pixel of the image, row and column of the filter origin
  float* sa = f32_smem;
  float* sb = f32_smem + kF32Stages * A_STAGE;
  float* sum = sb + kF32Stages * B_STAGE;  // [BM][64] sums of the finished chunks
  const ConvGeom& g = p.g;
  const int tid = threadIdx.x;
  const int tile = blockIdx.x;
  const int m_blk = tile / p.tiles_n, n_blk = tile - m_blk * p.tiles_n;
  const int m0 = m_blk * BM;  // (fewer than 2^31 rows and input pixels: the dispatch checks)
  const int n0 = n_blk * kF32Bn;
  const int M = static_cast<int>(g.images) * g.OH * g.OW;
  const int ohw = g.OH * g.OW;
  const int chunk0 = p.split ? static_cast<int>(blockIdx.y) : 0;
  const int chunk1 = p.split ? chunk0 + 1 : p.chunks;

  // A: this thread's pieces are column piece `apc` of rows arow + i * (NT / 4); with single elements (channel counts that
  // are no multiple of 4) element `tid % 16` of rows tid / 16 + i * (NT / 16), whose pixels are looked up per step
  const int apc = tid & 3, arow = tid >> 2;
  int a_img[A_ROWS], a_h[A_ROWS], a_w[A_ROWS];
#pragma unroll
  for (int i = 0; i < A_ROWS; ++i) {
    const int m = m0 + arow + i * (NT / 4);
    const int img = m / ohw;
    const int r = m - img * ohw;
    const int oh = r / g.OW;
    a_img[i] = img * g.H * g.W;
    a_h[i] = m < M ? oh * g.sh - g.pt : -(1 << 28);  // a row past the end lies outside every image
    a_w[i] = (r - oh * g.OW) * g.sw - g.pl;
    if (!p.vec_a && apc == 0) row_at[arow + i * (NT / 4)] = make_int3(a_img[i], a_h[i], a_w[i]);
  }
  if (!p.vec_a) __syncthreads();
  const uint32_t sa_u = static_cast<uint32_t>(__cvta_generic_to_shared(sa));
  const uint32_t sb_u = static_cast<uint32_t>(__cvta_generic_to_shared(sb));

  // channel and filter tap of this thread's next piece (stepped: a division per step is a long serial chain)
  const int k_begin = chunk0 * p.chunk_k;
  int k = k_begin + (p.vec_a ? apc * 4 : tid & 15);
  int c = k % g.C, kh = k / g.C / g.KW, kw = k / g.C - kh * g.KW;
  // (whole pieces: pointer and validity per row change with the tap only)
  const float* a_src[A_ROWS];
  bool a_in[A_ROWS];
  auto aim_a = [&]() {
    const int dh = kh * g.dh, dw = kw * g.dw;
#pragma unroll
    for (int i = 0; i < A_ROWS; ++i) {
      const int h = a_h[i] + dh, w = a_w[i] + dw;
      a_in[i] = k < p.K && static_cast<unsigned>(h) < static_cast<unsigned>(g.H) && static_cast<unsigned>(w) < static_cast<unsigned>(g.W);
      a_src[i] = a_in[i] ? x + static_cast<long long>(a_img[i] + h * g.W + w) * g.C + c : x;
    }
  };
  aim_a();
  auto load_a = [&](int stage) {
    if (p.vec_a) {
#pragma unroll
      for (int i = 0; i < A_ROWS; ++i) {
        cp_async_16(sa + stage * A_STAGE + (arow + i * (NT / 4)) * kF32Ak + apc * 4, a_src[i], a_in[i] ? 16 : 0);
        a_src[i] += a_in[i] ? kF32Bk : 0;
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < BM * 16 / NT; ++i) {
        const int row = (tid >> 4) + i * (NT / 16);
        const int3 at = row_at[row];
        const int h = at.y + kh * g.dh, w = at.z + kw * g.dw;
        const bool in = k < p.K && static_cast<unsigned>(h) < static_cast<unsigned>(g.H) && static_cast<unsigned>(w) < static_cast<unsigned>(g.W);
        const float* src = in ? x + static_cast<long long>(at.x + h * g.W + w) * g.C + c : x;
        cp_async_4(sa_u + static_cast<uint32_t>(stage * A_STAGE + row * kF32Ak + (tid & 15)) * 4u, src, in ? 4 : 0);
      }
    }
    k += kF32Bk;
    c += kF32Bk;
    if (c >= g.C) {
      do {
        c -= g.C;
        if (++kw == g.KW) {
          kw = 0;
          ++kh;
        }
      } while (c >= g.C);
      if (p.vec_a) aim_a();
    }
  };
  const float* b_src = p.weights + (static_cast<long long>(k_begin / 2 + (tid >> 5)) * g.O + n0 + (tid & 31) * 2) * 2;
  const long long b_piece = static_cast<long long>(NT / 32) * g.O * 2, b_step = static_cast<long long>(kF32Bk) * g.O;
  const bool b_in = n0 + (tid & 31) * 2 < g.O;
  auto load_b = [&](int stage, int k0) {
    // 8 rows of k pairs, 64 columns x 2 floats each
    if (p.vec_b) {
#pragma unroll
      for (int i = 0; i < B_PIECES; ++i) {
        const bool in = b_in && k0 + 2 * ((tid >> 5) + i * (NT / 32)) < p.K;
        cp_async_16(sb + stage * B_STAGE + (tid + i * NT) * 4, in ? b_src + i * b_piece : p.weights, in ? 16 : 0);
      }
      b_src += b_step;
    } else {
#pragma unroll 4
      for (int i = 0; i < B_STAGE / NT; ++i) {
        const int e = tid + i * NT;
        const int kr = e >> 7, n2 = e & 127;
        const bool in = k0 + 2 * kr < p.K && n0 + n2 / 2 < g.O;
        cp_async_4(sb_u + static_cast<uint32_t>(stage * B_STAGE + e) * 4u, in ? p.weights + (static_cast<long long>(k0 / 2 + kr) * g.O + n0) * 2 + n2 : p.weights, in ? 4 : 0);
      }
    }
  };

  const int tx = tid % TX, ty = tid / TX;
  uint64_t acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  bool first_chunk = true;
  // end of a chunk: even and odd sums together, onto the chunks before (this thread's own entries of `sum`)
  auto close_chunk = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2* at = reinterpret_cast<float2*>(sum + (ty + i * TY) * kF32Bn + 16 * j + 2 * tx);
        const float2 u = f32x2_get(acc[i][2 * j]), v = f32x2_get(acc[i][2 * j + 1]);
        float2 t = make_float2(__fadd_rn(u.x, u.y), __fadd_rn(v.x, v.y));
        if (!first_chunk) {
          const float2 before = *at;
          t = make_float2(__fadd_rn(before.x, t.x), __fadd_rn(before.y, t.y));
        }
        *at = t;
        acc[i][2 * j] = acc[i][2 * j + 1] = 0ull;
      }
    first_chunk = false;
  };

  const int k_end = min(p.K, chunk1 * p.chunk_k);
  const int steps = (k_end - k_begin + kF32Bk - 1) / kF32Bk;
  const int steps_per_chunk = p.chunk_k / kF32Bk;
#pragma unroll
  for (int s = 0; s < kF32Stages - 1; ++s) {
    if (s < steps) {
      load_a(s);
      load_b(s, k_begin + s * kF32Bk);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int stage = 0, fill = kF32Stages - 1, in_chunk = 0;
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kF32Stages - 2) : "memory");
    __syncthreads();  // step s has landed for every thread, and every thread has left the stage filled below
    if (s + kF32Stages - 1 < steps) {
      load_a(fill);
      load_b(fill, k_begin + (s + kF32Stages - 1) * kF32Bk);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* pa = sa + stage * A_STAGE + ty * kF32Ak;
    const float* pb = sb + stage * B_STAGE + tx * 4;  // (column pair 2 tx, both k: four floats)
#pragma unroll
    for (int kq = 0; kq < kF32Bk / 2; ++kq) {
      uint64_t a[8];
      ulonglong2 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(pb + kq * 2 * kF32Bn + 32 * j);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const uint64_t*>(pa + i * TY * kF32Ak + kq * 2);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          f32x2_fma(acc[i][2 * j], a[i], b[j].x);
          f32x2_fma(acc[i][2 * j + 1], a[i], b[j].y);
        }
    }
    if (++stage == kF32Stages) stage = 0;
    if (++fill == kF32Stages) fill = 0;
    if (++in_chunk == steps_per_chunk) {
      in_chunk = 0;
      close_chunk();
    }
  }
  if (in_chunk != 0) close_chunk();
  __syncthreads();  // from here on a thread handles four neighbouring columns of eight rows

  constexpr int ROWS = NT / 16;
  const int n = n0 + (tid & 15) * 4, r0 = tid >> 4;
  const float4* sum4 = reinterpret_cast<const float4*>(sum);
  float4* sum4w = reinterpret_cast<float4*>(sum);
  if (p.split) {
    // this chunk's sums to the workspace; the block that finishes last adds the tile's chunks in order
    __shared__ int last;
    float4* ws = reinterpret_cast<float4*>(p.partials) + static_cast<size_t>(tile) * p.chunks * BM * 16 + tid;
#pragma unroll
    for (int i = 0; i < 16; ++i) __stcg(ws + (static_cast<size_t>(chunk0) * 16 + i) * NT, sum4[i * NT + tid]);
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      last = atomicAdd(p.counters + tile, 1) == p.chunks - 1 ? 1 : 0;
      if (last) p.counters[tile] = 0;  // as the next launch expects it
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 t[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = __ldcg(ws + static_cast<size_t>(h * 8 + i) * NT);
      for (int ch = 1; ch < p.chunks; ++ch) {
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __ldcg(ws + (static_cast<size_t>(ch) * 16 + h * 8 + i) * NT);
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = make_float4(__fadd_rn(t[i].x, v[i].x), __fadd_rn(t[i].y, v[i].y), __fadd_rn(t[i].z, v[i].z), __fadd_rn(t[i].w, v[i].w));
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) sum4w[(h * 8 + i) * NT + tid] = t[i];  // (read again by this thread alone)
    }
  }
  if (n >= g.O) return;
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.e.bias != nullptr) {
    b.x = __ldg(p.e.bias + n);
    b.y = n + 1 < g.O ? __ldg(p.e.bias + n + 1) : 0.0f;
    b.z = n + 2 < g.O ? __ldg(p.e.bias + n + 2) : 0.0f;
    b.w = n + 3 < g.O ? __ldg(p.e.bias + n + 3) : 0.0f;
  }
  if (p.plain) {
    // fp32 rows, a clamp (or nothing) for an activation: what every layer of the CUDA-core mode has
#pragma unroll
    for (int h = 0; h < 8 / 4 * 2; ++h) {
      float4 y[4], r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = m0 + r0 + (4 * h + i) * ROWS;
        r[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.e.has_res && m < M) r[i] = *reinterpret_cast<const float4*>(p.e.res.p0 + static_cast<long long>(m) * g.O + n);
        y[i] = sum4[(4 * h + i) * NT + tid];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = m0 + r0 + (4 * h + i) * ROWS;
        y[i].x = fminf(fmaxf(__fadd_rn(__fadd_rn(y[i].x, b.x), r[i].x), p.clamp_lo), p.clamp_hi);
        y[i].y = fminf(fmaxf(__fadd_rn(__fadd_rn(y[i].y, b.y), r[i].y), p.clamp_lo), p.clamp_hi);
        y[i].z = fminf(fmaxf(__fadd_rn(__fadd_rn(y[i].z, b.z), r[i].z), p.clamp_lo), p.clamp_hi);
        y[i].w = fminf(fmaxf(__fadd_rn(__fadd_rn(y[i].w, b.w), r[i].w), p.clamp_lo), p.clamp_hi);
        if (m < M) *reinterpret_cast<float4*>(out.p0 + static_cast<long long>(m) * g.O + n) = y[i];
      }
    }
    return;
  }
  // one rolled loop: inlined copies of activation and store cost more in instruction fetch than a short layer's math
#pragma unroll 1
  for (int i = 0; i < 16; ++i) {
    const int m = m0 + r0 + i * ROWS;
    if (m >= M) break;
    float4 y = sum4[i * NT + tid];
    const long long o = static_cast<long long>(m) * g.O + n;
    y = make_float4(__fadd_rn(y.x, b.x), __fadd_rn(y.y, b.y), __fadd_rn(y.z, b.z), __fadd_rn(y.w, b.w));
    if (p.vec_o) {
      const float4 r = p.e.has_res ? act_load4(p.e.res, o) : make_float4(0.f, 0.f, 0.f, 0.f);
      act_store4(out, o, make_float4(conv_finish_f32(p.e, y.x, r.x), conv_finish_f32(p.e, y.y, r.y),
                                     conv_finish_f32(p.e, y.z, r.z), conv_finish_f32(p.e, y.w, r.w)));
    } else {
      const float v[4] = {y.x, y.y, y.z, y.w};
      for (int q = 0; q < 4 && n + q < g.O; ++q)
        act_store(out, o + q, conv_finish_f32(p.e, v[q], p.e.has_res ? act_load(p.e.res, o + q) : 0.0f));
    }
  }
}

// ---- InnerProduct / Gemm of few rows, fp32 on the CUDA cores: one pass over the weights for every 16 rows.
//
// k_conv_f32's tiles of 64 rows read every weight once too, but a block's 16 k at a time, and multiply mostly zeros.  Here a
// warp takes 32 columns of one chunk of K and requests all its weights (up to 32 KB) before it waits for the first; ROWS
// running pairs of sums per column, the rows of x broadcast from shared memory.  The chunks and the order of every sum are
// k_conv_f32's, so the results are its bits.
// Whole calls in us, tiles -> this kernel (the same bits, so the batch may decide):
//            512 -> 1000     1001 -> 1537    3001 -> 2501    4095 -> 4091    4097 -> 515     255 -> 33
//   1 row    22.6 -> 8.4     45.1 -> 10.3    65.6 -> 13.6   120.5 -> 19.7    49.3 -> 12.4    41.1 -> 8.3
//   8 rows   22.6 -> 12.4    45.2 -> 14.4    65.6 -> 22.1   120.9 -> 28.8    51.3 -> 16.5    41.1 -> 12.4
//   16 rows  22.6 -> 16.5    47.2 -> 20.6    67.7 -> 30.9   122.9 -> 51.5    51.3 -> 20.6    43.1 -> 14.5
//   32       22.6 -> 16.7    49.3 -> 20.6    69.7 -> 49.8   126.9 -> 90.1    55.4 -> 22.6    45.3 -> 16.5
//   48       22.6 -> 18.5    53.2 -> 22.6    73.8 -> 65.6   131.1 -> 127.3   57.5 -> 32.9    49.3 -> 16.5
//   64       22.6 -> 18.5    55.4 -> 32.5    76.1 -> 82.4   134.6 -> 163.8   61.4 -> 34.5    51.3 -> 16.5
// One group of 16 rows always takes it.  More groups bring every weight out of L2 again, and the tiles are slower where their
// operands come element by element (K, or the columns, no multiple of 4); so from 17 rows to kRowsF32Most the two are compared
// by an estimate fitted to 299 calls (K 130 to 4095, 33 to 12000 columns, 17 to 128 rows), of which it picks the slower form in
// 17, by 4 to 18 %:
//            300 -> 12000    513 -> 7000     700 -> 7000     1001 -> 2501    1001 -> 12000   4095 -> 2501
//   17       25.0 / 35.5!    39.3 -> 33.0    33.1 / 39.3!    47.6 -> 27.0    80.3 -> 69.4   102.8 -> 60.3    (! tiles stay)
//   48       24.9 / 51.7!    40.2 / 47.6!    33.2 / 57.7!    53.6 -> 33.0    82.4 / 102.8!  108.9 -> 85.0
//   96                       61.8 / 83.3!                    70.0 -> 53.7                   162.2 / 153.2!
// 7 -> 5: 8 rows 8.3 -> 6.2, 16 rows 8.4 -> 10.3: short rows take it up to eight.
// The chunks of all 32-column blocks meet in the workspace of split contractions (21 MB, 16384 counters): with 4096 inputs that is
// one row through 327680 columns, 8 through 40960, 16 through 20480; wider calls stay on tiles.  Beyond the 640 counters that
// other kernels share: 513 -> 20512, one row 71.9 -> 14.5, 16 rows 73.9 -> 49.3; 4096 -> 32000, one row 445 -> 139, 8 rows 445 -> 199.
// What bounds it: one row, the weights' way from HBM (4095 -> 4091: 67 MB at 3.4 TB/s, launch included); many rows, the 48 KB
// of a warp, of which an SM holds four, and the broadcasts (one 16-byte read for two packed FMAs).
constexpr int kRowsF32Cols = 32;
constexpr int kRowsF32Max = 16;    // rows of a warp
constexpr int kRowsF32Most = 128;  // rows of a call

__device__ __forceinline__ void cp_async_8(uint32_t smem_dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_dst), "l"(src) : "memory");
}

template <int ROWS>
static __global__ void __launch_bounds__(kRowsF32Cols) k_rows_f32(const float* __restrict__ x, ActRef out, const F32ConvParams p) {
  ptx::grid_dependency_trigger();
  constexpr int PAIRS = kF32Chunk / 2;
  __shared__ __align__(16) uint64_t sw[PAIRS][kRowsF32Cols];
  __shared__ __align__(16) float sx[ROWS][kF32Chunk];
  const int lane = threadIdx.x, chunk = blockIdx.y, row0 = blockIdx.z * ROWS;
  const int tile = blockIdx.x + blockIdx.z * gridDim.x;
  const int o = blockIdx.x * kRowsF32Cols + lane, O = p.g.O, M = static_cast<int>(p.g.images) - row0;
  const int k_begin = chunk * p.chunk_k, k_end = min(p.K, k_begin + p.chunk_k);
  const int pairs = (k_end - k_begin + 1) / 2;
  const bool in = o < O;
  // (no kernel writes weights: they come while the kernel before this one runs)
  const float* w = p.weights + (static_cast<long long>(k_begin / 2) * O + (in ? o : 0)) * 2;
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&sw[0][lane]));
#pragma unroll 16
  for (int j = 0; j < pairs; ++j) cp_async_8(dst + static_cast<uint32_t>(j) * (kRowsF32Cols * 8), w + static_cast<long long>(j) * O * 2);
  if (pairs & 1) sw[pairs][lane] = 0ull;  // (pairs are taken two at a time; a chunk holds an even number unless it is the last)
  ptx::grid_dependency_wait();
  const uint32_t xdst = static_cast<uint32_t>(__cvta_generic_to_shared(&sx[0][lane]));
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float* row = x + static_cast<long long>(row0 + r) * p.K + k_begin;
#pragma unroll 8
    for (int k = lane; k < 4 * ((pairs + 1) / 2); k += kRowsF32Cols) {
      const bool there = r < M && k_begin + k < k_end;
      cp_async_4(xdst + static_cast<uint32_t>(r * kF32Chunk + k - lane) * 4u, there ? row + k : x, there ? 4 : 0);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  uint64_t acc[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r] = 0ull;
#pragma unroll 4
  for (int j = 0; j < pairs; j += 2) {
    const uint64_t w0 = sw[j][lane], w1 = sw[j + 1][lane];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&sx[r][2 * j]);
      f32x2_fma(acc[r], a.x, w0);
      f32x2_fma(acc[r], a.y, w1);
    }
  }
  float y[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float2 t = f32x2_get(acc[r]);
    y[r] = __fadd_rn(t.x, t.y);
  }
  if (p.chunks > 1) {
    // the block that finishes a tile last adds its chunks in order
    float* const ws = p.partials + static_cast<size_t>(tile) * p.chunks * ROWS * kRowsF32Cols + lane;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) __stcg(ws + (chunk * ROWS + r) * kRowsF32Cols, y[r]);
    __threadfence();
    __syncwarp();
    int before = 0;
    if (lane == 0) before = atomicAdd(p.counters + tile, 1);
    if (__shfl_sync(0xffffffffu, before, 0) != p.chunks - 1) return;
    if (lane == 0) p.counters[tile] = 0;  // as the next launch expects it
    __threadfence();
#pragma unroll
    for (int r = 0; r < ROWS; ++r) y[r] = __ldcg(ws + r * kRowsF32Cols);
#pragma unroll 2
    for (int c = 1; c < p.chunks; ++c)
#pragma unroll
      for (int r = 0; r < ROWS; ++r) y[r] = __fadd_rn(y[r], __ldcg(ws + (c * ROWS + r) * kRowsF32Cols));
  }
  if (!in) return;
  const float b = p.e.bias != nullptr ? __ldg(p.e.bias + o) : 0.0f;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (r >= M) break;
    const long long at = static_cast<long long>(row0 + r) * O + o;
    act_store(out, at, conv_finish_f32(p.e, __fadd_rn(y[r], b), p.e.has_res ? act_load(p.e.res, at) : 0.0f));
  }
}

constexpr int f32_smem_bytes(int bm) { return (kF32Stages * (bm * kF32Ak + kF32Bk * kF32Bn) + bm * kF32Bn) * 4; }

}  // namespace nb
