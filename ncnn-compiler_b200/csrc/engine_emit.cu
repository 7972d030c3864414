// Nodes -> kernel launches: every node of a plan becomes one Step (a closure that enqueues its kernel), and the
// edges between the caller's CHW arrays and the channel-last arena.
#include "engine_impl.h"

namespace nb {

static cudaError_t launch_ok() { return cudaGetLastError(); }

// Launches one of the plain kernels with programmatic stream serialisation, like the tensor-core kernels: its blocks are
// set up while the kernel before it drains, and wait (grid_begin) before they touch any tensor.  A single image's pass
// is a chain of launches of a few microseconds each, of which one or two were the gap to the next.
template <class... Params, class... Args>
static void launch_plain(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = tc_pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// fp32 contraction on the CUDA cores as a tiled kernel (conv_f32.cuh).  Needs plain fp32 input and 32-bit pixel numbers.
static bool conv_f32_applies(const ActRef& in, const ConvGeom& g) {
  const long long rows = g.images * g.OH * g.OW, pixels = g.images * g.H * g.W;
  return in.fmt == FMT_F32 && rows < (1ll << 30) && pixels < (1ll << 30) && static_cast<long long>(g.KH) * g.KW * g.C < (1ll << 30);
}
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

std::string EngineImpl::emit_conv_f32(Step* s, const ActRef& in, const ActRef& out, const void* w, const ConvGeom& g, const ConvEpilogue& e) {
  F32ConvParams p{};
  p.g = g;
  p.weights = static_cast<const float*>(w);
  p.e = e;
  p.K = g.KH * g.KW * g.C;
  f32_chunks(p.K, &p.chunks, &p.chunk_k);
  const long long rows = g.images * g.OH * g.OW;
  p.tiles_n = (g.O + kF32Bn - 1) / kF32Bn;
  // 128-row tiles move 25 % fewer operand bytes; 64-row tiles fill the last wave better.  Two 128-thread blocks or four
  // 64-thread blocks live on an SM, so the large tiles pay from about two full waves on.
  const bool large = (rows + 127) / 128 * p.tiles_n >= 4ll * sm_count_;
  const int bm = large ? 128 : 64;
  const long long tiles = (rows + bm - 1) / bm * p.tiles_n;
  // fewer tiles than the four blocks an SM holds: the chunks of a tile go to different blocks (as far as the workspace reaches)
  const size_t ws = static_cast<size_t>(tiles) * p.chunks * bm * kF32Bn * 4;
  p.split = !large && p.chunks > 1 && tiles < 4ll * sm_count_ && tiles <= kTcSplitFlagCount && ws <= kTcSplitWorkspaceBytes ? 1 : 0;
  p.partials = reinterpret_cast<float*>(d_split_ws_);
  p.counters = d_split_flags_;
  p.vec_a = g.C % 4 == 0 && aligned16(in.p0) ? 1 : 0;
  p.vec_b = g.O % 2 == 0 ? 1 : 0;
  p.vec_o = g.O % 4 == 0 ? 1 : 0;
  p.plain = p.vec_o && out.fmt == FMT_F32 && (!e.has_res || e.res.fmt == FMT_F32) && (e.act == ACT_NONE || e.act == ACT_RELU || e.act == ACT_CLIP) ? 1 : 0;
  p.clamp_lo = e.act == ACT_RELU ? 0.0f : (e.act == ACT_CLIP ? e.act_a : -std::numeric_limits<float>::infinity());
  p.clamp_hi = e.act == ACT_CLIP ? e.act_b : std::numeric_limits<float>::infinity();
  const float* x = in.p0;
  // a handful of rows: a pass over the weights (k_rows_f32, which says where; NCNN_B200_ROWS_F32=0: tiles everywhere)
  const int cols = (g.O + kRowsF32Cols - 1) / kRowsF32Cols;
  const long long groups = (rows + kRowsF32Max - 1) / kRowsF32Max, warps = cols * groups * p.chunks;
  const int warp_rows = rows <= 1 ? 1 : (rows <= 2 ? 2 : (rows <= 4 ? 4 : (rows <= 8 ? 8 : kRowsF32Max)));
  const bool flat = g.H == 1 && g.W == 1 && g.OH == 1 && g.OW == 1 && g.KH == 1 && g.KW == 1;
  // expected us (conv_f32.cuh): waves of warps or of 64-row tiles, each in chunks of up to 256 k
  const double places = 4.0 * sm_count_, chunk = p.chunk_k / 256.0;
  const double rows_us = chunk * (13.0 * static_cast<double>(warps) / places + 3.0) + 0.35 * static_cast<double>(groups);
  const double tile_waves = static_cast<double>(tiles) * (p.split ? p.chunks : 1) / places;
  const double tiles_us = chunk * (p.split ? 1 : p.chunks) * ((p.vec_a ? 12.0 : 28.0) * std::ceil(tile_waves) + 20.0 * tile_waves) + (p.vec_o ? 0.0 : 10.0);
  const bool few = p.K >= 128 ? groups == 1 || (rows <= kRowsF32Most && rows_us < tiles_us) : rows <= 8;
  if (flat && few && p.chunks < 65536 && !env_flag_off("NCNN_B200_ROWS_F32") &&
      (p.chunks == 1 || (cols * groups <= kTcFlagWords && static_cast<size_t>(warps) * warp_rows * kRowsF32Cols * 4 <= kTcSplitWorkspaceBytes))) {
    const dim3 rgrid(static_cast<unsigned>(cols), static_cast<unsigned>(p.chunks), static_cast<unsigned>(groups));
    s->kernel = "k_rows_f32";
    s->run = [=](cudaStream_t st) {
      if (warp_rows == 1) launch_plain(k_rows_f32<1>, rgrid, kRowsF32Cols, 0, st, x, out, p);
      else if (warp_rows == 2) launch_plain(k_rows_f32<2>, rgrid, kRowsF32Cols, 0, st, x, out, p);
      else if (warp_rows == 4) launch_plain(k_rows_f32<4>, rgrid, kRowsF32Cols, 0, st, x, out, p);
      else if (warp_rows == 8) launch_plain(k_rows_f32<8>, rgrid, kRowsF32Cols, 0, st, x, out, p);
      else launch_plain(k_rows_f32<kRowsF32Max>, rgrid, kRowsF32Cols, 0, st, x, out, p);
      return launch_ok();
    };
    return {};
  }
  const dim3 grid(static_cast<unsigned>(tiles), p.split ? p.chunks : 1);
  const cudaError_t ae = large ? cudaFuncSetAttribute(k_conv_f32<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_smem_bytes(128))
                               : cudaFuncSetAttribute(k_conv_f32<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_smem_bytes(64));
  if (ae != cudaSuccess) return cudaGetErrorString(ae);
  s->kernel = p.split ? "k_conv_f32:split" : "k_conv_f32";
  s->run = [=](cudaStream_t st) {
    if (large) launch_plain(k_conv_f32<128>, grid, 128, f32_smem_bytes(128), st, x, out, p);
    else launch_plain(k_conv_f32<64>, grid, 64, f32_smem_bytes(64), st, x, out, p);
    return launch_ok();
  };
  return {};
}


// Where the patch-resident kernel on CTA pairs beats the im2col kernel: layers of one 64-channel block and at most 64
// outputs, whose im2col tiles fetch every pixel nine times from L2 for few MMAs (64 -> 64 on 56x56, batch 64: 53.5
// against 60 us, 59.4 against 63.7 us with a residual; 128 channels tie, one image is 0.5-1.5 us slower), and whose
// 16x8 tiles overhang the image little and fill the SMs several times over.  With one channel block (and no chunks) both
// kernels add up an output's products in the same order, so the batch may decide.
static bool halo_pays(int kind, int channels, const Node& node, int64_t n, int sm_count) {
  if (kind != GEMM_BF16X3 || channels != 64 || node.O > 64 || node.KH * node.KW < 9 || node.KH * node.KW >= kTcChunkFrom) return false;
  const int64_t tiles = static_cast<int64_t>((node.OH + kHaloTileH - 1) / kHaloTileH) * ((node.OW + kHaloTileW - 1) / kHaloTileW);
  return n * tiles >= 4 * sm_count && static_cast<double>(node.OH) * node.OW >= 0.85 * (tiles * kHaloTileH * kHaloTileW);
}

// Where the depthwise layer inside a projection is a launch of its own again.  The fused kernel walks the channels in
// blocks of 32, ~1 us each and one after the other however few tiles there are; two launches cost ~5 us and a trip of the
// depthwise result through L2 that grows with the pixels.  Whole calls of one block, fused -> apart in us, on 14x14 maps
// but for the last column (16x16):
//   channels   192 (16x16)      240                384                576                768
//   images     1: 18.7 -> 19.0   1: 21.8 -> 20.7    1: 24.8 -> 20.7    1: 30.9 -> 22.8    1: 37.2 -> 24.8
//              2: 18.6 -> 19.3   4: 22.7 -> 23.0    6: 26.8 -> 24.8   16: 38.1 -> 34.6   16: 47.4 -> 43.0
//              4: 18.7 -> 20.7   8: 24.4 -> 26.5   16: 29.6 -> 30.4   32: 43.4 -> 45.3   24: 53.3 -> 51.5
// So it takes more than six blocks, and from there on few pixels.  The limit of two tiles of 128 lies below every crossover
// measured (700 pixels with 8 blocks, 2 500 with 12, 4 700 with 18): it keeps the small batches between in one kernel.
// The same products in the same order (below the depth that is summed in chunks), so the batch may decide.
static bool depthwise_apart(const Node& node, int64_t n) {
  if (env_int_or("NCNN_B200_FUSE_DW", 1) >= 2) return false;  // in one kernel wherever it applies
  const int blocks = (node.dw_c + 31) / 32;
  return !node.ex_fused && blocks > 6 && blocks < kTcChunkFrom && n * node.OH * node.OW <= 256 && tc_row_bytes(GEMM_BF16X3, node.dw_c) != 0;
}

// And where a whole block is three launches again: blocks with too many weights to stay are long chains of channel blocks.  The
// expanded tensor and the depthwise result then pass through the workspace.  Calls of stride-2 blocks in us, as three layers of
// the network / whole:
//   28x28x384 -> 64    images 1: 22.5 / 28.7    4: 28.6 / 28.7    8: 34.8 / 30.5   64: 73.7 / 47.1
//   28x28x768 -> 128          1: 28.7 / 43.0    8: 36.9 / 43.0   16: 47.1 / 47.1   64: 133 / 75.8
//   28x28x1024 -> 64          1: 30.7 / 51.2    8: 43.0 / 49.2   16: 55.3 / 51.2   64: 160 / 83.9
//   56x56x384 -> 128          1: 28.6 / 28.7    4: 34.8 / 32.7    8: 47.1 / 34.8   64: 264 / 139
// The crossover moves out with the channels, to ~2 400 result pixels.
static int64_t block_apart_images(const Node& node) {
  if (!node.ex_fused || env_int_or("NCNN_B200_FUSE_DW", 1) >= 2 || !tc_block_streams(node.ex_cin, node.dw_c, node.O, node.dw_stride) ||
      tc_row_bytes(GEMM_BF16X3, node.dw_c) == 0 || tc_row_bytes(GEMM_BF16X3, node.ex_cin) == 0)
    return 0;
  return std::max(0, std::min(4 * (node.dw_c - 192), 2400)) / (node.OH * node.OW);
}
// What they need for it: the depthwise result as two planes, then the expanded tensor.
static size_t block_apart_bytes(const Node& node, int64_t n) {
  return static_cast<size_t>(n) * (node.OH * node.OW + node.dw_hin * node.dw_win) * node.dw_c * 4 + 1024;
}
size_t EngineImpl::split_workspace_bytes() const {
  size_t bytes = kTcSplitWorkspaceBytes;
  for (const Node& node : nodes_)
    if (const int64_t n = block_apart_images(node)) bytes = std::max(bytes, (block_apart_bytes(node, n) + 255) / 256 * 256);
  return bytes;
}

// True when an InnerProduct / Gemm of this batch size runs on the kernel for a handful of rows (ip_rows.cuh): one pass
// over the weights on the CUDA cores instead of mostly empty 128-row tiles.
bool EngineImpl::takes_rows(const Node& node, int64_t n) const {
  if ((node.kind != N_IP && node.kind != N_GEMM) || node.impl != IMPL_TC || env_flag_off("NCNN_B200_IP_ROWS")) return false;
  const Tensor& ti = tensors_[resolve(node.in[0])];
  const Tensor& to = tensors_[resolve(node.out)];
  const bool i8 = node.term != 0;
  if (!i8 && ti.fmt != FMT_BF16X2) return false;
  const long long M = (to.rank == 2 ? static_cast<long long>(ti.h) : 1) * n;
  const int out_mode = to.fmt == FMT_I8 ? OUT_I8 : (to.fmt == FMT_BF16X2 ? OUT_BF16X2 : (to.fmt == FMT_F32 ? OUT_F32 : OUT_F32_SPLIT));
  return ip_rows_applies(M, ti.row_pitch > 0 ? ti.row_pitch : node.K, node.O, i8, out_mode, node.res >= 0, !node.side_q.empty());
}

// The Quantize step that the rows kernel of an int8 InnerProduct does itself while it loads its rows, or -1: a step of
// its own for this layer, reading one plain fp32 plane.
int EngineImpl::absorbed_quantize(const Node& node, int64_t n) const {
  if (node.kind != N_IP || node.term == 0 || !takes_rows(node, n)) return -1;
  for (size_t k = 0; k < nodes_.size(); ++k) {
    const Node& q = nodes_[k];
    if (q.kind != N_UNARY || q.un.op != UN_QUANT || resolve(q.out) != resolve(node.in[0])) continue;
    return q.side_q.empty() && q.un.nscale == 1 && tensors_[resolve(q.in[0])].fmt == FMT_F32 ? static_cast<int>(k) : -1;
  }
  return -1;
}

// A graph input whose storage is the caller's own layout is read where it is: plain fp32 in channel-last order that
// equals the caller's order (one channel, or one pixel), or rows for the kernel that converts them itself.
bool EngineImpl::reads_caller_array(int input, int64_t n, const void* ptr) const {
  const int id = resolve(inputs_[input]);
  const Tensor& t = tensors_[id];
  const bool flat = t.rank != 3 || ((t.c == 1 || t.h * t.w == 1) && t.Cp == t.c && t.Wp == t.w && t.w_off == 0);
  if (!flat || t.dedicated || t.input_quant_scale > 0.0f || !aligned16(ptr)) return false;
  if (t.fmt == FMT_F32) return true;
  if (t.fmt != FMT_BF16X2) return false;
  for (int o : outputs_)
    if (resolve(o) == id) return false;
  for (const Node& node : nodes_) {
    if (node.res >= 0 && resolve(node.res) == id) return false;
    for (int in : node.in)
      if (resolve(in) == id && !(takes_rows(node, n) && node.term == 0)) return false;
  }
  return true;
}

// True when the tensor is a graph output in [channel][pixel] order whose only toucher is a convolution on
// tc_gemm_kernel: its epilogue can write that order (one lane per pixel), which saves a pass over the result.
bool EngineImpl::chw_result(int id) const {
  const Tensor& t = tensors_[id];
  if (t.rank != 3 || t.c == 1 || t.h * t.w == 1 || t.fmt != FMT_F32 || t.is_input || t.Cp != t.c || t.Wp != t.w) return false;
  int entries = 0;
  for (int o : outputs_) entries += resolve(o) == id ? 1 : 0;
  if (entries != 1) return false;
  const Node* producer = nullptr;
  for (const Node& node : nodes_) {
    for (int in : node.in)
      if (resolve(in) == id) return false;
    if (node.res >= 0 && resolve(node.res) == id) return false;
    if (resolve(node.out) != id) continue;
    if (producer != nullptr) return false;
    producer = &node;
  }
  if (producer == nullptr) return false;
  const Node& p = *producer;
  if (p.kind != N_CONV || p.impl != IMPL_TC || p.stem || p.dw_fused || p.out_ld > 0 || !p.side_q.empty()) return false;
  // (residual rows are read in 16-byte pieces)
  if (p.res < 0) return true;
  const int res_fmt = tensors_[resolve(p.res)].fmt;
  return (res_fmt == FMT_F32 && p.O % 4 == 0) || (res_fmt == FMT_BF16X2 && p.O % 8 == 0);
}

// A graph output that a node writes as plain fp32 in the caller's order goes straight into the caller's array.
// (A tensor-core convolution whose result nobody else reads writes [channel][pixel] order itself: OUT_CHW.)
bool EngineImpl::writes_caller_array(int output, const void* ptr) const {
  const int id = resolve(outputs_[output]);
  const Tensor& t = tensors_[id];
  if (chw_result(id)) return true;
  const bool flat = t.rank != 3 || ((t.c == 1 || t.h * t.w == 1) && t.Cp == t.c && t.Wp == t.w && t.w_off == 0);
  if (!flat || t.is_input || t.fmt != FMT_F32 || t.row_pitch > 0 || !aligned16(ptr)) return false;
  for (const Node& node : nodes_)
    if (resolve(node.out) == id) return true;
  return false;
}

bool EngineImpl::emit_node(std::vector<Step>& steps, const Node& node, int64_t n, std::string* err) {
  const Tensor& to = tensors_[resolve(node.out)];
  const ActRef out = ref(node.out, n);
  Step s;
  s.name = node.name;
  s.flops = node.flops * n;
  const int f32_kind = opt_.accuracy_mode == kAccuracyTf32 ? GEMM_TF32 : GEMM_TF32X3;
  auto bytes_of = [&](int t) {
    const Tensor& x = tensors_[resolve(t)];
    return static_cast<double>(x.logical()) * (x.i8 ? 1 : 4) * n;
  };
  s.bytes = bytes_of(node.out);
  for (int t : node.in) s.bytes += bytes_of(t);
  if (node.res >= 0) s.bytes += bytes_of(node.res);

  if (node.kind == N_CONV || node.kind == N_IP || node.kind == N_GEMM || node.kind == N_DW) {
    const Tensor& ti = tensors_[resolve(node.in[0])];
    const ActRef in = ref(node.in[0], n);
    const bool i8 = node.term != 0;
    ConvEpilogue e{};
    e.bias = node.d_bias;
    e.scale = node.d_deq;
    e.out_scale = node.s_out;
    e.act = node.act;
    e.act_a = node.act_a;
    e.act_b = node.act_b;
    e.has_res = node.res >= 0;
    if (e.has_res) e.res = ref(node.res, n);
    if (node.kind == N_GEMM && i8) {
      const int K = node.K, N = node.O;
      const long long M = static_cast<long long>(ti.h) * n;
      const int8_t* wq = static_cast<const int8_t*>(node.d_w0);
      const float s_b = node.s_b, alpha = node.alpha, beta = 1.0f;
      const float* c_bias = node.d_bias;
      const int has_c = node.has_bias, scale_alpha = node.alpha != 1.0f;
      s.kernel = "k_gemm_i8_rowscale";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_gemm_i8_rowscale, static_cast<unsigned>(M), 128, K, st, in, out, wq, K, N, s_b, c_bias, alpha, beta, has_c, scale_alpha);
        return launch_ok();
      };
      steps.push_back(std::move(s));
      return true;
    }
    if (node.impl == IMPL_TC) {
      TcEpilogue te;
      te.bias = node.d_bias;
      te.scale = node.d_deq;
      te.out0 = out.p0;
      te.out1 = out.p1;
      te.outq = out.q;
      te.ldo = node.O;
      if (node.out_ld > 0) {
        // a view into a Concat result: longer rows, starting `out_ch_off` channels in
        te.ldo = node.out_ld;
        const size_t skip = static_cast<size_t>(node.out_ch_off) * to.elem_bytes();
        te.out0 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(out.p0) + skip);
        if (out.p1 != nullptr) te.out1 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(out.p1) + skip);
      }
      te.act = node.act;
      te.act_a = node.act_a;
      te.act_b = node.act_b;
      // Gemm: (A*B^T + beta*C) * alpha; beta is in the bias already, alpha multiplies in the epilogue
      const bool alpha_fused = node.kind == N_GEMM && node.alpha != 1.0f && node.act == ACT_NONE;
      if (alpha_fused) {
        te.act = ACT_SCALE;
        te.act_a = node.alpha;
      }
      te.out_scale = node.s_out;
      te.status = d_status_;
      te.side_count = static_cast<int>(node.side_q.size());
      for (int i = 0; i < te.side_count; ++i) {
        te.side_q[i] = ref(node.side_q[i].first, n).q;
        te.side_scale[i] = node.side_q[i].second;
      }
      te.sk_ws = d_split_ws_;
      te.sk_ws_bytes = kTcSplitWorkspaceBytes;
      te.sk_flags = d_split_flags_;
      te.sk_flag_count = kTcSplitFlagCount;
      const bool caller_chw = !caller_array_.empty() && caller_array_[resolve(node.out)] != nullptr && chw_result(resolve(node.out));
      te.out_mode = caller_chw ? OUT_CHW : to.fmt == FMT_I8 ? OUT_I8 : (to.fmt == FMT_SPLIT ? OUT_F32_SPLIT : (to.fmt == FMT_TF32 ? OUT_F32_TF32 : (to.fmt == FMT_BF16X2 ? OUT_BF16X2 : OUT_F32)));
      if (node.res >= 0) {
        const ActRef r = ref(node.res, n);
        te.res0 = r.p0;
        te.res1 = r.p1;
        te.res_bf16 = r.fmt == FMT_BF16X2;
      }
      const int kind = i8 ? GEMM_I8 : (ti.fmt == FMT_BF16X2 ? GEMM_BF16X3 : f32_kind);
      const char* kind_name = kind == GEMM_I8 ? "i8" : (kind == GEMM_TF32 ? "tf32" : (kind == GEMM_BF16X3 ? "bf16x3" : "tf32x3"));
      auto launch = std::make_shared<TcLaunch>();
      std::string perr;
      if (node.dw_fused && (depthwise_apart(node, n) || (n <= block_apart_images(node) && block_apart_bytes(node, n) <= split_ws_bytes_))) {
        // the depthwise result as bf16 pairs in the workspace of split contractions (a whole block's expanded tensor behind it),
        // which these layers therefore go without: their tiles stay whole, also where every other convolution is split
        // (NCNN_B200_STREAMK=1)
        te.sk_ws = nullptr;
        te.sk_flags = nullptr;
        auto view = [&](const ActRef& x, int channels, int h, int w) {
          TcIm2colView v;
          v.plane0 = x.p0;
          v.plane1 = x.p1;
          v.C = channels;
          v.W = v.OW = w;
          v.H = v.OH = h;
          v.N = n;
          v.stride_w = static_cast<uint64_t>(channels) * 2;
          v.stride_h = v.stride_w * w;
          v.stride_n = v.stride_h * h;
          return v;
        };
        const size_t plane = (static_cast<size_t>(n) * node.OH * node.OW * node.dw_c * 2 + 255) / 256 * 256;
        ActRef mid;
        mid.fmt = FMT_BF16X2;
        mid.p0 = reinterpret_cast<float*>(d_split_ws_);
        mid.p1 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(d_split_ws_) + plane);
        ActRef wide = in;  // the depthwise layer's input
        if (node.ex_fused) {
          wide = ActRef{};
          wide.fmt = FMT_F32;
          wide.p0 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(d_split_ws_) + 2 * plane);
          TcEpilogue xe;
          xe.bias = node.ex_bias;
          xe.act = node.ex_act;
          xe.act_a = node.ex_act_a;
          xe.act_b = node.ex_act_b;
          xe.out0 = wide.p0;
          xe.ldo = node.dw_c;
          xe.out_mode = OUT_F32;
          xe.status = d_status_;
          auto expand = std::make_shared<TcLaunch>();
          perr = tc_plan_conv(expand.get(), GEMM_BF16X3, view(in, node.ex_cin, node.dw_hin, node.dw_win), node.ex_w0, node.ex_w1, node.dw_c, xe, sm_count_);
          if (!perr.empty()) return fail(err, "layer " + node.ex_name + ": " + perr);
          Step x = s;
          x.name = node.ex_name;
          x.kernel = "tc_gemm_kernel<bf16x3>";
          x.flops = 2.0 * node.ex_cin * node.dw_c * node.dw_hin * node.dw_win * n;
          x.run = [expand](cudaStream_t st) { return tc_launch(*expand, st); };
          s.flops -= x.flops;
          steps.push_back(std::move(x));
        }
        ConvGeom g{};
        g.images = n;
        g.H = node.dw_hin;
        g.W = node.dw_win;
        g.OH = node.OH;
        g.OW = node.OW;
        g.C = g.O = node.dw_c;
        g.KH = g.KW = 3;
        g.sh = g.sw = node.dw_stride;
        g.dh = g.dw = 1;
        g.pt = node.dw_pt;
        g.pl = node.dw_pl;
        ConvEpilogue de{};
        de.bias = node.dw_bias;
        de.act = node.dw_act;
        de.act_a = node.dw_act_a;
        de.act_b = node.dw_act_b;
        const dim3 grid(((node.OH + 7) / 8) * ((node.OW + 7) / 8), (node.dw_c / 4 + 7) / 8, static_cast<unsigned>(n));
        const float* dw = node.dw_w;
        const int stride = node.dw_stride;
        Step d = s;
        d.name = node.dw_name;
        d.kernel = "k_depthwise3x3_tile";
        d.run = [=](cudaStream_t st) {
          if (stride == 1) launch_plain(k_depthwise3x3_tile<1>, grid, 256, 0, st, wide, mid, dw, g, de);
          else launch_plain(k_depthwise3x3_tile<2>, grid, 256, 0, st, wide, mid, dw, g, de);
          return launch_ok();
        };
        perr = tc_plan_conv(launch.get(), GEMM_BF16X3, view(mid, node.dw_c, node.OH, node.OW), node.d_w0, node.d_w1, node.O, te, sm_count_);
        if (!perr.empty()) return fail(err, "layer " + node.name + ": " + perr);
        d.flops = 18.0 * node.dw_c * node.OH * node.OW * n;
        s.flops -= d.flops;
        s.kernel = "tc_gemm_kernel<bf16x3>";
        s.run = [launch](cudaStream_t st) { return tc_launch(*launch, st); };
        steps.push_back(std::move(d));
        steps.push_back(std::move(s));
        return true;
      }
      if (node.dw_fused) {
        TcDwProjConv dc;
        dc.x = in.p0;
        dc.images = static_cast<int>(n);
        dc.H = node.OH;
        dc.W = node.OW;
        dc.Hin = node.dw_hin;
        dc.Win = node.dw_win;
        dc.C = node.dw_c;
        dc.stride = node.dw_stride;
        if (node.ex_fused) {
          dc.Cin = node.ex_cin;
          dc.x1 = in.p1;
          dc.ex_w0 = node.ex_w0;
          dc.ex_w1 = node.ex_w1;
          dc.ex_bias = node.ex_bias;
          dc.ex_act = node.ex_act;
          dc.ex_act_a = node.ex_act_a;
          dc.ex_act_b = node.ex_act_b;
        }
        dc.pad_t = node.dw_pt;
        dc.pad_l = node.dw_pl;
        dc.dw_weights = node.dw_w;
        dc.dw_bias = node.dw_bias;
        dc.dw_act = node.dw_act;
        dc.dw_act_a = node.dw_act_a;
        dc.dw_act_b = node.dw_act_b;
        dc.w0 = node.d_w0;
        dc.w1 = node.d_w1;
        dc.out_channels = node.O;
        auto dl = std::make_shared<TcDwProjLaunch>();
        const std::string derr = tc_plan_dw_project(dl.get(), dc, te, sm_count_);
        if (!derr.empty()) return fail(err, "layers " + node.dw_name + " + " + node.name + ": " + derr);
        s.name = (node.ex_fused ? node.ex_name + "+" : std::string()) + node.dw_name + "+" + node.name;
        s.kernel = node.ex_fused ? (node.dw_stride == 2 ? "tc_dw_project_kernel:expand+stride2<bf16x3>" : "tc_dw_project_kernel:expand<bf16x3>")
                                 : "tc_dw_project_kernel<bf16x3>";
        s.run = [dl](cudaStream_t st) { return tc_launch_dw_project(*dl, st); };
        steps.push_back(std::move(s));
        return true;
      }
      // stride-1 filters with spatial extent: the patch-resident kernel loads each input pixel
      // once per tile instead of once per tap
      const bool halo_pairs = halo_level() >= 2 || (halo_level() < 0 && halo_pays(kind, ti.c, node, n, sm_count_));
      if (node.kind == N_CONV && !i8 && !node.stem && node.out_ld == 0 && (halo_pairs || halo_level() >= 1) &&
          tc_halo_applies(kind, ti.c, node.KH, node.KW, node.sh, node.sw, node.dh, node.dw, node.OH, node.OW, node.O,
                          te.out_mode)) {
        TcHaloConv hc;
        hc.in0 = in.p0;
        hc.in1 = in.p1;
        hc.images = static_cast<int>(n);
        hc.H = ti.h;
        hc.W = ti.w;
        hc.C = ti.c;
        hc.KH = node.KH;
        hc.KW = node.KW;
        hc.pad_t = node.pt;
        hc.pad_l = node.pl;
        hc.OH = node.OH;
        hc.OW = node.OW;
        hc.w0 = node.d_w0;
        hc.w1 = node.d_w1;
        hc.out_channels = node.O;
        auto hl = std::make_shared<TcHaloLaunch>();
        if (tc_plan_conv_halo(hl.get(), kind, hc, te, sm_count_, halo_pairs).empty()) {
          s.kernel = std::string(hl->pair ? "tc_conv_halo_kernel:pairs<" : "tc_conv_halo_kernel<") + kind_name + ">";
          s.run = [hl](cudaStream_t st) { return tc_launch_halo(*hl, st); };
          steps.push_back(std::move(s));
          return true;
        }
      }
      if (node.kind == N_CONV && node.stem && node.stem_rows && node.res < 0 && node.out_ld == 0) {
        TcStemConv sc;
        sc.kind = kind;
        sc.in0 = i8 ? static_cast<const void*>(in.q) : static_cast<const void*>(in.p0);
        sc.in1 = in.p1;
        sc.images = static_cast<int>(n);
        sc.H = ti.h;
        sc.row_bytes = ti.Wp * ti.Cp * (i8 ? 1 : 2);
        sc.KH = node.KH;
        sc.stride_h = node.sh;
        sc.pad_t = node.pt;
        sc.OH = node.OH;
        sc.OW = node.OW;
        sc.w0 = node.d_w0;
        sc.w1 = node.d_w1;
        sc.out_channels = node.O;
        if (node.pool_fused) {
          auto pl = std::make_shared<TcStemPoolLaunch>();
          const std::string perr2 = tc_plan_stem_pool(pl.get(), sc, te, node.pool_oh, node.pool_ow, sm_count_);
          if (!perr2.empty()) return fail(err, "layers " + node.name + " + " + node.pool_name + ": " + perr2);
          s.name = node.name + "+" + node.pool_name;
          s.kernel = std::string("tc_stem_pool_kernel<") + kind_name + ">";
          s.run = [pl](cudaStream_t st) { return tc_launch_stem_pool(*pl, st); };
          steps.push_back(std::move(s));
          return true;
        }
        auto sl = std::make_shared<TcStemLaunch>();
        if (tc_plan_stem(sl.get(), sc, te, sm_count_).empty()) {
          s.kernel = std::string("tc_stem_kernel<") + kind_name + ">";
          s.run = [sl](cudaStream_t st) { return tc_launch_stem(*sl, st); };
          steps.push_back(std::move(s));
          return true;
        }
      }
      if (node.kind == N_CONV) {
        TcIm2colView v;
        v.plane0 = i8 ? static_cast<const void*>(in.q) : static_cast<const void*>(in.p0);
        v.plane1 = in.p1;
        const size_t es = static_cast<size_t>(tc_elem_bytes(kind));
        if (node.stem) {
          v.C = node.k_elems;
          v.W = node.OW;
          v.H = ti.h;
          v.N = n;
          v.stride_w = static_cast<uint64_t>(node.sw) * ti.Cp * es;
          v.stride_h = static_cast<uint64_t>(ti.Wp) * ti.Cp * es;
          v.stride_n = v.stride_h * ti.h;
          v.KH = node.KH;
          v.KW = 1;
          v.stride_conv_h = node.sh;
          v.stride_conv_w = 1;
          v.pad_t = node.pt;
          v.pad_l = 0;
          v.dil_h = node.dh;
          v.dil_w = 1;
        } else {
          v.C = ti.c;
          v.W = ti.w;
          v.H = ti.h;
          v.N = n;
          v.stride_w = static_cast<uint64_t>(ti.c) * es;
          v.stride_h = v.stride_w * ti.w;
          v.stride_n = v.stride_h * ti.h;
          v.KH = node.KH;
          v.KW = node.KW;
          v.stride_conv_h = node.sh;
          v.stride_conv_w = node.sw;
          v.pad_t = node.pt;
          v.pad_l = node.pl;
          v.dil_h = node.dh;
          v.dil_w = node.dw;
        }
        v.OH = node.OH;
        v.OW = node.OW;
        perr = tc_plan_conv_tiles(launch.get(), kind, v, node.O, te, sm_count_);
        const bool forced = launch->cta2 != 0 && (env_int_or("NCNN_B200_CTA2_ALWAYS", 0) != 0 || env_int_or("NCNN_B200_STREAMK", 0) == 1);
        // int8 filters of several taps that fit shared memory (unless a switch asks for pairs of CTAs or split tiles)
        if (perr.empty() && i8 && !node.stem && conv_i8_level() != 0 && !forced) {
          auto cl = std::make_shared<TcConvI8Launch>();
          if (tc_plan_conv_i8(cl.get(), v, node.d_w0, node.O, te, sm_count_, conv_i8_level() > 0).empty()) {
            s.kernel = "tc_conv_i8_kernel<i8>";
            s.run = [cl](cudaStream_t st) { return tc_launch_conv_i8(*cl, st); };
            steps.push_back(std::move(s));
            return true;
          }
        }
        // few pixels: small tiles out of input patches (unless a switch asks for pairs of CTAs or split tiles)
        if (perr.empty() && !node.stem && patch_level() != 0 && !forced) {
          auto pl = std::make_shared<TcPatchLaunch>();
          if (tc_plan_conv_patch(pl.get(), kind, v, node.d_w0, node.d_w1, node.O, te, sm_count_, *launch, patch_level() > 0).empty()) {
            s.kernel = std::string("tc_conv_patch_kernel<") + kind_name + ">";
            s.run = [pl](cudaStream_t st) { return tc_launch_patch(*pl, st); };
            steps.push_back(std::move(s));
            return true;
          }
        }
        if (perr.empty()) perr = tc_encode_conv(launch.get(), kind, v, node.d_w0, node.d_w1, node.O);
      } else {
        const long long M = (to.rank == 2 ? static_cast<long long>(ti.h) : 1) * n;
        const void* a0 = i8 ? static_cast<const void*>(in.q) : static_cast<const void*>(in.p0);
        // a handful of rows: one pass over the weights on the CUDA cores instead of mostly empty 128-row tiles
        const int row = ti.row_pitch > 0 ? ti.row_pitch : node.K;  // elements between rows of the operand
        if (takes_rows(node, n)) {
          IpRowsParams ip{};
          ip.M = static_cast<int>(M);
          ip.K = i8 ? row : node.K;  // (padded rows end in zeros on both sides)
          ip.N = node.O;
          ip.lda = row;
          const int q = absorbed_quantize(node, n);
          if (q >= 0 || in.fmt == FMT_F32) {
            // rows straight from the fp32 tensor (the caller's own array, or what a Quantize step would have read)
            const ActRef src = q >= 0 ? ref(nodes_[q].in[0], n) : in;
            ip.x = src.p0;
            ip.x_len = node.K;
            ip.x_scale = node.s_in;
          }
          ip.ldw = (node.K + node.k_elems - 1) / node.k_elems * node.k_elems;
          ip.a0 = a0;
          ip.a1 = in.p1;
          ip.w0 = node.d_w0;
          ip.w1 = node.d_w1;
          ip.bias = te.bias;
          ip.scale = te.scale;
          ip.out_scale = te.out_scale;
          ip.act = te.act;
          ip.act_a = te.act_a;
          ip.act_b = te.act_b;
          ip.out_mode = te.out_mode;
          ip.out0 = te.out0;
          ip.out1 = te.out1;
          ip.outq = te.outq;
          ip.ldo = te.ldo;
          ip.x_vec = ip.x != nullptr && node.K % 4 == 0 && aligned16(ip.x) ? 1 : 0;
          const int smem = static_cast<int>(ip_rows_smem_bytes(ip.M, ip.K, i8));
          const cudaError_t ae = i8 ? cudaFuncSetAttribute(k_ip_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024)
                                    : cudaFuncSetAttribute(k_ip_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
          if (ae != cudaSuccess) return fail(err, "layer " + node.name + ": " + cudaGetErrorString(ae));
          const int tasks = (ip.N + kIpRowsCols - 1) / kIpRowsCols;
          const int grid = std::max(1, std::min(sm_count_, tasks));
          s.kernel = i8 ? "k_ip_rows<i8>" : "k_ip_rows<bf16x2>";
          s.direct = true;
          s.run = [=](cudaStream_t st) {
            if (i8) launch_plain(k_ip_rows<true>, grid, kIpRowsThreads, smem, st, ip);
            else launch_plain(k_ip_rows<false>, grid, kIpRowsThreads, smem, st, ip);
            return launch_ok();
          };
          steps.push_back(std::move(s));
          return true;
        }
        perr = tc_plan_gemm(launch.get(), kind, a0, in.p1, M, node.K, row, node.d_w0, node.d_w1, node.O, te, sm_count_);
      }
      if (!perr.empty()) return fail(err, "layer " + node.name + ": " + perr);
      s.kernel = std::string(launch->cta2 == 2 ? (launch->p.streamk ? "tc_gemm2_kernel:pairs+split<" : "tc_gemm2_kernel:pairs<") : (launch->cta2 == 1 ? "tc_gemm2_kernel:split<" : "tc_gemm_kernel<")) + kind_name + ">";
      s.run = [launch](cudaStream_t st) { return tc_launch(*launch, st); };
      steps.push_back(std::move(s));
    } else if (node.kind == N_CONV || node.kind == N_DW) {
      ConvGeom g{};
      g.images = n;
      g.H = ti.h;
      g.W = ti.w;
      g.C = ti.c;
      g.OH = node.OH;
      g.OW = node.OW;
      g.O = node.O;
      g.KH = node.KH;
      g.KW = node.KW;
      g.sh = node.sh;
      g.sw = node.sw;
      g.pt = node.pt;
      g.pl = node.pl;
      g.dh = node.dh;
      g.dw = node.dw;
      const void* w = node.d_w0;
      if (node.kind == N_DW && !i8 && ti.c % 4 == 0 && node.KH == 3 && node.KW == 3 && node.dh == 1 &&
          node.dw == 1 && node.sh == node.sw && (node.sh == 1 || node.sh == 2) && n <= 65535) {
        const dim3 grid(((node.OH + 7) / 8) * ((node.OW + 7) / 8), (ti.c / 4 + 7) / 8, static_cast<unsigned>(n));
        const int stride = node.sh;
        const float* wf = static_cast<const float*>(w);
        const int pairs = (node.OW + 1) / 2;
        const long long threads = n * pairs * (ti.c / 4);
        // A thread of the columns kernel walks OH rows one after the other, so it needs enough threads, and more the longer the
        // walk.  At stride 2, whose rows come from memory twice as fast, it is only a little faster than the tile kernel when
        // the last of its waves of 2 blocks an SM is full, and slower when that is not.  Whole calls of expand layer,
        // depthwise layer and projection, tile / columns in us (the launch alone, its input in L2, flatters columns):
        //   stride 1: 14x14x384 8 700 threads 24.6 / 30.7, 16 800 30.7 / 30.7, 24 200 36.8 / 32.8; 32x32x384 16 900 41.0 / 45.1,
        //             24 600 49.2 / 47.1; 56x56x384 24 200 73.7 / 73.8, 37 600 109 / 98, 250 000 604 / 471
        //   stride 2: 28 -> 14x14x384 16 800 43.0 / 45.1, 24 200 51.2 / 49.2; 34 -> 17x17x384 51 000 102 / 90; 40 -> 20x20x384
        //             38 400 90.1 / 96.3, 49 900 117 / 115; 56 -> 28x28x384 24 200 79.9 / 102, 75 300 (a wave)
        //             215 / 197, 90 000 252 / 266; 64 -> 32x32x384 16 900 65.6 / 94.2, 75 300 232 / 221, 119 800 352 / 358;
        //             112 -> 56x56x96 49 700 361 / 389, 75 300 533 / 528
        const long long wave = 2ll * sm_count_ * 256, waves = (threads + wave - 1) / wave;
        const bool enough = node.sh == 1       ? threads >= 16384 + 250 * std::max(0, node.OH - 14)
                            : node.OH <= 16 ? threads >= 16384 + 1024 * std::max(0, node.OH - 8)
                                            : threads * 100 >= waves * wave * (node.OH <= 20 ? 62 : node.OH <= 28 ? 72 : 88);
        const int clamp = node.act == ACT_RELU || node.act == ACT_CLIP ? 1 : 0;
        const bool columns = in.fmt == FMT_F32 && (out.fmt == FMT_F32 || out.fmt == FMT_BF16X2) && (clamp || node.act == ACT_NONE) && !e.has_res &&
                             enough && n * pairs <= 0x7fffffffll && (threads + 255) / 256 <= 0x7fffffffll;
        const float lo = node.act == ACT_CLIP ? e.act_a : 0.0f, hi = node.act == ACT_CLIP ? e.act_b : INFINITY;
        const unsigned blocks = static_cast<unsigned>((threads + 255) / 256);
        s.kernel = columns ? "k_depthwise3x3_columns" : "k_depthwise3x3_tile";
        s.run = [=](cudaStream_t st) {
          if (columns && stride == 1) launch_plain(k_depthwise3x3_columns<1>, blocks, 256, 0, st, in.p0, out, wf, e.bias, g, clamp, lo, hi, pairs, threads);
          else if (columns) launch_plain(k_depthwise3x3_columns<2>, blocks, 256, 0, st, in.p0, out, wf, e.bias, g, clamp, lo, hi, pairs, threads);
          else if (stride == 1) launch_plain(k_depthwise3x3_tile<1>, grid, 256, 0, st, in, out, wf, g, e);
          else launch_plain(k_depthwise3x3_tile<2>, grid, 256, 0, st, in, out, wf, g, e);
          return launch_ok();
        };
      } else if (node.kind == N_DW) {
        const bool vec = ti.c % 4 == 0;
        const long long work = n * node.OH * node.OW * (vec ? ti.c / 4 : ti.c);
        const int grid = grid_for(work);
        s.kernel = i8 ? "k_depthwise<i8>" : "k_depthwise<f32>";
        s.run = [=](cudaStream_t st) {
          if (i8) {
            if (vec) launch_plain(k_depthwise<4, true>, grid, 256, 0, st, in, out, w, g, e);
            else launch_plain(k_depthwise<1, true>, grid, 256, 0, st, in, out, w, g, e);
          } else {
            if (vec) launch_plain(k_depthwise<4, false>, grid, 256, 0, st, in, out, w, g, e);
            else launch_plain(k_depthwise<1, false>, grid, 256, 0, st, in, out, w, g, e);
          }
          return launch_ok();
        };
      } else if (!i8 && conv_f32_applies(in, g)) {
        const std::string ferr = emit_conv_f32(&s, in, out, w, g, e);
        if (!ferr.empty()) return fail(err, "layer " + node.name + ": " + ferr);
      } else {
        const int grid = grid_for(n * node.OH * node.OW * node.O);
        s.kernel = i8 ? "k_conv_direct<i8>" : "k_conv_direct<f32>";
        s.run = [=](cudaStream_t st) {
          if (i8) launch_plain(k_conv_direct<true>, grid, 256, 0, st, in, out, w, g, e);
          else launch_plain(k_conv_direct<false>, grid, 256, 0, st, in, out, w, g, e);
          return launch_ok();
        };
      }
      steps.push_back(std::move(s));
    } else {
      const long long M = (to.rank == 2 ? static_cast<long long>(ti.h) : 1) * n;
      const int K = node.K, N = node.O;
      const void* w = node.d_w0;
      ConvGeom g{};
      g.images = M;
      g.C = K;
      g.O = N;
      g.H = g.W = g.OH = g.OW = g.KH = g.KW = g.sh = g.sw = g.dh = g.dw = 1;
      if (!i8 && conv_f32_applies(in, g)) {
        const std::string ferr = emit_conv_f32(&s, in, out, w, g, e);
        if (!ferr.empty()) return fail(err, "layer " + node.name + ": " + ferr);
      } else {
      const int grid = grid_for(M * N);
      s.kernel = i8 ? "k_matmul_direct<i8>" : "k_matmul_direct<f32>";
      s.run = [=](cudaStream_t st) {
        if (i8) launch_plain(k_matmul_direct<true>, grid, 256, 0, st, in, out, w, M, K, N, e, 0.0f);
        else launch_plain(k_matmul_direct<false>, grid, 256, 0, st, in, out, w, M, K, N, e, 0.0f);
        return launch_ok();
      };
      }
      steps.push_back(std::move(s));
    }
    if (node.kind == N_GEMM && node.alpha != 1.0f && !(node.impl == IMPL_TC && node.act == ACT_NONE)) {
      Step m;
      m.name = node.name + ":alpha";
      m.kernel = "k_binary";
      BinaryParams bp{};
      bp.op = BIN_MUL;
      bp.use_scalar = 1;
      bp.scalar = node.alpha;
      const long long count = to.logical() * n;
      const int grid = grid_for(count);
      m.run = [=](cudaStream_t st) {
        launch_plain(k_binary<1>, grid, 256, 0, st, out, out, out, count, bp);
        return launch_ok();
      };
      steps.push_back(std::move(m));
    }
    return true;
  }
  if (node.kind == N_POOL) {
    const ActRef in = ref(node.in[0], n);
    PoolParams p = node.pool;
    p.images = n;
    p.side_q = node.side_q.empty() ? nullptr : ref(node.side_q[0].first, n).q;
    p.side_scale = node.side_q.empty() ? 0.0f : node.side_q[0].second;
    const bool vec = p.C % 4 == 0;
    if (p.kind == 0 && p.KH == 3 && p.KW == 3 && p.sh == 2 && p.sw == 2 && vec && !tensors_[resolve(node.in[0])].i8 &&
        n <= 65535 && p.OH * p.OW >= 64) {
      const dim3 grid(((p.OH + 7) / 8) * ((p.OW + 7) / 8), (p.C / 4 + 7) / 8, static_cast<unsigned>(n));
      s.kernel = "k_maxpool3x3s2_tile";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_maxpool3x3s2_tile, grid, 256, 0, st, in, out, p);
        return launch_ok();
      };
      steps.push_back(std::move(s));
      return true;
    }
    // one window over the whole image (global pooling, or a window at least as large as an unpadded image)
    const bool whole = !p.adaptive && p.OH == 1 && p.OW == 1 && p.pt == 0 && p.pl == 0 && p.KH >= p.H && p.KW >= p.W;
    if (whole && vec && n <= 65535) {
      const dim3 grid((p.C / 4 + 127) / 128, static_cast<unsigned>(n));
      s.kernel = "k_global_pool4";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_global_pool4, grid, 128, 0, st, in, out, p);
        return launch_ok();
      };
      steps.push_back(std::move(s));
      return true;
    }
    const int grid = grid_for(n * p.OH * p.OW * (vec ? p.C / 4 : p.C));
    s.kernel = "k_pool";
    s.run = [=](cudaStream_t st) {
      if (vec) launch_plain(k_pool<4>, grid, 256, 0, st, in, out, p);
      else launch_plain(k_pool<1>, grid, 256, 0, st, in, out, p);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_DECONV) {
    const Tensor& ti = tensors_[resolve(node.in[0])];
    const ActRef in = ref(node.in[0], n);
    DeconvParams dp{n, ti.h, ti.w, ti.c, node.O, node.act == ACT_RELU ? 1 : 0};
    const float* w = static_cast<const float*>(node.d_w0);
    const float* bias = node.d_bias;
    const int grid = grid_for(to.logical() * n);
    s.kernel = "k_deconv2x2";
    s.run = [=](cudaStream_t st) {
      launch_plain(k_deconv2x2, grid, 256, 0, st, in, out, w, bias, dp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_REDUCE) {
    const ActRef in = ref(node.in[0], n);
    ReduceParams rp = node.reduce;
    rp.images = n;
    const int grid = grid_for(to.logical() * n);
    s.kernel = "k_reduce_mean";
    s.run = [=](cudaStream_t st) {
      launch_plain(k_reduce_mean, grid, 256, 0, st, in, out, rp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_REMAP) {
    const ActRef in = ref(node.in[0], n);
    RemapParams rp = node.remap;
    rp.images = n;
    const int grid = grid_for(to.logical() * n);
    s.kernel = "k_remap";
    s.run = [=](cudaStream_t st) {
      launch_plain(k_remap, grid, 256, 0, st, in, out, rp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_BINARY && node.broadcast) {
    const ActRef a = ref(node.in[0], n);
    const ActRef b = ref(node.in[1], n);
    BroadcastParams bp = node.bcast;
    bp.images = n;
    bp.op = node.bin;
    const int grid = grid_for(bp.o_image * n);
    s.kernel = "k_binary_broadcast";
    s.run = [=](cudaStream_t st) {
      launch_plain(k_binary_broadcast, grid, 256, 0, st, a, b, out, bp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_BINARY) {
    const ActRef a = ref(node.in[0], n);
    const ActRef b = node.in.size() > 1 ? ref(node.in[1], n) : a;
    const BinaryParams bp = node.bin;
    const long long count = to.logical() * n;
    const bool vec = count % 4 == 0;
    const int grid = grid_for(vec ? count / 4 : count);
    s.kernel = "k_binary";
    s.run = [=](cudaStream_t st) {
      if (vec) launch_plain(k_binary<4>, grid, 256, 0, st, a, b, out, count, bp);
      else launch_plain(k_binary<1>, grid, 256, 0, st, a, b, out, count, bp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_UNARY) {
    if (node.un.op == UN_QUANT)
      for (const Node& ip : nodes_)
        if (ip.kind == N_IP && resolve(ip.in[0]) == resolve(node.out) && absorbed_quantize(ip, n) >= 0) return true;  // the rows kernel quantises
    const ActRef in = ref(node.in[0], n);
    if (to.row_pitch > 0) {
      const Tensor& ts = tensors_[resolve(node.in[0])];
      const int K = static_cast<int>(ts.rank == 2 ? ts.w : ts.logical());
      const long long rows = n * (ts.rank == 2 ? ts.h : 1);
      const int pitch = to.row_pitch;
      const float scale = node.un_scale[0];
      const int grid = grid_for(rows * (pitch / 4));
      s.kernel = "k_quantize_rows";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_quantize_rows, grid, 256, 0, st, in, out.q, rows, K, pitch, scale);
        return launch_ok();
      };
      steps.push_back(std::move(s));
      return true;
    }
    const UnaryParams up = node.un;
    const long long count = to.logical() * n;
    const bool vec = count % 4 == 0;
    if (up.op == UN_QUANT && up.nscale == 1 && in.fmt == FMT_F32 && out.fmt == FMT_I8 && count % 16 == 0 &&
        !node.un_scale.empty()) {
      const float scale = node.un_scale[0];
      const int grid16 = grid_for(count / 16);
      const float* xp = in.p0;
      int8_t* yp = out.q;
      int8_t* y2 = node.side_q.empty() ? nullptr : ref(node.side_q[0].first, n).q;
      const float scale2 = node.side_q.empty() ? 0.0f : node.side_q[0].second;
      s.kernel = node.side_q.empty() ? "k_quantize16" : "k_quantize16:two results";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_quantize16, grid16, 256, 0, st, xp, yp, count / 16, scale, y2, scale2);
        return launch_ok();
      };
      steps.push_back(std::move(s));
      return true;
    }
    const int grid = grid_for(vec ? count / 4 : count);
    s.kernel = "k_unary";
    s.run = [=](cudaStream_t st) {
      if (vec) launch_plain(k_unary<4>, grid, 256, 0, st, in, out, count, up);
      else launch_plain(k_unary<1>, grid, 256, 0, st, in, out, count, up);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_SOFTMAX) {
    const ActRef in = ref(node.in[0], n);
    SoftmaxParams sp = node.softmax;
    sp.images = n;
    const int grid = grid_for(n * sp.lines * 32);
    s.kernel = "k_softmax";
    s.run = [=](cudaStream_t st) {
      launch_plain(k_softmax, grid, 256, 0, st, in, out, sp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  if (node.kind == N_CONCAT) {
    for (size_t k = 0; k < node.in.size(); ++k) {
      Step c = s;
      c.name = node.name + ":" + std::to_string(k);
      c.flops = 0;
      c.bytes = 2.0 * bytes_of(node.in[k]);
      const ActRef in = ref(node.in[k], n);
      ConcatParams cp = node.concat[k];
      cp.images = n;
      const int grid = grid_for(n * cp.in_image_elems);
      c.kernel = "k_concat_copy";
      c.run = [=](cudaStream_t st) {
        launch_plain(k_concat_copy, grid, 256, 0, st, in, out, cp);
        return launch_ok();
      };
      steps.push_back(std::move(c));
    }
    return true;
  }
  if (node.kind == N_RELAYOUT) {
    const ActRef in = ref(node.in[0], n);
    RelayoutParams rp = node.relayout;
    rp.images = n;
    const int grid = grid_for(rp.count * n);
    s.kernel = "k_relayout";
    s.run = [=](cudaStream_t st) {
      launch_plain(k_relayout, grid, 256, 0, st, in, out, rp);
      return launch_ok();
    };
    steps.push_back(std::move(s));
    return true;
  }
  return fail(err, "internal: unknown node kind");
}

void EngineImpl::make_edge_steps(int64_t n, const std::vector<const float*>& d_in,
                                 const std::vector<float*>& d_out, std::vector<Step>* pre,
                                 std::vector<Step>* post) {
  for (size_t i = 0; i < inputs_.size(); ++i) {
    const Tensor& t = tensors_[resolve(inputs_[i])];
    if (!caller_array_.empty() && caller_array_[resolve(inputs_[i])] != nullptr) continue;
    const ActRef dst = ref(inputs_[i], n);
    const float* src_ptr = d_in[i];
    Step s;
    s.name = "input:" + t.name;
    s.bytes = static_cast<double>(t.logical()) * n * (4 + t.elem_bytes() * t.planes());
    // one channel, or one pixel: channel-last order is the caller's order, a flat copy does it
    const bool flat_layout = (t.c == 1 || t.h * t.w == 1) && t.Cp == t.c && t.Wp == t.w && t.w_off == 0;
    const bool flat_quant = t.rank == 3 && flat_layout && t.input_quant_scale > 0.0f && dst.fmt == FMT_I8 &&
                            (t.logical() * n) % 16 == 0 && (reinterpret_cast<uintptr_t>(src_ptr) & 15) == 0 &&
                            (reinterpret_cast<uintptr_t>(dst.q) & 15) == 0;
    const bool flat_in = t.rank != 3 || (flat_layout && t.input_quant_scale <= 0.0f);
    if (flat_quant) {
      const long long count16 = t.logical() * n / 16;
      const int grid = grid_for(count16);
      const float scale = t.input_quant_scale;
      int8_t* q = dst.q;
      s.kernel = "k_quantize16";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_quantize16, grid, 256, 0, st, src_ptr, q, count16, scale, nullptr, 0.0f);
        return launch_ok();
      };
    } else if (!flat_in) {
      EdgeParams ep{};
      ep.images = n;
      ep.C = t.c;
      ep.H = t.h;
      ep.W = t.w;
      ep.Cp = t.Cp;
      ep.Wp = t.Wp;
      ep.w_off = t.w_off;
      ep.quant_scale = t.input_quant_scale;
      if (t.c <= 4 && ((t.Cp == 4 && t.fmt != FMT_I8) || (t.Cp == 8 && t.fmt == FMT_I8)) && t.w % 4 == 0 &&
          n <= 65535 &&
          (reinterpret_cast<uintptr_t>(src_ptr) & 15) == 0) {
        const dim3 grid(static_cast<unsigned>(std::min(148 * 8, (t.h * t.w / 4 + 255) / 256)), static_cast<unsigned>(n));
        s.kernel = "k_chw_to_nhwc_small_x4";
        s.run = [=](cudaStream_t st) {
          launch_plain(k_chw_to_nhwc_small_x4, grid, 256, 0, st, src_ptr, dst, ep);
          return launch_ok();
        };
      } else if (t.c <= 4 && (t.Cp == 4 || t.Cp == 16 || (t.Cp == 8 && t.fmt == FMT_I8) || (t.Cp == t.c && t.input_quant_scale <= 0.0f))) {
        const int grid = grid_for(n * t.h * t.w);
        s.kernel = "k_chw_to_nhwc_small";
        s.run = [=](cudaStream_t st) {
          launch_plain(k_chw_to_nhwc_small, grid, 256, 0, st, src_ptr, dst, ep);
          return launch_ok();
        };
      } else {
        const dim3 grid((t.h * t.w + 31) / 32, (t.c + 31) / 32, static_cast<unsigned>(n));
        s.kernel = "k_chw_to_nhwc_tiled";
        s.run = [=](cudaStream_t st) {
          launch_plain(k_chw_to_nhwc_tiled, grid, dim3(32, 8), 0, st, src_ptr, dst, ep);
          return launch_ok();
        };
      }
    } else {
      ActRef src;
      src.fmt = FMT_F32;
      src.p0 = const_cast<float*>(src_ptr);
      UnaryParams up{};
      up.op = UN_COPY;
      const long long count = t.logical() * n;
      const bool vec = count % 4 == 0 && (reinterpret_cast<uintptr_t>(src_ptr) & 15) == 0;
      const int grid = grid_for(vec ? count / 4 : count);
      s.kernel = "k_unary";
      s.run = [=](cudaStream_t st) {
        if (vec) launch_plain(k_unary<4>, grid, 256, 0, st, src, dst, count, up);
        else launch_plain(k_unary<1>, grid, 256, 0, st, src, dst, count, up);
        return launch_ok();
      };
    }
    pre->push_back(std::move(s));
  }
  for (size_t i = 0; i < outputs_.size(); ++i) {
    const Tensor& t = tensors_[resolve(outputs_[i])];
    const ActRef src = ref(outputs_[i], n);
    float* dst_ptr = d_out[i];
    if (!caller_array_.empty() && caller_array_[resolve(outputs_[i])] == dst_ptr) continue;
    Step s;
    s.name = "output:" + t.name;
    s.bytes = static_cast<double>(t.logical()) * n * (4 + t.elem_bytes() * t.planes());
    const bool flat_out = t.rank != 3 || ((t.c == 1 || t.h * t.w == 1) && t.Cp == t.c && t.Wp == t.w && t.w_off == 0);
    if (!flat_out) {
      const dim3 grid((t.h * t.w + 31) / 32, (t.c + 31) / 32, static_cast<unsigned>(n));
      const int C = t.c, HW = t.h * t.w, Cp = t.Cp;
      s.kernel = "k_nhwc_to_chw_tiled";
      s.run = [=](cudaStream_t st) {
        launch_plain(k_nhwc_to_chw_tiled, grid, dim3(32, 8), 0, st, src, dst_ptr, n, C, HW, Cp);
        return launch_ok();
      };
    } else {
      ActRef dst;
      dst.fmt = FMT_F32;
      dst.p0 = dst_ptr;
      UnaryParams up{};
      up.op = UN_COPY;
      const long long count = t.logical() * n;
      const bool vec = count % 4 == 0 && (reinterpret_cast<uintptr_t>(dst_ptr) & 15) == 0;
      const int grid = grid_for(vec ? count / 4 : count);
      s.kernel = "k_unary";
      s.run = [=](cudaStream_t st) {
        if (vec) launch_plain(k_unary<4>, grid, 256, 0, st, src, dst, count, up);
        else launch_plain(k_unary<1>, grid, 256, 0, st, src, dst, count, up);
        return launch_ok();
      };
    }
    post->push_back(std::move(s));
  }
}

}  // namespace nb
