// Bindings of the MoE kernels (routing, split scan, dispatch, grouped GEMM, combine).
#include <cuda.h>
#include <cuda_runtime.h>

#include "../kernels/token_walker.h"
#include "py_types.h"

namespace py = pybind11;
using namespace fastb;
using namespace fastb_py;

namespace {

void cu_check(cudaError_t e, const char* what) { cuda_check(e, what); }
cudaStream_t stream_now() { return cur_stream(); }

template <class T> T* ptr_or_null(const c10::optional<torch::Tensor>& t) { return t.has_value() ? reinterpret_cast<T*>(t->data_ptr()) : nullptr; }
void want(const torch::Tensor& t, c10::ScalarType dt, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.is_contiguous() && t.scalar_type() == dt, name, ": expected a contiguous CUDA tensor of the right dtype");
}
// ... that a kernel reads or writes in words of `word` bytes: a view may start at any element, and a misaligned access costs the context.
void want_aligned(const torch::Tensor& t, c10::ScalarType dt, const char* name, int word) {
  want(t, dt, name);
  TORCH_CHECK(reinterpret_cast<uintptr_t>(t.data_ptr()) % word == 0, name, ": must start at a multiple of ", word, " bytes (clone a view that does not)");
}
void want16(const torch::Tensor& t, c10::ScalarType dt, const char* name) { want_aligned(t, dt, name, 16); }

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cu_check(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q), "cudaGetDriverEntryPoint");
    TORCH_CHECK(p != nullptr && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled is not available in this driver");
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// A 2-D bf16 row-major matrix [rows, cols] (row pitch in elements) tiled in boxes of
// {box_cols, box_rows} with the 128-byte swizzle. box_cols must be 64 (one 128-byte line).
struct TensorMap2D {
  alignas(64) CUtensorMap map;
  TensorMap2D() = default;
  // A 2-D byte matrix (e4m3 rows) tiled in boxes of {64 bytes, box_rows}, no swizzle: the ring the converter
  // warps of the e4m3-operand GEMM read from.
  static TensorMap2D bytes(int64_t ptr, int64_t rows, int64_t cols, int64_t pitch_bytes, int box_rows) {
    TORCH_CHECK(box_rows >= 1 && box_rows <= 256 && ptr % 16 == 0 && pitch_bytes % 16 == 0 && cols % 64 == 0, "byte tensor map: 16-byte aligned base and pitch, columns a multiple of 64");
    TensorMap2D t;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch_bytes)};
    cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_tiled()(&t.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, reinterpret_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (bytes) failed with code ", static_cast<int>(r));
    return t;
  }
  TensorMap2D(int64_t ptr, int64_t rows, int64_t cols, int64_t pitch_elems, int box_cols, int box_rows) {
    TORCH_CHECK(box_cols == 64, "128-byte swizzle wants boxes of 64 bf16 in the contiguous dimension");
    TORCH_CHECK(box_rows >= 1 && box_rows <= 256, "box rows out of range");
    TORCH_CHECK(ptr % 16 == 0 && (pitch_elems * 2) % 16 == 0, "tensor map base and pitch must be 16-byte aligned");
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch_elems) * 2};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_tiled()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, reinterpret_cast<void*>(ptr), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code ", static_cast<int>(r));
  }
};

CUtensorMap bf16_map(int rank, int64_t ptr, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  TORCH_CHECK(ptr % 16 == 0, "tensor map base must be 16-byte aligned");
  for (int i = 0; i + 1 < rank; ++i) TORCH_CHECK(strides[i] % 16 == 0, "tensor map strides must be multiples of 16 bytes");
  alignas(64) CUtensorMap m;
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, reinterpret_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code ", static_cast<int>(r));
  return m;
}
CUtensorMap bf16_map_2d(const torch::Tensor& t, int box_rows) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 2 && t.stride(1) == 1, "expected a CUDA bf16 matrix with contiguous rows");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(t.size(1)), static_cast<cuuint64_t>(t.size(0))}, strides[1] = {static_cast<cuuint64_t>(t.stride(0)) * 2};
  const cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
  return bf16_map(2, reinterpret_cast<int64_t>(t.data_ptr()), dims, strides, box);
}

// One contraction on fixed buffers (weights, tokens, outputs): everything about the launch of grouped_gemm_tokens that does not
// change from call to call, the tensor maps above all.
struct TokGemmPlan {
  alignas(64) CUtensorMap w, c, c2;
  TokMapsX x;
  GemmMode mode;
  GemmEpilogue epi;
  bool has_c2;
  int device;
  int64_t groups;
  int band_rows_;
  TokGemmArgs a{};
  // What the plan was made from.
  struct View {
    const void* ptr = nullptr;
    c10::ScalarType type = c10::ScalarType::Undefined;
    int64_t device = -1;
    c10::SmallVector<int64_t, 3> sizes, strides;
    View() = default;
    explicit View(const torch::Tensor& t) : ptr(t.data_ptr()), type(t.scalar_type()), device(t.get_device()), sizes(t.sizes().begin(), t.sizes().end()), strides(t.strides().begin(), t.strides().end()) {}
    bool is(const torch::Tensor& t) const {
      return t.data_ptr() == ptr && t.scalar_type() == type && t.get_device() == device && t.sizes() == at::IntArrayRef(sizes) && t.strides() == at::IntArrayRef(strides);
    }
  };
  View of_w, of_x, of_out, of_gu;
  bool matches(const torch::Tensor& weights, const torch::Tensor& tokens, const torch::Tensor& out, const c10::optional<torch::Tensor>& gate_up, int granule, int band_rows) const {
    return granule == a.granule && band_rows == band_rows_ && of_w.is(weights) && of_x.is(tokens) && of_out.is(out) && gate_up.has_value() == has_c2 && (!has_c2 || of_gu.is(*gate_up));
  }

  // weights [G, N, K]; forward: tokens [R, K] -> out [R, N] (SwiGLU [R, N / 2]); dgrad: tokens [R, N] -> out [R, K] (SwiGLU backward [R, 2 K]).
  TokGemmPlan(int mode_, int epi_, torch::Tensor weights, torch::Tensor tokens, torch::Tensor out, c10::optional<torch::Tensor> gate_up, int granule, int band_rows)
      : mode(static_cast<GemmMode>(mode_)), epi(static_cast<GemmEpilogue>(epi_)), has_c2(gate_up.has_value()), band_rows_(band_rows) {
    TORCH_CHECK(weights.is_cuda() && weights.scalar_type() == torch::kBFloat16 && weights.dim() == 3 && weights.is_contiguous(), "weights: contiguous CUDA bf16 [G, N, K]");
    const int64_t G = weights.size(0), N = weights.size(1), K = weights.size(2);
    const bool fwd = mode == GemmMode::kForward;
    const int64_t feats = fwd ? N : K, red = fwd ? K : N, cols = epi == GemmEpilogue::kSwiGLU ? N / 2 : epi == GemmEpilogue::kSwiGLUBwd ? 2 * K : feats;
    TORCH_CHECK(mode != GemmMode::kWgrad && feats % 256 == 0 && red % 64 == 0, "grouped_gemm_tokens: features must be a multiple of 256, the reduction of 64");
    TORCH_CHECK(tokens.dim() == 2 && tokens.size(1) == red && out.dim() == 2 && out.size(1) == cols && out.size(0) == tokens.size(0), "grouped_gemm_tokens: shapes");
    TORCH_CHECK(!has_c2 || (gate_up->size(0) == tokens.size(0) && gate_up->size(1) == (fwd ? N : 2 * K)), "grouped_gemm_tokens: gate|up shape");
    device = weights.get_device();
    groups = G;
    of_w = View(weights); of_x = View(tokens); of_out = View(out);
    if (has_c2) of_gu = View(*gate_up);
    const int64_t wp = reinterpret_cast<int64_t>(weights.data_ptr());
    if (fwd && epi == GemmEpilogue::kSwiGLU) {
      // [G * N / 256 tiles][8 groups of 16 features][gate, up][16][K], fetched as four groups with both halves
      const cuuint64_t k = static_cast<cuuint64_t>(K), dims[5] = {k, 16, 2, 8, static_cast<cuuint64_t>(G * N / 256)}, strides[4] = {2 * k, 256 * k, 32 * k, 512 * k};
      const cuuint32_t box[5] = {64, 16, 2, 4, 1};
      w = bf16_map(5, wp, dims, strides, box);
    } else {
      w = bf16_map_2d(weights.view({G * N, K}), fwd ? 128 : 64);
    }
    for (int j = 0; j < kTokBoxes; ++j) x.box[j] = bf16_map_2d(tokens, 16 << j);
    c = bf16_map_2d(out, 32);
    if (has_c2) c2 = bf16_map_2d(*gate_up, 32);
    a.num_groups = static_cast<int>(G);
    a.m_tiles = static_cast<int>(feats / 256); a.red_blocks = static_cast<int>(red / 64); a.w_rows_per_group = static_cast<int>(N);
    a.granule = granule; a.keep_gate_up = fwd && has_c2 ? 1 : 0;
  }

  // counters: int32 [2, >= tok_counters(ctas)], kept by the caller, parity alternating from launch to launch; none = cleared for this launch.
  void run(torch::Tensor group_off, c10::optional<torch::Tensor> group_rows, int64_t status_ptr, uint64_t timeout_ns, int ctas, int64_t gate_counter_ptr,
           c10::optional<torch::Tensor> gate_target, int gate_tile_rows, c10::optional<torch::Tensor> counters, int parity, int tile_n, bool early) const {
    TORCH_CHECK(group_off.is_cuda() && group_off.dtype() == torch::kInt32 && group_off.is_contiguous() && group_off.numel() == groups + 1, "group_off: cuda int32[G+1]");
    TokGemmArgs g = a;
    g.tile_n = tile_n;
    g.band_tiles = gemm::tok_band(band_rows_, 64 * g.red_blocks, g.m_tiles, tile_n);
    g.back_tiles = gemm::tok_back_tiles(64 * g.red_blocks, g.band_tiles, std::max(tile_n, gemm::kTokAccN));
    g.early = early ? 1 : 0;
    g.group_off = group_off.data_ptr<int>();
    if (group_rows.has_value()) {
      want(*group_rows, torch::kInt32, "group_rows");
      TORCH_CHECK(group_rows->numel() >= groups, "group_rows: int32 [G]");
      g.group_rows = group_rows->data_ptr<int>();
    }
    g.status = reinterpret_cast<DeviceStatus*>(status_ptr);
    g.timeout_ns = timeout_ns;
    if (gate_counter_ptr != 0) {
      TORCH_CHECK(gate_target.has_value() && gate_target->is_cuda() && gate_target->scalar_type() == torch::kInt64 &&
                  gate_target->numel() >= (gate_tile_rows > 0 ? 1 : groups), "gate_target: cuda int64[G], or one entry per tile with gate_tile_rows");
      g.gate_slots = static_cast<int>(gate_target->numel());
      g.gate_counter = reinterpret_cast<const unsigned long long*>(gate_counter_ptr);
      g.gate_target = reinterpret_cast<const unsigned long long*>(gate_target->data_ptr());
      g.gate_tile_rows = gate_tile_rows;
    }
    ctas &= ~1;
    const auto i32 = torch::TensorOptions().dtype(torch::kInt32).device(torch::kCUDA, device);
    auto partials = torch::empty({tok_partial_floats(ctas, tile_n)}, i32.dtype(torch::kFloat32));  // stream-ordered, as the launch is
    torch::Tensor cnt = counters.has_value() ? *counters : torch::zeros({2, tok_counters(ctas)}, i32);
    TORCH_CHECK(cnt.dim() == 2 && cnt.size(0) == 2 && cnt.is_contiguous() && cnt.scalar_type() == torch::kInt32, "counters: int32 [2, n]");
    unsigned int* base = reinterpret_cast<unsigned int*>(cnt.data_ptr<int>());
    g.partials = partials.data_ptr<float>();
    g.num_counters = static_cast<int>(cnt.size(1));
    g.counters = base + (parity & 1) * g.num_counters;
    g.counters_next = base + (~parity & 1) * g.num_counters;
    const TokGemmMaps maps{&w, &x, &c, has_c2 ? &c2 : nullptr};
    cu_check(launch_grouped_gemm_tokens(mode, epi, maps, g, ctas, stream_now()), "grouped_gemm_tokens launch");
  }
};

void grouped_gemm(int mode, int epilogue, const TensorMap2D& a, const TensorMap2D& b, torch::Tensor group_off, int tiles_n, int fixed_m_tiles,
                  int red_len, int b_rows_per_group, int c_rows_per_group, torch::Tensor c, c10::optional<torch::Tensor> c2, int64_t status_ptr,
                  uint64_t timeout_ns, int ctas, int64_t gate_counter_ptr, c10::optional<torch::Tensor> gate_target, bool pair, int band_rows,
                  const TensorMap2D* map_c, const TensorMap2D* map_c2, bool direct_epilogue, c10::optional<torch::Tensor> a_scales,
                  c10::optional<torch::Tensor> group_rows, int gate_tile_rows, bool wide) {
  TORCH_CHECK(group_off.is_cuda() && group_off.dtype() == torch::kInt32 && group_off.is_contiguous() && group_off.numel() >= 2, "group_off: cuda int32[G+1]");
  TORCH_CHECK(c.is_cuda() && c.dtype() == torch::kBFloat16 && c.dim() == 2 && c.stride(1) == 1, "c: cuda bf16 [rows, cols]");
  TORCH_CHECK(red_len % 64 == 0 && tiles_n >= 1, "reduction length must be a multiple of 64");
  GemmArgs g{};
  g.group_off = group_off.data_ptr<int>();
  g.num_groups = static_cast<int>(group_off.numel()) - 1;
  g.tiles_n = tiles_n; g.fixed_m_tiles = fixed_m_tiles; g.red_len = red_len;
  g.b_rows_per_group = b_rows_per_group; g.c_rows_per_group = c_rows_per_group;
  g.c = reinterpret_cast<__nv_bfloat16*>(c.data_ptr()); g.ldc = c.stride(0);
  if (c2.has_value()) {
    TORCH_CHECK(c2->is_cuda() && c2->dtype() == torch::kBFloat16 && c2->dim() == 2 && c2->stride(1) == 1, "c2: cuda bf16 [rows, cols]");
    g.c2 = reinterpret_cast<__nv_bfloat16*>(c2->data_ptr()); g.ldc2 = c2->stride(0);
  }
  g.status = reinterpret_cast<DeviceStatus*>(status_ptr);
  g.timeout_ns = timeout_ns;
  g.band_rows = band_rows;
  g.direct_epilogue = direct_epilogue ? 1 : 0;
  g.gate_tile_rows = gate_tile_rows;
  TORCH_CHECK(!wide || (pair && mode == static_cast<int>(GemmMode::kWgrad) && c.size(1) == 512ll * tiles_n), "grouped_gemm: tiles of 512 columns are for CTA-pair weight gradients of a multiple of 512 columns");
  g.wide = wide ? 1 : 0;
  if (a_scales.has_value()) {
    want(*a_scales, torch::kFloat32, "a_scales");
    TORCH_CHECK(pair && red_len % 128 == 0 && a_scales->dim() == 2 && a_scales->size(1) == red_len / 128, "a_scales: float [rows, red_len / 128], CTA-pair kernel");
    g.a_scales = a_scales->data_ptr<float>();
  }
  if (group_rows.has_value()) {
    want(*group_rows, torch::kInt32, "group_rows");
    TORCH_CHECK(group_rows->numel() >= g.num_groups, "group_rows: int32 [G]");
    g.group_rows = group_rows->data_ptr<int>();
  }
  if (gate_counter_ptr != 0) {
    TORCH_CHECK(gate_target.has_value() && gate_target->is_cuda() && gate_target->scalar_type() == torch::kInt64 &&
                gate_target->numel() >= (gate_tile_rows > 0 ? 1 : g.num_groups), "gate_target: cuda int64[G], or one entry per tile with gate_tile_rows");
    g.gate_slots = static_cast<int>(gate_target->numel());
    g.gate_counter = reinterpret_cast<const unsigned long long*>(gate_counter_ptr);
    g.gate_target = reinterpret_cast<const unsigned long long*>(gate_target->data_ptr());
  }
  if (pair) {
    TORCH_CHECK(map_c != nullptr && (map_c2 != nullptr) == c2.has_value(), "the CTA-pair kernel stores through tensor maps: give one for c, and one for c2 when c2 is given");
    cu_check(launch_grouped_gemm_pair(static_cast<GemmMode>(mode), static_cast<GemmEpilogue>(epilogue), a.map, b.map, map_c->map, map_c2 ? &map_c2->map : nullptr, g,
                                      ctas, stream_now()), "grouped_gemm pair launch");
  } else
    cu_check(launch_grouped_gemm(static_cast<GemmMode>(mode), static_cast<GemmEpilogue>(epilogue), a.map, b.map, g, ctas, stream_now()), "grouped_gemm launch");
}

void route_topk(torch::Tensor logits, c10::optional<torch::Tensor> bias, int K, torch::Tensor topk_idx, torch::Tensor topk_w,
                torch::Tensor slot_in_block, torch::Tensor block_cnt) {
  want(logits, torch::kFloat32, "logits"); want(topk_idx, torch::kInt32, "topk_idx"); want(topk_w, torch::kFloat32, "topk_w");
  want(slot_in_block, torch::kInt32, "slot_in_block"); want(block_cnt, torch::kInt32, "block_cnt");
  const int T = static_cast<int>(logits.size(0)), E = static_cast<int>(logits.size(1));
  const int blocks = (T + kRouteTokensPerBlock - 1) / kRouteTokensPerBlock;
  TORCH_CHECK(topk_idx.numel() == static_cast<int64_t>(T) * K && slot_in_block.numel() >= static_cast<int64_t>(blocks) * kRouteTokensPerBlock * K &&
              block_cnt.numel() == static_cast<int64_t>(blocks) * E, "route_topk: output shapes");
  cu_check(launch_route_topk(logits.data_ptr<float>(), ptr_or_null<const float>(bias), T, E, K, topk_idx.data_ptr<int>(), topk_w.data_ptr<float>(),
                             slot_in_block.data_ptr<int>(), block_cnt.data_ptr<int>(), stream_now()), "route_topk");
}

// The split scan of one engine: everything that stays the same from step to step (and the tensors it points into).
struct SplitsPlan {
  SplitsArgs a{};
  unsigned int* ticket = nullptr;
  std::vector<torch::Tensor> keep;
  int max_blocks = 0;

  SplitsPlan(const HeapPy& heap, int64_t counts_off, int64_t flags_off, torch::Tensor block_cnt, torch::Tensor block_base, torch::Tensor send_base, torch::Tensor send_cnt,
             torch::Tensor group_off, torch::Tensor group_rows, torch::Tensor arrive_target, c10::optional<torch::Tensor> traffic, int num_channels, int row_align, int cap_rows,
             const StatusPy& st, uint64_t timeout_ns, c10::optional<torch::Tensor> send_pos, int64_t epoch_dev_ptr, c10::optional<torch::Tensor> tile_target, int tile_rows,
             torch::Tensor ticket_word) {
    if (tile_target.has_value()) {
      want(*tile_target, torch::kInt64, "tile_target");
      TORCH_CHECK(tile_target->dim() == 2 && tile_target->size(0) == num_channels && tile_rows > 0, "tile_target: int64 [channels, tiles]");
      a.tile_target = reinterpret_cast<unsigned long long*>(tile_target->data_ptr());
      a.tile_rows = tile_rows;
      a.num_tiles = static_cast<int>(tile_target->size(1));
      keep.push_back(*tile_target);
    }
    a.row_align = row_align;
    a.cap_rows = cap_rows;
    a.peer_table = heap.h->device_peer_table(); a.rank = heap.h->rank(); a.world = heap.h->world();
    a.num_experts = static_cast<int>(send_base.numel()); a.num_channels = num_channels;
    max_blocks = static_cast<int>(block_cnt.numel() / a.num_experts);
    a.counts_heap_off = counts_off; a.flags_heap_off = flags_off;
    want(block_cnt, torch::kInt32, "block_cnt"); want(block_base, torch::kInt32, "block_base"); want(send_base, torch::kInt32, "send_base");
    want(send_cnt, torch::kInt32, "send_cnt"); want(group_off, torch::kInt32, "group_off"); want(group_rows, torch::kInt32, "group_rows");
    want(arrive_target, torch::kInt64, "arrive_target"); want(ticket_word, torch::kInt32, "ticket");
    const int El = a.num_experts / a.world;
    TORCH_CHECK(group_off.numel() == El + 1 && group_rows.numel() == El && arrive_target.numel() == static_cast<int64_t>(num_channels) * El && block_base.numel() >= block_cnt.numel(),
                "split scan: shapes");
    a.block_cnt = block_cnt.data_ptr<int>(); a.block_base = block_base.data_ptr<int>(); a.send_base = send_base.data_ptr<int>();
    a.send_cnt = send_cnt.data_ptr<int>(); a.group_off = group_off.data_ptr<int>(); a.group_rows = group_rows.data_ptr<int>();
    a.arrive_target = reinterpret_cast<unsigned long long*>(arrive_target.data_ptr());
    a.traffic_matrix = ptr_or_null<int>(traffic);
    a.send_pos = ptr_or_null<int>(send_pos);
    a.epoch_dev = reinterpret_cast<unsigned long long*>(epoch_dev_ptr);
    a.status = st.d; a.timeout_ns = timeout_ns;
    ticket = reinterpret_cast<unsigned int*>(ticket_word.data_ptr<int>());
    for (const auto& t : {block_cnt, block_base, send_base, send_cnt, group_off, group_rows, arrive_target, ticket_word}) keep.push_back(t);
    if (traffic.has_value()) keep.push_back(*traffic);
    if (send_pos.has_value()) keep.push_back(*send_pos);
  }
  SplitsArgs for_tokens(int64_t T, uint64_t epoch) const {
    SplitsArgs b = a;
    b.num_blocks = static_cast<int>((T + kRouteTokensPerBlock - 1) / kRouteTokensPerBlock);
    TORCH_CHECK(b.num_blocks <= max_blocks, "more tokens than the engine was made for");
    b.epoch = epoch;
    return b;
  }
};

void check_route_outputs(const SplitsPlan& p, int64_t T, int K, const torch::Tensor& topk_idx, const torch::Tensor& topk_w, const torch::Tensor& slot_in_block) {
  want(topk_idx, torch::kInt32, "topk_idx"); want(topk_w, torch::kFloat32, "topk_w"); want(slot_in_block, torch::kInt32, "slot_in_block");
  const int64_t blocks = (T + kRouteTokensPerBlock - 1) / kRouteTokensPerBlock;
  TORCH_CHECK(topk_idx.numel() == T * K && topk_w.numel() == T * K && slot_in_block.numel() >= blocks * kRouteTokensPerBlock * K, "route: output shapes");
}

// Top-k of ready-made logits and the split scan, one launch.
void route_splits(const SplitsPlan& p, torch::Tensor logits, c10::optional<torch::Tensor> bias, int K, torch::Tensor topk_idx, torch::Tensor topk_w,
                  torch::Tensor slot_in_block, uint64_t epoch) {
  want(logits, torch::kFloat32, "logits");
  const int64_t T = logits.size(0);
  TORCH_CHECK(logits.dim() == 2 && logits.size(1) == p.a.num_experts, "logits: float [T, experts]");
  check_route_outputs(p, T, K, topk_idx, topk_w, slot_in_block);
  const SplitsArgs a = p.for_tokens(T, epoch);
  if (T == 0) cu_check(launch_splits_scan(a, stream_now()), "splits_scan");   // no tokens of my own: the peers still want my counts
  else
    cu_check(launch_route_splits(logits.data_ptr<float>(), ptr_or_null<const float>(bias), static_cast<int>(T), K, topk_idx.data_ptr<int>(), topk_w.data_ptr<float>(),
                                 slot_in_block.data_ptr<int>(), a, p.ticket, stream_now()), "route_splits");
}

// The same from the activations of at most ROUTE_TOKENS_PER_BLOCK tokens: logits = bf16(x . gate^T).
void gate_route(const SplitsPlan& p, torch::Tensor x, torch::Tensor gate, c10::optional<torch::Tensor> bias, int K, torch::Tensor topk_idx, torch::Tensor topk_w,
                torch::Tensor slot_in_block, uint64_t epoch) {
  want16(x, torch::kBFloat16, "x"); want16(gate, torch::kBFloat16, "gate");
  const int64_t T = x.size(0);
  TORCH_CHECK(x.dim() == 2 && gate.dim() == 2 && gate.size(0) == p.a.num_experts && gate.size(1) == x.size(1) && T >= 1 && T <= kRouteTokensPerBlock, "gate_route: shapes");
  check_route_outputs(p, T, K, topk_idx, topk_w, slot_in_block);
  const SplitsArgs a = p.for_tokens(T, epoch);
  GateRouteArgs g{};
  g.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()); g.gate = reinterpret_cast<const __nv_bfloat16*>(gate.data_ptr()); g.bias = ptr_or_null<const float>(bias);
  g.T = static_cast<int>(T); g.H = static_cast<int>(x.size(1)); g.K = K;
  g.topk_idx = topk_idx.data_ptr<int>(); g.topk_w = topk_w.data_ptr<float>(); g.slot_in_block = slot_in_block.data_ptr<int>(); g.block_cnt = const_cast<int*>(a.block_cnt);
  cu_check(launch_gate_route(g, a, p.ticket, stream_now()), "gate_route");
}

void zero_pad_rows(torch::Tensor buf, torch::Tensor group_off, torch::Tensor group_rows, int align) {
  TORCH_CHECK(buf.is_cuda() && buf.dim() == 2 && buf.is_contiguous(), "buf: contiguous CUDA matrix");
  cu_check(launch_zero_pad_rows(buf.data_ptr(), buf.size(1) * buf.element_size(), group_off.data_ptr<int>(), group_rows.data_ptr<int>(),
                                static_cast<int>(group_rows.numel()), align, stream_now()), "zero_pad_rows");
}

// What every dispatch has: who sends (heap), the rows and the routing tables.
DispatchArgs dispatch_args(const HeapPy& heap, const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& slot_in_block, const torch::Tensor& block_base,
                           const torch::Tensor& send_base, const torch::Tensor& dest_row, const StatusPy& st, uint64_t timeout_ns) {
  want16(x, torch::kBFloat16, "x"); want(topk_idx, torch::kInt32, "topk_idx"); want(dest_row, torch::kInt32, "dest_row");
  DispatchArgs a{};
  a.peer_table = heap.h->device_peer_table(); a.rank = heap.h->rank(); a.world = heap.h->world();
  a.num_experts = static_cast<int>(send_base.numel()); a.T = static_cast<int>(x.size(0)); a.H = static_cast<int>(x.size(1));
  a.K = static_cast<int>(topk_idx.size(1));
  a.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()); a.topk_idx = topk_idx.data_ptr<int>();
  a.slot_in_block = slot_in_block.data_ptr<int>(); a.block_base = block_base.data_ptr<int>(); a.send_base = send_base.data_ptr<int>();
  a.dest_row = dest_row.data_ptr<int>();
  a.status = st.d; a.timeout_ns = timeout_ns;
  return a;
}
// ... and the receiver's matrix of bf16 rows that a rank alone may fill in place of the e4m3 one.
__nv_bfloat16* local_bf16_rows(const torch::Tensor& rows, const DispatchArgs& a) {
  want16(rows, torch::kBFloat16, "local_rows");
  TORCH_CHECK(a.fp8 && rows.dim() == 2 && rows.size(1) == a.H, "dispatch_push: local_rows belongs to the fp8 rows");
  return reinterpret_cast<__nv_bfloat16*>(rows.data_ptr());
}

void dispatch_push(const HeapPy& heap, torch::Tensor x, torch::Tensor topk_idx, c10::optional<torch::Tensor> row_scale, torch::Tensor slot_in_block,
                   torch::Tensor block_base, torch::Tensor send_base, torch::Tensor dest_row, bool compute_rows, bool fp8, int64_t recv_off,
                   int64_t scale_off, int64_t arrive_off, int64_t entry_flags_off, uint64_t entry_epoch, const StatusPy& st, uint64_t timeout_ns, int ctas,
                   c10::optional<torch::Tensor> send_list, int tile_rows, int num_tiles, c10::optional<torch::Tensor> xq,
                   c10::optional<torch::Tensor> xq_scales, c10::optional<torch::Tensor> local_rows, c10::optional<torch::Tensor> dot_out, int64_t y_off,
                   c10::optional<torch::Tensor> sum_with, c10::optional<torch::Tensor> grad_out, c10::optional<torch::Tensor> grad_loss, double grad_factor) {
  DispatchArgs a = dispatch_args(heap, x, topk_idx, slot_in_block, block_base, send_base, dest_row, st, timeout_ns);
  a.row_scale = ptr_or_null<const float>(row_scale);
  a.compute_rows = compute_rows; a.fp8 = fp8;
  a.send_list = ptr_or_null<const int>(send_list);
  a.tile_rows = tile_rows; a.num_tiles = num_tiles;
  if (xq.has_value()) {
    TORCH_CHECK(fp8 && xq_scales.has_value(), "dispatch_push: xq needs fp8 and xq_scales");
    want16(*xq, torch::kUInt8, "xq"); want(*xq_scales, torch::kFloat32, "xq_scales");
    TORCH_CHECK(xq->numel() >= x.numel() && xq_scales->numel() >= x.numel() / 128, "dispatch_push: xq / xq_scales too small");
    a.xq = xq->data_ptr<uint8_t>(); a.xq_scales = xq_scales->data_ptr<float>();
  }
  if (dot_out.has_value()) {
    want(*dot_out, torch::kFloat32, "dot_out");
    TORCH_CHECK(dot_out->numel() == topk_idx.numel(), "dispatch_push: dot_out is [T, K]");
    a.dot_out = dot_out->data_ptr<float>();
    a.y_heap_off = y_off;
    if (sum_with.has_value()) {
      TORCH_CHECK(grad_out.has_value() && grad_loss.has_value(), "dispatch_push: sum_with needs grad_out and grad_loss");
      want16(*sum_with, torch::kBFloat16, "sum_with"); want16(*grad_out, torch::kBFloat16, "grad_out"); want(*grad_loss, torch::kFloat32, "grad_loss");
      TORCH_CHECK(sum_with->sizes() == x.sizes() && grad_out->sizes() == x.sizes(), "dispatch_push: sum_with / grad_out shapes");
      a.sum_with = reinterpret_cast<const __nv_bfloat16*>(sum_with->data_ptr()); a.grad_out = reinterpret_cast<__nv_bfloat16*>(grad_out->data_ptr());
      a.grad_loss = grad_loss->data_ptr<float>(); a.grad_factor = static_cast<float>(grad_factor);
    }
  }
  if (local_rows.has_value()) a.local_rows = local_bf16_rows(*local_rows, a);
  a.recv_heap_off = recv_off; a.scale_heap_off = scale_off; a.arrive_heap_off = arrive_off;
  a.entry_flags_heap_off = entry_flags_off; a.entry_epoch = entry_epoch;
  cu_check(launch_dispatch_push(a, ctas, stream_now()), "dispatch_push");
}

// What every combine has: who pulls (heap), the routing tables, where the rows and the ready flags lie, and the output.
CombineArgs combine_args(const HeapPy& heap, int num_experts, const torch::Tensor& topk_idx, const torch::Tensor& dest_row, const c10::optional<torch::Tensor>& weights, int64_t src_off,
                         int64_t ready_off, uint64_t ready_epoch, const torch::Tensor& out, int H, const StatusPy& st, uint64_t timeout_ns) {
  CombineArgs a{};
  a.peer_table = heap.h->device_peer_table(); a.rank = heap.h->rank(); a.world = heap.h->world(); a.num_experts = num_experts;
  a.T = static_cast<int>(topk_idx.size(0)); a.K = static_cast<int>(topk_idx.size(1)); a.H = H;
  a.topk_idx = topk_idx.data_ptr<int>(); a.dest_row = dest_row.data_ptr<int>(); a.weights = ptr_or_null<const float>(weights);
  a.src_heap_off = src_off; a.ready_flags_heap_off = ready_off; a.ready_epoch = ready_epoch;
  want16(out, torch::kBFloat16, "out");
  a.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  a.status = st.d; a.timeout_ns = timeout_ns;
  return a;
}

// The two arguments after `out` are always None: positions that callers of an earlier form still fill.
void combine_pull(const HeapPy& heap, int num_experts, torch::Tensor topk_idx, torch::Tensor dest_row, c10::optional<torch::Tensor> weights, int64_t src_off,
                  int64_t ready_off, uint64_t ready_epoch, torch::Tensor out, py::none, py::none, int H, const StatusPy& st, uint64_t timeout_ns, int ctas, int64_t epoch_dev_ptr, bool signal,
                  c10::optional<torch::Tensor> residual, c10::optional<torch::Tensor> loss, double loss_scale, c10::optional<torch::Tensor> ticket) {
  CombineArgs a = combine_args(heap, num_experts, topk_idx, dest_row, weights, src_off, ready_off, ready_epoch, out, H, st, timeout_ns);
  torch::Tensor partials;
  if (residual.has_value()) {
    TORCH_CHECK(loss.has_value() && ticket.has_value(), "combine_pull: residual needs loss and ticket");
    want16(*residual, torch::kBFloat16, "residual"); want(*loss, torch::kFloat32, "loss"); want(*ticket, torch::kInt32, "ticket");
    TORCH_CHECK(residual->dim() == 2 && residual->size(0) == topk_idx.size(0) && residual->size(1) == H, "combine_pull: residual shape");
    partials = torch::empty({kMaxLossPartials}, loss->options());
    a.residual = reinterpret_cast<const __nv_bfloat16*>(residual->data_ptr()); a.loss = loss->data_ptr<float>(); a.loss_scale = static_cast<float>(loss_scale);
    a.loss_partials = partials.data_ptr<float>(); a.ticket = reinterpret_cast<unsigned int*>(ticket->data_ptr<int>());
  }
  a.signal = signal ? 1 : 0;
  a.epoch_dev = reinterpret_cast<const unsigned long long*>(epoch_dev_ptr);
  cu_check(launch_combine_pull(a, ctas, stream_now()), "combine_pull");
}

// Routing of few tokens, dispatch and combine of an engine that is alone (one rank, forward only, eager): the launches of the functions above
// with the engine's buffers bound once, so that a pass with few tokens, whose kernels take 45 us, is not paid for in interpreter time.
// What may change between passes (heap, rows, tables, grid, time limit) comes with every call.
struct LocalTransport {
  torch::Tensor slot_in_block, x_recv;
  bool fp8;
  int64_t recv_off, scale_off, y_off, ready_off;
  int K, tile_rows, num_tiles;

  // Returns (topk_idx, topk_w, dest_row).
  py::tuple gate_route(const SplitsPlan& splits, torch::Tensor x, torch::Tensor gate, c10::optional<torch::Tensor> bias, uint64_t epoch) const {
    const int64_t T = x.size(0);
    const auto i32 = torch::TensorOptions().dtype(torch::kInt32).device(x.device());
    auto topk_idx = torch::empty({T, K}, i32), dest_row = torch::empty({T, K}, i32), topk_w = torch::empty({T, K}, i32.dtype(torch::kFloat32));
    ::gate_route(splits, x, gate, bias, K, topk_idx, topk_w, slot_in_block, epoch);
    return py::make_tuple(topk_idx, topk_w, dest_row);
  }
  void dispatch(const HeapPy& heap, const StatusPy& st, torch::Tensor x, torch::Tensor topk_idx, torch::Tensor slots, torch::Tensor block_base, torch::Tensor send_base, torch::Tensor dest_row,
                uint64_t timeout_ns, int ctas) const {
    DispatchArgs a = dispatch_args(heap, x, topk_idx, slots, block_base, send_base, dest_row, st, timeout_ns);
    a.compute_rows = true; a.fp8 = fp8;
    if (fp8) a.local_rows = local_bf16_rows(x_recv, a);
    a.recv_heap_off = recv_off; a.scale_heap_off = scale_off;
    a.arrive_heap_off = -1;   // the rows are in when the kernel ends: nobody waits for a count
    a.tile_rows = tile_rows; a.num_tiles = num_tiles;
    cu_check(launch_dispatch_push(a, ctas, stream_now()), "dispatch_push");
  }
  torch::Tensor combine(const HeapPy& heap, const StatusPy& st, int num_experts, torch::Tensor topk_idx, torch::Tensor dest_row, c10::optional<torch::Tensor> weights,
                        uint64_t epoch, uint64_t timeout_ns, int ctas) const {
    const int H = static_cast<int>(x_recv.size(1));
    auto out = torch::empty({topk_idx.size(0), H}, x_recv.options());
    CombineArgs a = combine_args(heap, num_experts, topk_idx, dest_row, weights, y_off, ready_off, epoch, out, H, st, timeout_ns);
    a.signal = 1;
    cu_check(launch_combine_pull(a, ctas, stream_now()), "combine_pull");
    return out;
  }
};

}  // namespace

void bind_moe(py::module_& m) {
  py::class_<LocalTransport>(m, "LocalTransport")
      .def(py::init([](torch::Tensor slot_in_block, torch::Tensor x_recv, bool fp8, int64_t recv_off, int64_t scale_off, int64_t y_off, int64_t ready_off, int k, int tile_rows, int num_tiles) {
        want(slot_in_block, torch::kInt32, "slot_in_block"); want16(x_recv, torch::kBFloat16, "x_recv");
        return LocalTransport{slot_in_block, x_recv, fp8, recv_off, scale_off, y_off, ready_off, k, tile_rows, num_tiles};
      }), py::arg("slot_in_block"), py::arg("x_recv"), py::arg("fp8"), py::arg("recv_off"), py::arg("scale_off"), py::arg("y_off"), py::arg("ready_off"), py::arg("k"), py::arg("tile_rows"),
           py::arg("num_tiles"))
      .def("gate_route", &LocalTransport::gate_route)
      .def("dispatch", &LocalTransport::dispatch)
      .def("combine", &LocalTransport::combine);
  py::class_<TensorMap2D>(m, "TensorMap2D").def(py::init<int64_t, int64_t, int64_t, int64_t, int, int>()).def_static("bytes", &TensorMap2D::bytes);
  py::class_<TokGemmPlan>(m, "TokGemmPlan")
      .def(py::init<int, int, torch::Tensor, torch::Tensor, torch::Tensor, c10::optional<torch::Tensor>, int, int>())
      .def("matches", &TokGemmPlan::matches)
      .def("run", &TokGemmPlan::run, py::arg("group_off"), py::arg("group_rows"), py::arg("status_ptr"), py::arg("timeout_ns"), py::arg("ctas"),
           py::arg("gate_counter_ptr") = 0, py::arg("gate_target") = py::none(), py::arg("gate_tile_rows") = 0, py::arg("counters") = py::none(), py::arg("parity") = 0, py::arg("tile_n") = 256, py::arg("early") = false);
  m.attr("TOK_COUNTERS_PER_CTA") = tok_counters(1);
  // How a launch with these rows per group splits its work: what a test names the sizes of a path by.
  m.def("token_split", [](const std::vector<int>& rows, int m_tiles, int red_len, int tile_n, int granule, int pairs) {
    using namespace gemm;
    struct Groups { const int *group_off, *group_rows; int granule, tile_n, m_tiles; };
    const Groups q{nullptr, rows.data(), granule, tile_n, m_tiles};
    int tiles = 0, widest = 0, most = 0;
    for (int g = 0; g < static_cast<int>(rows.size()); ++g) {
      tiles += tok_group_tiles(q, g);
      widest = std::max(widest, tok_tile_size(tok_rows(q, g), tile_n));
      most = std::max(most, tok_tiles(tok_rows(q, g), tile_n));
    }
    const TokSplit s = TokSplit::make(tiles, red_len / 64, pairs, widest, most > 1);
    py::dict d;
    d["token_tiles"] = most; d["cut_tiles"] = s.cut_tiles; d["whole_tiles"] = s.whole_tiles; d["shares"] = s.shares; d["stream"] = s.stream;
    d["back_tiles"] = tok_back_tiles(red_len, tok_band(0, red_len, m_tiles, tile_n), std::max(tile_n, kTokAccN));
    return d;
  }, py::arg("rows"), py::arg("m_tiles"), py::arg("red_len"), py::arg("tile_n"), py::arg("granule"), py::arg("pairs"));
  m.def("grouped_gemm", &grouped_gemm, py::arg("mode"), py::arg("epilogue"), py::arg("a"), py::arg("b"), py::arg("group_off"), py::arg("tiles_n"),
        py::arg("fixed_m_tiles"), py::arg("red_len"), py::arg("b_rows_per_group"), py::arg("c_rows_per_group"), py::arg("c"), py::arg("c2"),
        py::arg("status_ptr"), py::arg("timeout_ns"), py::arg("ctas"), py::arg("gate_counter_ptr"), py::arg("gate_target"), py::arg("pair"),
        py::arg("band_rows"), py::arg("map_c") = nullptr, py::arg("map_c2") = nullptr, py::arg("direct_epilogue") = false, py::arg("a_scales") = py::none(),
        py::arg("group_rows") = py::none(), py::arg("gate_tile_rows") = 0, py::arg("wide") = false);
  m.def("grouped_gemm_smem_bytes", &grouped_gemm_smem_bytes);
  m.attr("ROUTE_TOKENS_PER_BLOCK") = kRouteTokensPerBlock;
  m.def("route_topk", &route_topk);
  py::class_<SplitsPlan>(m, "SplitsPlan")
      .def(py::init<const HeapPy&, int64_t, int64_t, torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor,
                    c10::optional<torch::Tensor>, int, int, int, const StatusPy&, uint64_t, c10::optional<torch::Tensor>, int64_t, c10::optional<torch::Tensor>, int, torch::Tensor>(),
           py::arg("heap"), py::arg("counts_off"), py::arg("flags_off"), py::arg("block_cnt"), py::arg("block_base"), py::arg("send_base"), py::arg("send_cnt"),
           py::arg("group_off"), py::arg("group_rows"), py::arg("arrive_target"), py::arg("traffic"), py::arg("num_channels"), py::arg("row_align"), py::arg("cap_rows"),
           py::arg("status"), py::arg("timeout_ns"), py::arg("send_pos"), py::arg("epoch_dev_ptr"), py::arg("tile_target"), py::arg("tile_rows"), py::arg("ticket"));
  m.def("route_splits", &route_splits);
  m.def("gate_route", &gate_route);
  m.def("gate_route_fits", &gate_route_fits, py::arg("world"), py::arg("experts"), py::arg("k"), py::arg("hidden"));
  m.def("zero_pad_rows", &zero_pad_rows, py::arg("buf"), py::arg("group_off"), py::arg("group_rows"), py::arg("align") = 0);
  m.def("build_send_list", [](torch::Tensor topk_idx, torch::Tensor slot_in_block, torch::Tensor block_base, torch::Tensor send_pos, torch::Tensor list, const StatusPy& st) {
    want(topk_idx, torch::kInt32, "topk_idx"); want(send_pos, torch::kInt32, "send_pos"); want(list, torch::kInt32, "list");
    TORCH_CHECK(list.numel() >= topk_idx.numel(), "build_send_list: list too short");
    cu_check(launch_build_send_list(topk_idx.data_ptr<int>(), slot_in_block.data_ptr<int>(), block_base.data_ptr<int>(), send_pos.data_ptr<int>(),
                                    static_cast<int>(topk_idx.size(0)), static_cast<int>(topk_idx.size(1)), static_cast<int>(send_pos.numel()),
                                    list.data_ptr<int>(), st.d, stream_now()), "build_send_list");
  });
  m.def("norm_gate_smem_bytes", [](int E, int H, int K, bool backward) { return static_cast<int64_t>(norm_gate_smem_bytes(E, H, K, backward)); });
  m.def("norm_gate_route", [](torch::Tensor h, torch::Tensor norm_w, torch::Tensor gate, c10::optional<torch::Tensor> bias, int K, double eps, torch::Tensor hn,
                              torch::Tensor rstd, torch::Tensor logits, torch::Tensor topk_idx, torch::Tensor topk_w, torch::Tensor slot_in_block,
                              torch::Tensor block_cnt, const SplitsPlan* splits, uint64_t epoch) {
    want16(h, torch::kBFloat16, "h"); want16(norm_w, torch::kBFloat16, "norm_w"); want16(gate, torch::kBFloat16, "gate"); want16(hn, torch::kBFloat16, "hn");
    want(rstd, torch::kFloat32, "rstd"); want(logits, torch::kFloat32, "logits"); want(topk_idx, torch::kInt32, "topk_idx"); want(topk_w, torch::kFloat32, "topk_w");
    want(slot_in_block, torch::kInt32, "slot_in_block"); want(block_cnt, torch::kInt32, "block_cnt");
    NormGateArgs a{};
    a.T = static_cast<int>(h.size(0)); a.H = static_cast<int>(h.size(1)); a.num_experts = static_cast<int>(gate.size(0)); a.K = K; a.eps = static_cast<float>(eps);
    const int blocks = (a.T + kRouteTokensPerBlock - 1) / kRouteTokensPerBlock;
    TORCH_CHECK(gate.size(1) == a.H && norm_w.numel() == a.H && hn.sizes() == h.sizes() && rstd.numel() >= a.T && logits.numel() == static_cast<int64_t>(a.T) * a.num_experts &&
                topk_idx.numel() == static_cast<int64_t>(a.T) * K && topk_w.numel() == topk_idx.numel() &&
                slot_in_block.numel() >= static_cast<int64_t>(blocks) * kRouteTokensPerBlock * K && block_cnt.numel() >= static_cast<int64_t>(blocks) * a.num_experts,
                "norm_gate_route: shapes");
    a.h = reinterpret_cast<const __nv_bfloat16*>(h.data_ptr()); a.norm_w = reinterpret_cast<const __nv_bfloat16*>(norm_w.data_ptr());
    a.gate = reinterpret_cast<const __nv_bfloat16*>(gate.data_ptr()); a.bias = ptr_or_null<const float>(bias);
    a.hn = reinterpret_cast<__nv_bfloat16*>(hn.data_ptr()); a.rstd = rstd.data_ptr<float>(); a.logits = logits.data_ptr<float>();
    a.topk_idx = topk_idx.data_ptr<int>(); a.topk_w = topk_w.data_ptr<float>(); a.slot_in_block = slot_in_block.data_ptr<int>(); a.block_cnt = block_cnt.data_ptr<int>();
    if (splits == nullptr) {
      auto tickets = torch::zeros({norm_gate_tickets(a.T)}, topk_idx.options());
      cu_check(launch_norm_gate_route(a, nullptr, reinterpret_cast<unsigned int*>(tickets.data_ptr<int>()), stream_now()), "norm_gate_route");
      return;
    }
    const SplitsArgs sp = splits->for_tokens(a.T, epoch);
    if (a.T == 0) cu_check(launch_splits_scan(sp, stream_now()), "splits_scan");
    else cu_check(launch_norm_gate_route(a, &sp, splits->ticket, stream_now()), "norm_gate_route");
  }, py::arg("h"), py::arg("norm_w"), py::arg("gate"), py::arg("bias"), py::arg("k"), py::arg("eps"), py::arg("hn"), py::arg("rstd"), py::arg("logits"), py::arg("topk_idx"),
     py::arg("topk_w"), py::arg("slot_in_block"), py::arg("block_cnt"), py::arg("splits") = nullptr, py::arg("epoch") = 0);
  m.def("norm_gate_bwd", [](torch::Tensor h, torch::Tensor norm_w, torch::Tensor gate, torch::Tensor rstd, torch::Tensor topk_idx, torch::Tensor topk_w,
                            torch::Tensor grad_w, torch::Tensor grad_hn, torch::Tensor grad_h, torch::Tensor d_gate, torch::Tensor d_norm_w,
                            c10::optional<torch::Tensor> residual) {
    want16(h, torch::kBFloat16, "h"); want16(norm_w, torch::kBFloat16, "norm_w"); want16(gate, torch::kBFloat16, "gate"); want(rstd, torch::kFloat32, "rstd");
    want(topk_idx, torch::kInt32, "topk_idx"); want(topk_w, torch::kFloat32, "topk_w"); want(grad_w, torch::kFloat32, "grad_w");
    want16(grad_hn, torch::kBFloat16, "grad_hn"); want16(grad_h, torch::kBFloat16, "grad_h");
    const bool as_bf16 = d_gate.scalar_type() == torch::kBFloat16;   // written as bf16, or accumulated into as fp32
    want(d_gate, as_bf16 ? torch::kBFloat16 : torch::kFloat32, "d_gate"); want(d_norm_w, as_bf16 ? torch::kBFloat16 : torch::kFloat32, "d_norm_w");
    NormGateBwdArgs a{};
    a.T = static_cast<int>(h.size(0)); a.H = static_cast<int>(h.size(1)); a.num_experts = static_cast<int>(gate.size(0)); a.K = static_cast<int>(topk_idx.size(1));
    TORCH_CHECK(gate.size(1) == a.H && grad_hn.sizes() == h.sizes() && grad_h.sizes() == h.sizes() && d_gate.numel() == gate.numel() && d_norm_w.numel() == a.H &&
                grad_w.sizes() == topk_idx.sizes() && topk_w.sizes() == topk_idx.sizes() && rstd.numel() >= a.T, "norm_gate_bwd: shapes");
    a.h = reinterpret_cast<const __nv_bfloat16*>(h.data_ptr()); a.norm_w = reinterpret_cast<const __nv_bfloat16*>(norm_w.data_ptr());
    a.gate = reinterpret_cast<const __nv_bfloat16*>(gate.data_ptr()); a.rstd = rstd.data_ptr<float>(); a.topk_idx = topk_idx.data_ptr<int>();
    a.topk_w = topk_w.data_ptr<float>(); a.grad_w = grad_w.data_ptr<float>(); a.grad_hn = reinterpret_cast<const __nv_bfloat16*>(grad_hn.data_ptr());
    a.grad_h = reinterpret_cast<__nv_bfloat16*>(grad_h.data_ptr());
    if (as_bf16) { a.d_gate_bf16 = reinterpret_cast<__nv_bfloat16*>(d_gate.data_ptr()); a.d_norm_w_bf16 = reinterpret_cast<__nv_bfloat16*>(d_norm_w.data_ptr()); }
    else { a.d_gate = d_gate.data_ptr<float>(); a.d_norm_w = d_norm_w.data_ptr<float>(); }
    if (residual.has_value()) {
      want16(*residual, torch::kBFloat16, "residual");
      TORCH_CHECK(residual->sizes() == h.sizes(), "norm_gate_bwd: residual shape");
      a.residual = reinterpret_cast<const __nv_bfloat16*>(residual->data_ptr());
    }
    const int blocks = norm_gate_bwd_blocks(a.T, a.H, a.num_experts, at::cuda::getCurrentDeviceProperties()->multiProcessorCount);
    auto partials = torch::empty({blocks, a.num_experts + 1, a.H}, h.options().dtype(torch::kFloat32));
    a.partials = partials.data_ptr<float>();
    if (a.T == 0 && as_bf16) { d_gate.zero_(); d_norm_w.zero_(); }
    cu_check(launch_norm_gate_bwd(a, blocks, stream_now()), "norm_gate_bwd");
  }, py::arg("h"), py::arg("norm_w"), py::arg("gate"), py::arg("rstd"), py::arg("topk_idx"), py::arg("topk_w"), py::arg("grad_w"), py::arg("grad_hn"), py::arg("grad_h"),
     py::arg("d_gate"), py::arg("d_norm_w"), py::arg("residual") = py::none());
  m.def("dispatch_push", &dispatch_push, py::arg("heap"), py::arg("x"), py::arg("topk_idx"), py::arg("row_scale"), py::arg("slot_in_block"), py::arg("block_base"),
        py::arg("send_base"), py::arg("dest_row"), py::arg("compute_rows"), py::arg("fp8"), py::arg("recv_off"), py::arg("scale_off"), py::arg("arrive_off"),
        py::arg("entry_flags_off"), py::arg("entry_epoch"), py::arg("status"), py::arg("timeout_ns"), py::arg("ctas"), py::arg("send_list"),
        py::arg("tile_rows") = 0, py::arg("num_tiles") = 0, py::arg("xq") = py::none(), py::arg("xq_scales") = py::none(), py::arg("local_rows") = py::none(), py::arg("dot_out") = py::none(),
        py::arg("y_off") = 0, py::arg("sum_with") = py::none(), py::arg("grad_out") = py::none(), py::arg("grad_loss") = py::none(), py::arg("grad_factor") = 0.0);
  m.def("quantise_rows", [](torch::Tensor x, torch::Tensor q, torch::Tensor scales, int ctas) {
    want16(x, torch::kBFloat16, "x"); want16(q, torch::kUInt8, "q"); want(scales, torch::kFloat32, "scales");
    TORCH_CHECK(x.dim() == 2 && q.numel() >= x.numel() && scales.numel() >= x.numel() / 128, "quantise_rows: q / scales too small");
    cu_check(launch_quantise_rows(reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()), static_cast<int>(x.size(0)), static_cast<int>(x.size(1)),
                                  q.data_ptr<uint8_t>(), scales.data_ptr<float>(), ctas, stream_now()), "quantise_rows");
  });
  m.def("combine_pull", &combine_pull, py::arg("heap"), py::arg("num_experts"), py::arg("topk_idx"), py::arg("dest_row"), py::arg("weights"), py::arg("src_off"), py::arg("ready_off"),
        py::arg("ready_epoch"), py::arg("out"), py::arg("unused1"), py::arg("unused2"), py::arg("hidden"), py::arg("status"), py::arg("timeout_ns"), py::arg("ctas"),
        py::arg("epoch_dev_ptr"), py::arg("signal") = false, py::arg("residual") = py::none(), py::arg("loss") = py::none(), py::arg("loss_scale") = 1.0, py::arg("ticket") = py::none());
  m.def("wait_counters", [](int64_t counter_ptr, torch::Tensor target, const StatusPy& st, uint64_t timeout_ns) {
    cu_check(launch_wait_counters(reinterpret_cast<const unsigned long long*>(counter_ptr), reinterpret_cast<const unsigned long long*>(target.data_ptr()),
                                  static_cast<int>(target.numel()), st.d, timeout_ns, stream_now()), "wait_counters");
  });
  m.def("swiglu_fwd", [](torch::Tensor gu, torch::Tensor act) {
    want16(gu, torch::kBFloat16, "gate_up"); want16(act, torch::kBFloat16, "act");
    cu_check(launch_swiglu_fwd(reinterpret_cast<const __nv_bfloat16*>(gu.data_ptr()), reinterpret_cast<__nv_bfloat16*>(act.data_ptr()), gu.size(0),
                               static_cast<int>(act.size(1)), stream_now()), "swiglu_fwd");
  });
  m.def("swiglu_bwd", [](torch::Tensor gu, torch::Tensor dact, torch::Tensor dgu, int64_t rows_dev_ptr) {
    want16(gu, torch::kBFloat16, "gate_up"); want16(dact, torch::kBFloat16, "d_act"); want16(dgu, torch::kBFloat16, "d_gate_up");
    cu_check(launch_swiglu_bwd(reinterpret_cast<const __nv_bfloat16*>(gu.data_ptr()), reinterpret_cast<const __nv_bfloat16*>(dact.data_ptr()),
                               reinterpret_cast<__nv_bfloat16*>(dgu.data_ptr()), gu.size(0), static_cast<int>(dact.size(1)), reinterpret_cast<const int*>(rows_dev_ptr),
                               stream_now()), "swiglu_bwd");
  });
  m.def("dequant_fp8", [](torch::Tensor q, torch::Tensor scales, torch::Tensor out, int64_t rows_dev_ptr) {
    want_aligned(q, torch::kUInt8, "q", 8); want(scales, torch::kFloat32, "scales"); want16(out, torch::kBFloat16, "out");
    cu_check(launch_dequant_fp8(q.data_ptr<uint8_t>(), scales.data_ptr<float>(), reinterpret_cast<__nv_bfloat16*>(out.data_ptr()), q.size(0),
                                static_cast<int>(q.size(1)), reinterpret_cast<const int*>(rows_dev_ptr), stream_now()), "dequant_fp8");
  });
  m.def("sumsq_add", [](torch::Tensor a, torch::Tensor b, double scale, torch::Tensor partial, torch::Tensor out) {
    want16(a, torch::kBFloat16, "a"); want16(b, torch::kBFloat16, "b"); want(partial, torch::kFloat32, "partial"); want(out, torch::kFloat32, "out");
    TORCH_CHECK(a.numel() == b.numel(), "sumsq_add: shapes");
    cu_check(launch_sumsq_add(reinterpret_cast<const __nv_bfloat16*>(a.data_ptr()), reinterpret_cast<const __nv_bfloat16*>(b.data_ptr()), a.numel(),
                              static_cast<float>(scale), partial.data_ptr<float>(), static_cast<int>(partial.numel()), out.data_ptr<float>(), stream_now()), "sumsq_add");
  });
  m.def("scaled_sum", [](torch::Tensor a, torch::Tensor b, torch::Tensor gscale, double factor, torch::Tensor out) {
    want16(a, torch::kBFloat16, "a"); want16(b, torch::kBFloat16, "b"); want(gscale, torch::kFloat32, "gscale"); want16(out, torch::kBFloat16, "out");
    cu_check(launch_scaled_sum(reinterpret_cast<const __nv_bfloat16*>(a.data_ptr()), reinterpret_cast<const __nv_bfloat16*>(b.data_ptr()), a.numel(),
                               gscale.data_ptr<float>(), static_cast<float>(factor), reinterpret_cast<__nv_bfloat16*>(out.data_ptr()), stream_now()), "scaled_sum");
  });
  // grad_out [T, H] summed by id in position order -> a new table gradient [V, H] (rows that no id names are zero).
  m.def("embedding_grad", [](torch::Tensor ids, int V, torch::Tensor grad_out) {
    want(ids, torch::kInt64, "ids"); want16(grad_out, torch::kBFloat16, "grad_out");
    const int64_t T = ids.numel(), H = grad_out.size(1);
    TORCH_CHECK(grad_out.dim() == 2 && grad_out.size(0) == T, "embedding_grad: one gradient row per id");
    auto table = torch::empty({V, H}, grad_out.options());
    const long long* idp = reinterpret_cast<const long long*>(ids.data_ptr());
    const __nv_bfloat16* g = reinterpret_cast<const __nv_bfloat16*>(grad_out.data_ptr());
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(table.data_ptr());
    // What a block can file in shared memory; above, the sort's six launches.
    if (T <= 4096) {
      cu_check(launch_embedding_few(idp, g, out, static_cast<int>(T), V, static_cast<int>(H), stream_now()), "embedding_grad");
      return table;
    }
    const int64_t blocks = (T + embedding_index_block() - 1) / embedding_index_block();
    auto i32 = torch::TensorOptions().dtype(torch::kInt32).device(ids.device());
    auto hist = torch::empty({blocks, V}, i32), rank = torch::empty({T}, i32), total = torch::empty({V}, i32), start = torch::empty({V + 1}, i32);
    auto sorted_ids = torch::empty({T}, ids.options()), perm = torch::empty({T}, ids.options());
    cu_check(launch_embedding_index(idp, T, V, hist.data_ptr<int>(), rank.data_ptr<int>(), total.data_ptr<int>(), start.data_ptr<int>(),
                                    reinterpret_cast<long long*>(sorted_ids.data_ptr()), reinterpret_cast<long long*>(perm.data_ptr()), stream_now()), "embedding_grad");
    cu_check(launch_embedding_rows(start.data_ptr<int>(), reinterpret_cast<const long long*>(perm.data_ptr()), g, out, V, static_cast<int>(H), stream_now()), "embedding_grad");
    return table;
  });
  m.def("embedding_index", [](torch::Tensor ids, int V) {
    want(ids, torch::kInt64, "ids");
    const int64_t T = ids.numel();
    const int64_t blocks = (T + embedding_index_block() - 1) / embedding_index_block();
    auto i32 = torch::TensorOptions().dtype(torch::kInt32).device(ids.device());
    auto hist = torch::empty({blocks, V}, i32), rank = torch::empty({T}, i32), total = torch::empty({V}, i32), start = torch::empty({V + 1}, i32);
    auto sorted_ids = torch::empty({T}, ids.options()), perm = torch::empty({T}, ids.options());
    cu_check(launch_embedding_index(reinterpret_cast<const long long*>(ids.data_ptr()), T, V, hist.data_ptr<int>(), rank.data_ptr<int>(), total.data_ptr<int>(),
                                    start.data_ptr<int>(), reinterpret_cast<long long*>(sorted_ids.data_ptr()), reinterpret_cast<long long*>(perm.data_ptr()), stream_now()),
             "embedding_index");
    return std::make_tuple(sorted_ids, perm);
  });
  // One step of several tensors: lists of equal length, steps[k] = the step number that tensor k takes now.
  const auto adamw_step = [](const std::vector<torch::Tensor>& params, const std::vector<torch::Tensor>& masters, const std::vector<torch::Tensor>& ms, const std::vector<torch::Tensor>& vs,
                    const std::vector<torch::Tensor>& grads, const std::vector<int64_t>& steps, double lr, double b1, double b2, double eps, double wd, double grad_scale) {
    const size_t n = params.size();
    TORCH_CHECK(masters.size() == n && ms.size() == n && vs.size() == n && grads.size() == n && steps.size() == n, "adamw: lists of equal length");
    for (size_t k0 = 0; k0 < n; k0 += kAdamWTensors) {
      AdamWArgs a{};
      a.lr = static_cast<float>(lr); a.b1 = static_cast<float>(b1); a.b2 = static_cast<float>(b2); a.eps = static_cast<float>(eps); a.wd = static_cast<float>(wd);
      a.gscale = static_cast<float>(grad_scale);
      for (size_t k = k0; k < std::min(n, k0 + kAdamWTensors); ++k) {
        want_aligned(params[k], torch::kBFloat16, "param", 8); want16(masters[k], torch::kFloat32, "master"); want16(ms[k], torch::kFloat32, "m"); want16(vs[k], torch::kFloat32, "v");
        want_aligned(grads[k], torch::kBFloat16, "grad", 8);
        const int64_t len = params[k].numel();
        TORCH_CHECK(masters[k].numel() == len && ms[k].numel() == len && vs[k].numel() == len && grads[k].numel() == len, "adamw: sizes");
        AdamWTensor& t = a.t[a.count++];
        t.param = reinterpret_cast<__nv_bfloat16*>(params[k].data_ptr());
        t.master = masters[k].data_ptr<float>(); t.m = ms[k].data_ptr<float>(); t.v = vs[k].data_ptr<float>();
        t.grad = reinterpret_cast<const __nv_bfloat16*>(grads[k].data_ptr());
        t.n = len;
        t.c1 = static_cast<float>(1.0 / (1.0 - std::pow(b1, static_cast<double>(steps[k])))); t.c2 = static_cast<float>(1.0 / (1.0 - std::pow(b2, static_cast<double>(steps[k]))));
      }
      cu_check(launch_adamw(a, stream_now()), "adamw");
    }
  };
  m.def("adamw_step", adamw_step);
  m.def("adamw", [adamw_step](torch::Tensor param, torch::Tensor master, torch::Tensor m1, torch::Tensor v, torch::Tensor grad, double lr, double b1, double b2, double eps, double wd,
                              int64_t step, double grad_scale) { adamw_step({param}, {master}, {m1}, {v}, {grad}, {step}, lr, b1, b2, eps, wd, grad_scale); });
}
