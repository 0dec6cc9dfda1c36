// MoE routing on the device, with no host round trip between the gate and the expert GEMMs:
//   route_topk   : softmax(+bias) top-k per token, per-block expert histogram and the stable rank
//                  of every (token, slot) inside its block;
//   splits_scan  : prefix sums over blocks -> per-expert send counts, all-gather of the counts by
//                  direct stores into every peer's symmetric pad, then receive offsets, padded
//                  group offsets for the grouped GEMM and cumulative arrival targets.
// The reference has no router; its counterpart of the count exchange is the host-side workload
// broadcast (nvidia/alltoall_nvshmem.cpp:452-472), which this replaces with ~1 KB of NVLink stores.
#include <algorithm>

#include "early_start.cuh"
#include "route_rank.cuh"
#include "route_splits.cuh"

namespace fastb {

namespace {

constexpr int kTokensPerBlock = kRouteTokensPerBlock;
constexpr int kRouteThreads = 1024;
// ints in front of the token's row in gate_route_kernel's shared memory: a sum per expert, or per warp where several share one; whole 16 bytes.
__host__ __device__ constexpr int gate_route_parts_ints(int E) { return ((E > 32 ? E : 32) + 3) & ~3; }

// One warp per token at a time. E <= 256 (8 values per lane). 32 warps: a block owns 128 tokens whatever T is, so at small T
// the warps of one block are all the parallelism there is.
// SPLITS: the last block goes on with the split scan.
template <int MAX_PER_LANE, bool SPLITS>
__global__ void __launch_bounds__(kRouteThreads) route_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int T, int E,
                                                                   int K, int* __restrict__ topk_idx, float* __restrict__ topk_w,
                                                                   int* __restrict__ slot_in_block, int* __restrict__ block_cnt, const SplitsArgs sp,
                                                                   unsigned int* ticket) {
  extern __shared__ int s_eid[];  // [kTokensPerBlock * K], then the counts of block_stable_ranks; later the split scan's tables
  grid_dependency_wait();
  launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = kRouteThreads / 32;
  const int t0 = blockIdx.x * kTokensPerBlock;
  const int nt = min(kTokensPerBlock, T - t0);
  for (int lt = warp; lt < kTokensPerBlock; lt += nwarps) {
    const int t = t0 + lt;
    if (lt >= nt) {
      for (int j = lane; j < K; j += 32) s_eid[lt * K + j] = -1;
      continue;
    }
    // Selection uses logits + bias; the weights are the softmax of the raw logits over the
    // chosen experts (renormalised), which for bias == 0 is Mixtral's softmax-over-top-k.
    float sel[MAX_PER_LANE], raw[MAX_PER_LANE];
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
      const int e = lane + 32 * i;
      // NaN logits count as -inf: the selection stays total and the weights stay finite.
      float r = e < E ? logits[static_cast<long long>(t) * E + e] : -INFINITY;
      if (r != r) r = -INFINITY;
      float s = e < E ? r + (bias ? bias[e] : 0.0f) : -INFINITY;
      if (s != s) s = -INFINITY;
      raw[i] = r;
      sel[i] = s;
    }
    int my_e;
    float my_w;
    route::warp_topk<MAX_PER_LANE>(sel, raw, E, K, my_e, my_w);
    if (lane < K) {
      topk_idx[static_cast<long long>(t) * K + lane] = my_e;
      topk_w[static_cast<long long>(t) * K + lane] = my_w;
      s_eid[lt * K + lane] = my_e;
    }
  }
  __syncthreads();
  route::block_stable_ranks(s_eid, reinterpret_cast<unsigned short*>(s_eid + kTokensPerBlock * K), E, K, slot_in_block + static_cast<long long>(t0) * K,
                            block_cnt + static_cast<long long>(blockIdx.x) * E);
  if (SPLITS && route::last_block(ticket)) route::splits_block(sp, s_eid);
}

__global__ void __launch_bounds__(1024) splits_scan_kernel(const SplitsArgs a) {
  extern __shared__ int s_splits[];
  route::splits_block(a, s_splits);
}

// Router logits of a few tokens with the whole routing behind them, in one launch: a block per token computes its logits (fp32
// sums of bf16 products, rounded to bf16 as a bf16 GEMM returns them) and chooses its experts; the last block then ranks
// all entries and does the split scan. Up to kRouteTokensPerBlock tokens. A library GEMM, a conversion, route_topk and
// splits_scan took 20 us for one token, 35 us for 64.
// Bound by latency, a chain of dependent steps: the block's read of the gate from L2 (eight 16-byte words of it in flight per lane, the token's
// row in shared memory), the choice, the meeting of the blocks, the ranks, the scan. A single token meets nobody, and the one routing
// block's counts go to the scan through shared memory. Thousands of cycles inside, before -> after: 1 token and 8 experts of 1024 14.5 -> 9.7, of 4096
// 16.5 -> 12, 100 tokens 19 -> 15.5; 8 and 128 tokens and 32 experts of 7168 34 -> 30, 36 -> 33. (1024 threads have 64 registers each: 16 bytes are spilled.)
constexpr int kGateSmallThreads = 1024;
template <int PER_LANE>
__global__ void __launch_bounds__(kGateSmallThreads) gate_route_kernel(const GateRouteArgs g, const SplitsArgs sp, unsigned int* ticket) {
  extern __shared__ __align__(16) int s_mem[];   // first the logits of the token and its row, later the entries' expert ids, their counts and the split scan's tables
  __shared__ int s_counts[256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = kGateSmallThreads / 32;
  grid_dependency_wait();
  launch_dependents();
  const int E = sp.num_experts, K = g.K, chunks = g.H / 8, t = blockIdx.x, T = gridDim.x;
  float* s_part = reinterpret_cast<float*>(s_mem);              // [parts][E]
  float4* s_x = reinterpret_cast<float4*>(s_mem + gate_route_parts_ints(E));   // first halves of the 8-element words, then second halves, as fp32
  const int parts = max(1, kWarps / E);                         // warps that share an expert's row
  const uint4* x = reinterpret_cast<const uint4*>(g.x + static_cast<long long>(t) * g.H);
  constexpr int U = 8;   // words of the gate in flight
  uint4 b[U];
  auto load = [&](int u, int c0) {
    const int e = u % E, c1 = chunks * (u / E + 1) / parts;
    const uint4* w = reinterpret_cast<const uint4*>(g.gate + static_cast<long long>(e) * g.H);
#pragma unroll
    for (int k = 0; k < U; ++k) b[k] = c0 + 32 * k < c1 ? __ldg(w + c0 + 32 * k) : make_uint4(0, 0, 0, 0);
  };
  auto begin = [&](int u) { return chunks * (u / E) / parts + lane; };
  if (warp < E * parts) load(warp, begin(warp));
  for (int i = threadIdx.x; i < chunks; i += kGateSmallThreads) {
    const uint4 a = __ldg(x + i);
    s_x[i] = make_float4(__uint_as_float(a.x << 16), __uint_as_float(a.x & 0xFFFF0000u), __uint_as_float(a.y << 16), __uint_as_float(a.y & 0xFFFF0000u));
    s_x[chunks + i] = make_float4(__uint_as_float(a.z << 16), __uint_as_float(a.z & 0xFFFF0000u), __uint_as_float(a.w << 16), __uint_as_float(a.w & 0xFFFF0000u));
  }
  __syncthreads();
  for (int u = warp; u < E * parts; u += kWarps) {
    const int e = u % E, part = u / E, c1 = chunks * (part + 1) / parts;
    float acc = 0.0f;
    for (int c0 = begin(u); c0 < c1; c0 += 32 * U) {
      if (u != warp || c0 != begin(u)) load(u, c0);
#pragma unroll
      for (int k = 0; k < U; ++k) {
        if (c0 + 32 * k >= c1) break;
        const float4 lo = s_x[c0 + 32 * k], hi = s_x[chunks + c0 + 32 * k];
        const float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        const uint32_t q[4] = {b[k].x, b[k].y, b[k].z, b[k].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc = fmaf(f[2 * i], __uint_as_float(q[i] << 16), acc);
          acc = fmaf(f[2 * i + 1], __uint_as_float(q[i] & 0xFFFF0000u), acc);
        }
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) s_part[part * E + e] = acc;
  }
  __syncthreads();
  int my_e = -1;
  if (warp == 0) {
    float sel[PER_LANE], raw[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      float r = -INFINITY, s = -INFINITY;
      if (e < E) {
        r = 0.0f;
        for (int j = 0; j < parts; ++j) r += s_part[j * E + e];
        r = __bfloat162float(__float2bfloat16_rn(r));
        if (r != r) r = -INFINITY;
        s = r + (g.bias ? g.bias[e] : 0.0f);
        if (s != s) s = -INFINITY;
      }
      raw[i] = r;
      sel[i] = s;
    }
    float my_w;
    route::warp_topk<PER_LANE>(sel, raw, E, K, my_e, my_w);
    if (lane < K) {
      g.topk_idx[static_cast<long long>(t) * K + lane] = my_e;
      g.topk_w[static_cast<long long>(t) * K + lane] = my_w;
    }
  }
  if (T == 1) {                                                 // nobody to meet, every chosen expert gets its first row
    for (int e = threadIdx.x; e < E; e += blockDim.x) s_counts[e] = 0;
    __syncthreads();
    if (warp == 0 && lane < K) { s_counts[my_e] = 1; g.slot_in_block[lane] = 0; }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) g.block_cnt[e] = s_counts[e];
  } else {
    if (!route::last_block(ticket)) return;
    const int entries = (T * K + 31) & ~31;                     // ranked 32 at a time, the rest of a routing block is not there
    for (int i = threadIdx.x; i < entries; i += blockDim.x) s_mem[i] = i < T * K ? __ldcg(g.topk_idx + i) : -1;
    __syncthreads();
    route::block_stable_ranks(s_mem, reinterpret_cast<unsigned short*>(s_mem + kTokensPerBlock * K), E, K, g.slot_in_block, g.block_cnt, entries / 32, s_counts);
    __syncthreads();
  }
  if (sp.world == 1 && sp.send_pos == nullptr) route::splits_alone(sp, s_counts);
  else route::splits_block(sp, s_mem, s_counts);
}

__global__ void build_send_list_kernel(const int* __restrict__ topk_idx, const int* __restrict__ slot_in_block, const int* __restrict__ block_base,
                                       const int* __restrict__ send_pos, int T, int K, int E, int* __restrict__ list, DeviceStatus* status) {
  const long long tj = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (tj >= static_cast<long long>(T) * K) return;
  const int e = topk_idx[tj];
  if (e < 0 || e >= E) {  // an id no router of this library produces: skip the entry, say so, touch nothing
    if (status) report_failure(status, kStatusBadArg, kSiteExpertId, static_cast<unsigned long long>(tj), static_cast<unsigned long long>(static_cast<unsigned int>(e)), static_cast<unsigned long long>(E));
    return;
  }
  const int t = static_cast<int>(tj / K);
  list[send_pos[e] + block_base[static_cast<long long>(t / kTokensPerBlock) * E + e] + slot_in_block[tj]] = static_cast<int>(tj);
}

// Zeroes the rows between each group's real end and its padded end, or the next multiple of `align` rows.
__global__ void zero_pad_rows_kernel(unsigned char* buf, long long row_bytes, const int* __restrict__ group_off, const int* __restrict__ group_rows, int groups, int align) {
  const int g = blockIdx.y;
  grid_dependency_wait();
  launch_dependents();
  if (g >= groups) return;
  const long long begin = (static_cast<long long>(group_off[g]) + group_rows[g]) * row_bytes;
  const long long last = align > 0 ? static_cast<long long>(group_off[g]) + (group_rows[g] + align - 1) / align * align : group_off[g + 1];
  const long long end = last * row_bytes;
  uint4* p = reinterpret_cast<uint4*>(buf + begin);
  const long long n = (end - begin) / 16;
  for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += static_cast<long long>(gridDim.x) * blockDim.x) p[i] = make_uint4(0, 0, 0, 0);
}

}  // namespace

namespace {

bool splits_args_ok(const SplitsArgs& a) {
  if (a.tile_target != nullptr && (a.tile_rows < 1 || a.row_align % a.tile_rows || a.num_tiles < 1)) return false;
  return (a.row_align == 128 || a.row_align == 256) && a.num_experts >= 1 && a.num_experts <= 1024 && a.world >= 1 && a.world <= a.num_experts && a.num_experts % a.world == 0;
}

template <bool SPLITS>
cudaError_t route_topk_any(const float* logits, const float* bias, int T, int E, int K, int* topk_idx, float* topk_w, int* slot_in_block, int* block_cnt,
                           const SplitsArgs& sp, unsigned int* ticket, cudaStream_t stream) {
  if (E < 1 || E > 256 || K < 1 || K > 32 || K > E) return cudaErrorInvalidValue;
  const int blocks = (T + kTokensPerBlock - 1) / kTokensPerBlock;
  if (blocks == 0) return cudaSuccess;
  const size_t smem = std::max(route::rank_smem_bytes(E, K), SPLITS ? route::splits_smem_bytes(sp.world, E) : size_t{0});
  auto go = [&](auto kern) {
    cudaError_t e = allow_smem(kern, smem);
    if (e == cudaSuccess) e = launch_early(kern, dim3(blocks), kRouteThreads, smem, stream, logits, bias, T, E, K, topk_idx, topk_w, slot_in_block, block_cnt, sp, ticket);
    if (e == cudaSuccess) note_launch();
    return e;
  };
  if (E <= 32) return go(route_topk_kernel<1, SPLITS>);
  if (E <= 64) return go(route_topk_kernel<2, SPLITS>);
  if (E <= 128) return go(route_topk_kernel<4, SPLITS>);
  return go(route_topk_kernel<8, SPLITS>);
}

}  // namespace

cudaError_t launch_route_topk(const float* logits, const float* bias, int T, int E, int K, int* topk_idx, float* topk_w, int* slot_in_block,
                              int* block_cnt, cudaStream_t stream) {
  return route_topk_any<false>(logits, bias, T, E, K, topk_idx, topk_w, slot_in_block, block_cnt, SplitsArgs{}, nullptr, stream);
}

cudaError_t launch_route_splits(const float* logits, const float* bias, int T, int K, int* topk_idx, float* topk_w, int* slot_in_block, const SplitsArgs& sp,
                                unsigned int* ticket, cudaStream_t stream) {
  if (T < 1 || ticket == nullptr || !splits_args_ok(sp) || sp.num_blocks != (T + kTokensPerBlock - 1) / kTokensPerBlock) return cudaErrorInvalidValue;
  return route_topk_any<true>(logits, bias, T, sp.num_experts, K, topk_idx, topk_w, slot_in_block, const_cast<int*>(sp.block_cnt), sp, ticket, stream);
}

static size_t gate_route_smem_bytes(int world, int E, int K, int H) {
  return std::max({route::rank_smem_bytes(E, K), route::splits_smem_bytes(world, E), sizeof(int) * gate_route_parts_ints(E) + sizeof(float) * static_cast<size_t>(H)});
}
bool gate_route_fits(int world, int E, int K, int H) { return gate_route_smem_bytes(world, E, K, H) <= 225 * 1024; }   // of 227 KiB; the rest is static

cudaError_t launch_gate_route(const GateRouteArgs& g, const SplitsArgs& sp, unsigned int* ticket, cudaStream_t stream) {
  const int E = sp.num_experts;
  if (g.T < 1 || g.T > kTokensPerBlock || E > 256 || g.K < 1 || g.K > 32 || g.K > E || g.H % 8 || ticket == nullptr || !splits_args_ok(sp) || sp.num_blocks != 1) return cudaErrorInvalidValue;
  if (!gate_route_fits(sp.world, E, g.K, g.H)) return cudaErrorInvalidValue;
  const size_t smem = gate_route_smem_bytes(sp.world, E, g.K, g.H);
  auto go = [&](auto kern) {
    cudaError_t e = allow_smem(kern, smem);
    if (e == cudaSuccess) e = launch_early(kern, dim3(g.T), kGateSmallThreads, smem, stream, g, sp, ticket);
    if (e == cudaSuccess) note_launch();
    return e;
  };
  return E <= 32 ? go(gate_route_kernel<1>) : E <= 64 ? go(gate_route_kernel<2>) : go(gate_route_kernel<8>);
}

cudaError_t launch_splits_scan(const SplitsArgs& a, cudaStream_t stream) {
  if (!splits_args_ok(a)) return cudaErrorInvalidValue;
  // a thread per expert at least; more warps take experts and routing blocks in parallel
  const int threads = std::max(256, (std::max(a.num_experts, a.world) + 31) / 32 * 32);
  splits_scan_kernel<<<1, threads, route::splits_smem_bytes(a.world, a.num_experts), stream>>>(a);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_build_send_list(const int* topk_idx, const int* slot_in_block, const int* block_base, const int* send_pos, int T, int K, int E,
                                   int* list, DeviceStatus* status, cudaStream_t stream) {
  const long long n = static_cast<long long>(T) * K;
  if (n == 0) return cudaSuccess;
  build_send_list_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(topk_idx, slot_in_block, block_base, send_pos, T, K, E, list, status);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_zero_pad_rows(void* buf, long long row_bytes, const int* group_off, const int* group_rows, int groups, int align, cudaStream_t stream) {
  if (row_bytes % 16 || align < 0) return cudaErrorInvalidValue;
  if (groups == 0) return cudaSuccess;
  const cudaError_t e = launch_early(zero_pad_rows_kernel, dim3(8, groups), 256, 0, stream, static_cast<unsigned char*>(buf), row_bytes, group_off, group_rows, groups, align);
  note_launch();
  return e;
}

}  // namespace fastb

// ---------------------------------------------------------------------------------------------
// Allocation-free entry point (declared in route_noalloc.h).
// ---------------------------------------------------------------------------------------------
#include <atomic>
#include <cstdio>

#include "route_noalloc.h"

namespace fastb {
namespace {

constexpr int kNoAllocMaxTokens = 16384, kNoAllocMaxExperts = 256, kNoAllocMaxTopK = 8;
constexpr int kNoAllocMaxBlocks = kNoAllocMaxTokens / kRouteTokensPerBlock;
constexpr size_t kNoAllocCntBytes = sizeof(int) * kNoAllocMaxBlocks * kNoAllocMaxExperts;    // per-block histograms
constexpr size_t kNoAllocSlotBytes = sizeof(int) * kNoAllocMaxTokens * kNoAllocMaxTopK;       // in-block ranks
constexpr size_t kNoAllocBytes = kNoAllocCntBytes + kNoAllocSlotBytes;                        // 640 KiB

// Scratch of the allocation-free entry point. In host code this name is only a handle for
// cudaGetSymbolAddress; kernels receive the device address obtained from it.
static __device__ __align__(256) unsigned char g_route_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
// One address per device, filled by the first call on that device. Atomic: several host threads
// may make that first call at once (they would all store the same value).
std::atomic<void*> g_scratch_addr[kMaxDevices] = {};
thread_local char g_noalloc_error[256] = "";

__global__ void sum_block_counts_kernel(const int* __restrict__ block_cnt, int blocks, int E, int* __restrict__ expert_counts) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  int s = 0;
  for (int b = 0; b < blocks; ++b) s += block_cnt[static_cast<long long>(b) * E + e];
  expert_counts[e] = s;
}

int refuse(cudaError_t code, const char* fmt, int a = 0, int b = 0) {
  snprintf(g_noalloc_error, sizeof(g_noalloc_error), fmt, a, b);
  return static_cast<int>(code);
}

}  // namespace
}  // namespace fastb

extern "C" void fastb_route_topk_noalloc_limits(int* max_tokens, int* max_experts, int* max_top_k) {
  if (max_tokens) *max_tokens = fastb::kNoAllocMaxTokens;
  if (max_experts) *max_experts = fastb::kNoAllocMaxExperts;
  if (max_top_k) *max_top_k = fastb::kNoAllocMaxTopK;
}

extern "C" const char* fastb_noalloc_last_error(void) { return fastb::g_noalloc_error; }

extern "C" int fastb_route_topk_noalloc(const float* logits, const float* bias, int T, int E, int K, int* topk_idx, float* topk_w,
                                        int* expert_counts, void* stream_v) {
  using namespace fastb;
  g_noalloc_error[0] = '\0';
  if (!logits || !topk_idx || !topk_w || !expert_counts) return refuse(cudaErrorInvalidValue, "fastb_route_topk_noalloc: null buffer");
  if (T < 0 || T > kNoAllocMaxTokens) return refuse(cudaErrorInvalidValue, "fastb_route_topk_noalloc: %d tokens exceed the fixed scratch (max %d)", T, kNoAllocMaxTokens);
  if (E < 1 || E > kNoAllocMaxExperts) return refuse(cudaErrorInvalidValue, "fastb_route_topk_noalloc: %d experts exceed the fixed scratch (max %d)", E, kNoAllocMaxExperts);
  if (K < 1 || K > kNoAllocMaxTopK || K > E) return refuse(cudaErrorInvalidValue, "fastb_route_topk_noalloc: top-%d is outside 1..min(%d, experts)", K, kNoAllocMaxTopK);
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return refuse(e, "fastb_route_topk_noalloc: cudaGetDevice failed");
  if (dev < 0 || dev >= kMaxDevices) return refuse(cudaErrorInvalidDevice, "fastb_route_topk_noalloc: device index %d not supported (max %d)", dev, kMaxDevices - 1);
  void* scratch = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    // Once per device, with that device current: translate the symbol into its device address.
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_route_scratch);
    if (e != cudaSuccess || p == nullptr) return refuse(e != cudaSuccess ? e : cudaErrorInvalidSymbol, "fastb_route_topk_noalloc: cudaGetSymbolAddress failed");
    g_scratch_addr[dev].store(p, std::memory_order_release);
    scratch = p;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  const int blocks = (T + kRouteTokensPerBlock - 1) / kRouteTokensPerBlock;
  int* block_cnt = reinterpret_cast<int*>(static_cast<unsigned char*>(scratch));
  int* slot_in_block = reinterpret_cast<int*>(static_cast<unsigned char*>(scratch) + kNoAllocCntBytes);
  if (blocks > 0) {
    e = launch_route_topk(logits, bias, T, E, K, topk_idx, topk_w, slot_in_block, block_cnt, stream);
    if (e != cudaSuccess) return refuse(e, "fastb_route_topk_noalloc: routing kernel launch failed");
  }
  sum_block_counts_kernel<<<(E + 127) / 128, 128, 0, stream>>>(block_cnt, blocks, E, expert_counts);
  e = cudaGetLastError();
  if (e != cudaSuccess) return refuse(e, "fastb_route_topk_noalloc: count kernel launch failed");
  note_launch();
  return 0;
}
