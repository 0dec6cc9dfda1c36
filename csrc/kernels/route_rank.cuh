// Pieces shared by the routing kernels: the expert choice of one token by a warp, and the stable rank of every
// (token, slot) entry of a routing block among the block's entries for the same expert.
#pragma once
#include "api.h"

namespace fastb {
namespace route {

constexpr int kTokensPerBlock = kRouteTokensPerBlock;

// Shared memory of block_stable_ranks behind the entries' expert ids: a 16-bit count per (32 entries, expert).
__host__ __device__ constexpr size_t rank_smem_bytes(int E, int K) {
  return sizeof(int) * kTokensPerBlock * K + sizeof(unsigned short) * (kTokensPerBlock * K / 32) * static_cast<size_t>((E + 1) & ~1);
}

// s_eid[n] (n = kTokensPerBlock * K; ids, -1 for tokens past the end) -> slot_in_block[n] and block_cnt[E], called by the whole
// block after the ids are in place. A warp takes 32 entries at a time and finds equal ids with match_any; counts per
// 32 entries are then summed up by one thread per expert. One thread per expert walking all n entries took
// 60 us at top-8 of 32 experts (1024 dependent steps); this takes about 2 us.
// used: how many groups of 32 entries there are (the others hold -1); s_cnt: the counts in shared memory too.
__device__ __forceinline__ void block_stable_ranks(const int* s_eid, unsigned short* s_hist, int E, int K, int* __restrict__ slot_in_block, int* __restrict__ block_cnt,
                                                   int used = 1 << 30, int* s_cnt = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int groups = min(kTokensPerBlock * K / 32, used), pitch = (E + 1) & ~1;
  for (int i = threadIdx.x; i < groups * pitch / 2; i += blockDim.x) reinterpret_cast<unsigned int*>(s_hist)[i] = 0u;
  __syncthreads();
  for (int g = warp; g < groups; g += nwarps) {
    const int e = s_eid[g * 32 + lane];
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e >= 0 && lane == __ffs(same) - 1) s_hist[g * pitch + e] = static_cast<unsigned short>(__popc(same));
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = 0;
    for (int g = 0; g < groups; ++g) {
      const int c = s_hist[g * pitch + e];
      s_hist[g * pitch + e] = static_cast<unsigned short>(run);
      run += c;
    }
    block_cnt[e] = run;
    if (s_cnt != nullptr) s_cnt[e] = run;
  }
  __syncthreads();
  for (int g = warp; g < groups; g += nwarps) {
    const int e = s_eid[g * 32 + lane];
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e >= 0) slot_in_block[g * 32 + lane] = s_hist[g * pitch + e] + __popc(same & ((1u << lane) - 1u));
  }
}

// Floats as unsigned integers of the same order; both zeros give the same key. 0 is below every key.
__device__ __forceinline__ unsigned order_key(float x) {
  const unsigned b = x == 0.0f ? 0u : __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}

// The warp chooses the K largest of E selection values (value of expert lane + 32 i in sel[i]; NaN and values past E are given
// as -inf / taken) and the softmax of the raw logits over them, renormalised. Lane j < K leaves with choice j.
// The selection is total: equal values go to the lower id, and a token with fewer than K selectable values still gets K
// distinct ids in range, the lowest unchosen ones, with weight 0.
template <int PER_LANE>
__device__ __forceinline__ void warp_topk(const float (&sel)[PER_LANE], const float (&raw)[PER_LANE], int E, int K, int& my_e, float& my_w) {
  const int lane = threadIdx.x & 31;
  unsigned key[PER_LANE];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    key[i] = lane + 32 * i < E ? order_key(sel[i]) : 0u;
    mx = fmaxf(mx, raw[i]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float wsum = 0.0f;
  my_w = 0.0f;
  my_e = -1;
  for (int j = 0; j < K; ++j) {
    unsigned best = key[0];
    int id = lane;
#pragma unroll
    for (int i = 1; i < PER_LANE; ++i)
      if (key[i] > best) { best = key[i]; id = lane + 32 * i; }
    const unsigned top = __reduce_max_sync(0xffffffffu, best);
    const int e = static_cast<int>(__reduce_min_sync(0xffffffffu, best == top ? static_cast<unsigned>(id) : 0x7fffffffu));
    float r = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (lane + 32 * i == e) { r = raw[i]; key[i] = 0u; }
    r = __shfl_sync(0xffffffffu, r, e & 31);
    const float p = r > -INFINITY ? __expf(r - mx) : 0.0f;
    wsum += p;
    if (lane == j) { my_w = p; my_e = e; }
  }
  my_w = wsum > 0.0f ? my_w / wsum : 0.0f;
}

}  // namespace route
}  // namespace fastb
