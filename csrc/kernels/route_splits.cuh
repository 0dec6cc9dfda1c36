// The split scan of one block of threads: block histograms -> per-expert send counts, all-gather of the counts by direct
// stores into every peer's symmetric pad, then receive offsets, padded group offsets for the grouped GEMM and cumulative
// arrival targets. It runs as a kernel of its own or, one launch less, in the last block of a routing kernel.
// Bound by latency (one block, dependent steps): sums over experts and routing blocks are warp scans, 32 at a time (one
// thread per expert summing 256 routing blocks took 43 us at 32768 tokens), and a single rank skips the exchange.
#pragma once
#include "api.h"

namespace fastb {
namespace route {

// ints of shared memory: my counts, padded totals and first rows per expert, and the count matrix when it fits.
__host__ __device__ constexpr bool splits_matrix_fits(int world, int E) { return static_cast<long long>(world) * E <= 8192; }
__host__ __device__ constexpr size_t splits_smem_bytes(int world, int E) { return sizeof(int) * (3 * static_cast<size_t>(E) + (splits_matrix_fits(world, E) ? static_cast<size_t>(world) * E : 0)); }

__device__ __forceinline__ int warp_incl_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += y; }
  return v;
}
__device__ __forceinline__ int warp_total(int v) { return static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(v))); }

// True in the block that is the last of the grid to get here (everything the others wrote before is visible to it then).
// The ticket is back at zero afterwards.
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) { __threadfence(); s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1; __threadfence(); }
  __syncthreads();
  return s_last != 0;
}

// Every thread of the block calls this; blockDim.x is a multiple of 32 and at least max(E, world) threads are there.
// s_only: counts of the one routing block there is, in shared memory (not where this function works); null: read from a.block_cnt.
__device__ __forceinline__ void splits_block(const SplitsArgs& a, int* s_mine, const int* s_only = nullptr) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int E = a.num_experts, W = a.world, El = E / W;
  int* s_tot = s_mine + E;    // rows of each expert over all ranks, padded
  int* s_base = s_tot + E;    // first row of each expert on its owner
  int* s_cnt = s_base + E;    // [W][E] when it fits
  const bool in_smem = splits_matrix_fits(W, E);
  unsigned char* my_slab = static_cast<unsigned char*>(a.peer_table[a.rank]);
  int* my_counts = reinterpret_cast<int*>(my_slab + a.counts_heap_off);                       // [W][E]
  unsigned long long* my_flags = reinterpret_cast<unsigned long long*>(my_slab + a.flags_heap_off);  // [W]
  __shared__ unsigned long long s_epoch;
  __shared__ int s_ok, s_over;
  if (tid == 0) {
    if (W == 1 && a.epoch_dev) atomicAdd(a.epoch_dev, 1ull);   // nobody here needs its value
    else s_epoch = a.epoch_dev ? (*a.epoch_dev = *a.epoch_dev + 1ull) : a.epoch;
    s_ok = 1;
    s_over = 0;
  }
  // A warp per expert: running sum over the routing blocks, 128 of them requested at a time. The counts may come from
  // other blocks of this very launch: read past L1.
  if (s_only != nullptr) {
    for (int e = tid; e < E; e += blockDim.x) { s_mine[e] = s_only[e]; a.block_base[e] = 0; }
  } else
  for (int e = warp; e < E; e += nwarps) {
    int run = 0;
    for (int b0 = 0; b0 < a.num_blocks; b0 += 128) {
      int c[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) c[u] = b0 + 32 * u + lane < a.num_blocks ? __ldcg(a.block_cnt + static_cast<long long>(b0 + 32 * u + lane) * E + e) : 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (b0 + 32 * u >= a.num_blocks) break;
        const int incl = warp_incl_scan(c[u]);
        if (b0 + 32 * u + lane < a.num_blocks) a.block_base[static_cast<long long>(b0 + 32 * u + lane) * E + e] = run + incl - c[u];
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    if (lane == 0) s_mine[e] = run;
  }
  __syncthreads();
  if (W > 1) {
    // All-gather by stores: my row of the count matrix goes to every rank (myself included).
    for (int i = tid; i < W * E; i += blockDim.x) reinterpret_cast<int*>(static_cast<unsigned char*>(a.peer_table[i / E]) + a.counts_heap_off)[a.rank * E + i % E] = s_mine[i % E];
    __threadfence_system();
    __syncthreads();
    if (tid < W) {
      unsigned long long* dst = reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(a.peer_table[tid]) + a.flags_heap_off);
      st_release_sys(dst + a.rank, s_epoch);
      if (!wait_ge_bounded(my_flags + tid, s_epoch, a.status, kSiteCountsArrive, tid, a.timeout_ns)) s_ok = 0;
    }
    __syncthreads();
    if (!s_ok) return;
    if (in_smem) {
      for (int i = tid; i < W * E; i += blockDim.x) s_cnt[i] = *reinterpret_cast<volatile int*>(my_counts + i);
      __syncthreads();
    }
  }
  auto count_at = [&](int src, int q) { return W == 1 ? s_mine[q] : in_smem ? s_cnt[src * E + q] : *reinterpret_cast<volatile int*>(my_counts + src * E + q); };
  const int e = tid;
  int tot = 0, before_me = 0;
  if (e < E) {
    for (int s = 0; s < W; ++s) {
      const int c = count_at(s, e);
      tot += c;
      if (s < a.rank) before_me += c;
    }
    s_tot[e] = (tot + a.row_align - 1) / a.row_align * a.row_align;
  }
  __syncthreads();
  // First rows: padded sizes of the owner's earlier experts. Every rank sees the same count matrix, so every rank reaches the
  // same verdict: if any rank's padded rows exceed the receive capacity, the step is refused everywhere (no rows are sent,
  // the GEMMs get empty groups) and the status block says how many rows were needed.
  for (int d = warp; d < W; d += nwarps) {
    int run = 0;
    for (int q0 = 0; q0 < El; q0 += 32) {
      const int v = q0 + lane < El ? s_tot[d * El + q0 + lane] : 0;
      const int incl = warp_incl_scan(v);
      if (q0 + lane < El) s_base[d * El + q0 + lane] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0 && run > a.cap_rows) atomicMax(&s_over, run);
  }
  __syncthreads();
  if (s_over) {
    if (tid == 0) report_failure(a.status, kStatusBadArg, kSiteCapacity, a.rank, static_cast<unsigned long long>(s_over), static_cast<unsigned long long>(a.cap_rows));
    if (e < E) { a.send_base[e] = 0; a.send_cnt[e] = 0; }
    if (e <= El) a.group_off[e] = 0;
    if (e < El) a.group_rows[e] = 0;
    return;
  }
  if (e < E) {
    // Row where my first token for expert e lands on its owner: the expert's first row there plus the rows of lower-ranked sources.
    const int d = e / El, le = e % El, base = s_base[e];
    a.send_base[e] = base + before_me;
    a.send_cnt[e] = s_mine[e];
    if (a.send_pos) {
      // Entries are sent expert-slot by expert-slot: all ranks' local expert 0, then 1, ... Within a
      // slot every sender starts with itself and walks the ranks upwards, so that at any moment the
      // senders aim at different receivers.
      int pos = 0;
      for (int q = 0; q < E; ++q) {
        const int key_q = (q % El) * W + (q / El - a.rank + W) % W, key_e = le * W + (d - a.rank + W) % W;
        if (key_q < key_e) pos += s_mine[q];
      }
      a.send_pos[e] = pos;
    }
    if (d == a.rank) {
      a.group_off[le] = base;
      a.group_rows[le] = tot;
      if (le == El - 1) a.group_off[El] = base + s_tot[e];
      // Monotone arrival targets, one per channel (forward dispatch, backward dispatch).
      // (Additions that return nothing: no step of this chain waits for the words to come back.)
      for (int ch = 0; ch < a.num_channels; ++ch) atomicAdd(a.arrive_target + ch * El + le, static_cast<unsigned long long>(tot));
    }
  }
  if (a.tile_target != nullptr) {
    // The same per tile of the receive buffer: an expert's rows fill its tiles from its first row on (a warp per expert).
    for (int le = warp; le < El; le += nwarps) {
      const int q = a.rank * El + le, base = s_base[q];
      int rows = 0;
      for (int s = 0; s < W; ++s) rows += count_at(s, q);
      for (int r0 = lane * a.tile_rows; r0 < rows; r0 += 32 * a.tile_rows) {
        const int t = (base + r0) / a.tile_rows;
        if (t >= a.num_tiles) break;
        const unsigned long long n = static_cast<unsigned long long>(min(a.tile_rows, rows - r0));
        for (int ch = 0; ch < a.num_channels; ++ch) atomicAdd(a.tile_target + static_cast<long long>(ch) * a.num_tiles + t, n);
      }
    }
  }
  // Token traffic matrix of this step, [src][dst], for the scheduler / observability (a warp per entry).
  if (a.traffic_matrix)
    for (int i = warp; i < W * W; i += nwarps) {
      int sent = 0;
      for (int q = lane; q < El; q += 32) sent += count_at(i / W, (i % W) * El + q);
      sent = warp_total(sent);
      if (lane == 0) a.traffic_matrix[i] = sent;
    }
}

// The same for a rank that is alone, with the counts of its one routing block in shared memory and no send list to place: one warp, straight
// through. What splits_block does besides (exchange, other ranks' rows, several routing blocks) is code that a kernel of few tokens
// fetches and steps over: 5500 to 6000 cycles from the ranks to the end, so 3000 to 3700.
__device__ __forceinline__ void splits_alone(const SplitsArgs& a, const int* s_only) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x, E = a.num_experts;
  int padded_rows = 0, sent = 0;
  for (int e = lane; e < E; e += 32) {
    padded_rows += (s_only[e] + a.row_align - 1) / a.row_align * a.row_align;
    sent += s_only[e];
  }
  padded_rows = warp_total(padded_rows);
  sent = warp_total(sent);
  const bool over = padded_rows > a.cap_rows;
  if (lane == 0) {
    if (a.epoch_dev) atomicAdd(a.epoch_dev, 1ull);
    if (over) report_failure(a.status, kStatusBadArg, kSiteCapacity, a.rank, static_cast<unsigned long long>(padded_rows), static_cast<unsigned long long>(a.cap_rows));
    a.group_off[E] = over ? 0 : padded_rows;
    if (a.traffic_matrix && !over) a.traffic_matrix[0] = sent;
  }
  int run = 0;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int e = e0 + lane, rows = e < E && !over ? s_only[e] : 0, padded = (rows + a.row_align - 1) / a.row_align * a.row_align;
    const int incl = warp_incl_scan(padded), base = run + incl - padded;
    run += __shfl_sync(0xffffffffu, incl, 31);
    if (e >= E) continue;
    a.block_base[e] = 0;
    a.send_base[e] = base; a.send_cnt[e] = rows;
    a.group_off[e] = base; a.group_rows[e] = rows;
    if (rows == 0) continue;
    for (int ch = 0; ch < a.num_channels; ++ch) {
      atomicAdd(a.arrive_target + ch * E + e, static_cast<unsigned long long>(rows));
      if (a.tile_target != nullptr)
        for (int r0 = 0, t = base / a.tile_rows; r0 < rows && t < a.num_tiles; r0 += a.tile_rows, ++t)
          atomicAdd(a.tile_target + static_cast<long long>(ch) * a.num_tiles + t, static_cast<unsigned long long>(min(a.tile_rows, rows - r0)));
    }
  }
}

}  // namespace route
}  // namespace fastb
