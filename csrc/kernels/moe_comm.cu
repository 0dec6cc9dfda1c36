// Fused MoE transport kernels over peer memory (NVLink P2P loads/stores issued inside the kernel):
//   dispatch_push : gather token rows by routing index, optional per-row scale, optional e4m3
//                   quantisation with 1x128 block scales, and store them straight into the final
//                   row of the owning expert's receive buffer on the peer; per-expert arrival
//                   counters are bumped with release semantics once a CTA's rows are out.
//   combine_pull  : un-permute + top-k weighted reduction: every token pulls its k expert rows
//                   from the peers and accumulates them in fp32 (fixed slot order => reproducible).
// In FAST's terms these are the all-to-all of the forward pass and its transpose
// (amd/flash.cpp:400-408 `backward` flag) with the permute / reduce fused in; the reference moves
// opaque bytes with ncclSend/ncclRecv groups or NVSHMEM puts and leaves the packing to the caller.
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>

#include "announce_blocks.h"
#include "api.h"
#include "early_start.cuh"
#include "route_splits.cuh"

namespace fastb {

namespace {

constexpr int kCommThreads = 256;

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v;
}

__device__ __forceinline__ uint4 add8(const uint4& a, const uint4& b) {
  uint4 v;
  const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162*>(&a), *y = reinterpret_cast<const __nv_bfloat162*>(&b);
  __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = __hadd2_rn(x[i], y[i]);
  return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int kMaxK = 8;
constexpr int kMaxScaleGroups = 128;  // fp8 dispatch: rows of up to 128 x 128 = 16384 elements

// 16 bf16 elements of a lane -> 16 e4m3 bytes; 8 consecutive lanes (128 elements) share one scale.
// Every lane of the warp calls this together (lanes past the row's end pass zeros).
// The scale is amax / 448 rounded UP to the next value a bf16 can hold: quantised values still fit
// e4m3, and a receiver that multiplies in bf16 (the expert GEMM's converter warps) reproduces
// value x scale without a second rounding. The abs / max run on bf16 pairs, the conversion on float pairs.
__device__ __forceinline__ uint4 quantise16(const uint4 (&raw)[2], float& sc) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[0]);  // 8 pairs = my 16 elements
  __nv_bfloat162 m2 = __habs2(h[0]);
#pragma unroll
  for (int i = 1; i < 8; ++i) m2 = __hmax2(m2, __habs2(h[i]));
  float amax = fmaxf(__low2float(m2), __high2float(m2));
#pragma unroll
  for (int o = 4; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  sc = __uint_as_float((__float_as_uint(fmaxf(amax, 1e-12f) * (1.0f / 448.0f)) + 0xFFFFu) & 0xFFFF0000u);
  const float inv = 1.0f / sc;
  uint4 q;
  unsigned short* qs = reinterpret_cast<unsigned short*>(&q);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    qs[i] = __nv_cvt_float2_to_fp8x2(make_float2(f.x * inv, f.y * inv), __NV_SATFINITE, __NV_E4M3);
  }
  return q;
}

// 8 bf16 elements of a lane (16 consecutive lanes = 128 elements share a scale) -> what a receiver makes of their e4m3 values:
// quantised as in quantise16, multiplied back in fp32 as dequant_fp8_kernel does, rounded to bf16.
__device__ __forceinline__ uint4 through_e4m3(const uint4& raw) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  __nv_bfloat162 m2 = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
  float amax = fmaxf(__low2float(m2), __high2float(m2));
#pragma unroll
  for (int o = 8; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float sc = __uint_as_float((__float_as_uint(fmaxf(amax, 1e-12f) * (1.0f / 448.0f)) + 0xFFFFu) & 0xFFFF0000u), inv = 1.0f / sc;
  float f[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h[i]);
    const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(__nv_cvt_float2_to_fp8x2(make_float2(v.x * inv, v.y * inv), __NV_SATFINITE, __NV_E4M3), __NV_E4M3);
    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&r));
    f[2 * i] = d.x * sc;
    f[2 * i + 1] = d.y * sc;
  }
  return pack8(f);
}

// One warp per row: x [T, H] bf16 -> q [T, H] e4m3 bytes + scales [T, H / 128], in this GPU's own memory.
// The sorted dispatch sends every (token, slot) entry from a warp of its own; with the rows quantised
// here first, a token's K entries copy bytes instead of each repeating the reduction and the conversions.
__global__ void __launch_bounds__(kCommThreads) quantise_rows_kernel(const __nv_bfloat16* __restrict__ x, int T, int H, unsigned char* __restrict__ q,
                                                                      float* __restrict__ scales) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int chunks16 = H / 16, sgroups = H / 128;
  for (long long t = blockIdx.x * wpb + warp; t < T; t += static_cast<long long>(gridDim.x) * wpb) {
    const uint4* src = reinterpret_cast<const uint4*>(x + t * H);
    uint4* out = reinterpret_cast<uint4*>(q + t * H);
    constexpr int U = 2;
    for (int c0 = 0; c0 < chunks16; c0 += 32 * U) {
      uint4 raw[U][2];
      bool active[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + 32 * u + lane;
        active[u] = c < chunks16;
        raw[u][0] = active[u] ? __ldg(src + 2 * c) : make_uint4(0, 0, 0, 0);
        raw[u][1] = active[u] ? __ldg(src + 2 * c + 1) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (c0 + 32 * u >= chunks16) break;  // warp-uniform
        const int c = c0 + 32 * u + lane;
        float sc;
        const uint4 v = quantise16(raw[u], sc);
        if (active[u]) {
          out[c] = v;
          if ((lane & 7) == 0) scales[t * sgroups + c / 8] = sc;
        }
      }
    }
  }
}

// FP8: rows leave as e4m3 + scales; SORTED: one warp per (token, slot) entry of send_list (one destination per warp, so the
// per-slot arrays shrink to one element); SCALED: bf16 rows are multiplied by row_scale on the way. The variants exist for
// their register counts: the copy loops are bound by the stores a SM keeps in flight, i.e. by resident warps.
// ROUNDED (one rank alone): nothing crosses a wire, so the rows go straight to the GEMM's bf16 operand, as the values that a
// receiver would make of their e4m3 form. Sent as e4m3 and converted afterwards, 32768 rows of 7168 took 85 + 145 us.
// DOT (backward): the row on its way out (w * grad) meets the expert's output row that lies at the same place of the owner's
// forward buffer, and their product is the gradient of w: one reading of the gradient rows serves both. With a.sum_with
// the gradient itself is made here, from the two terms whose mean square is the loss.
// KM: most destinations of a token, K <= KM (2 or 8): with 2 the rows of all of them are requested at once, and no empty slots
// are walked.
template <bool FP8, bool SORTED, bool SCALED, bool ROUNDED = false, bool DOT = false, int KM = kMaxK>
__global__ void __launch_bounds__(kCommThreads, DOT ? (KM <= 2 ? 3 : 2) : SORTED || KM <= 2 ? 4 : 3) dispatch_push_kernel(const DispatchArgs a) {
  extern __shared__ int s_cnt[];  // rows this CTA sent: [E] per expert, or [world][num_tiles] per destination tile
  __shared__ int s_ok;
  __shared__ __align__(16) float s_scales[(kCommThreads / 32) * kMaxScaleGroups];  // fp8 mode: the 1x128 scales of the row each warp is sending
  grid_dependency_wait();
  launch_dependents();
  __shared__ float s_dot[DOT ? kCommThreads / 32 : 1][kMaxK];
  const float gscale = DOT && a.sum_with != nullptr ? *a.grad_loss * a.grad_factor : 0.0f;
  const int E = a.num_experts, El = E / a.world;
  const int n_cnt = a.tile_rows > 0 ? a.world * a.num_tiles : E;
  const bool counted = a.arrive_heap_off >= 0;   // somebody waits for the rows while this kernel runs
  if (counted)
    for (int e = threadIdx.x; e < n_cnt; e += blockDim.x) s_cnt[e] = 0;
  if (threadIdx.x == 0) s_ok = 1;
  if (*reinterpret_cast<volatile unsigned long long*>(&a.status->abort) != 0ull) return;  // an earlier kernel of this rank refused the step
  __syncthreads();
  if (a.entry_epoch != 0 && a.world > 1) {
    // Entry handshake: publish that my receive buffers may be written, then wait for the peers.
    unsigned long long* my_flags = reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(a.peer_table[a.rank]) + a.entry_flags_heap_off);
    if (blockIdx.x == 0 && threadIdx.x < a.world) {
      unsigned long long* dst = reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(a.peer_table[threadIdx.x]) + a.entry_flags_heap_off);
      st_release_sys(dst + a.rank, a.entry_epoch);
    }
    if (threadIdx.x < a.world && !wait_ge_bounded(my_flags + threadIdx.x, a.entry_epoch, a.status, kSiteEntryReady, threadIdx.x, a.timeout_ns)) s_ok = 0;
    __syncthreads();
    if (!s_ok) return;
  }
  // a.warps_per_row warps of a CTA share a row (1, or all of them when there are fewer rows than CTAs: a few rows of 4096 took one
  // warp each through 16 dependent rounds). Warp `part` of them takes the rounds [part, part + 1) / warps_per_row.
  const int lane = threadIdx.x & 31, wpr = SORTED ? 1 : a.warps_per_row, wpb = (blockDim.x >> 5) / wpr;
  const int warp = (threadIdx.x >> 5) / wpr, part = (threadIdx.x >> 5) % wpr;
  const bool first = lane == 0 && part == 0;
  constexpr int tpb = kRouteTokensPerBlock;
  const int chunks = a.H / 8;  // 16-byte chunks per row
  // Unsorted mode: one warp (or warps_per_row) per token, the row is read once and stored to its K destinations.
  // Sorted mode (send_list != null): one warp per (token, slot) entry, entries ordered by
  // (local expert index, destination rank counted from the sender upwards), so that every rank's expert 0 fills first, then
  // expert 1, ... and the gated GEMM of the receivers can start while later experts still arrive.
  constexpr int NJ = SORTED ? 1 : KM;  // destinations one warp serves
  const long long n_work = SORTED ? static_cast<long long>(a.T) * a.K : a.T;
  // Adds this CTA's row counts to the receivers' arrival counters (release: the rows are stored before the counters move)
  // and clears them. Called by every thread of the CTA.
  auto publish_counts = [&]() {
    __syncthreads();  // every row of this CTA so far is stored
    for (int e = threadIdx.x; e < n_cnt; e += blockDim.x) {
      const int n = s_cnt[e];
      if (n == 0) continue;
      s_cnt[e] = 0;
      const int peer = a.tile_rows > 0 ? e / a.num_tiles : e / El;
      const int slot = a.tile_rows > 0 ? e % a.num_tiles : e % El;
      unsigned long long* cnt = reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(a.peer_table[peer]) + a.arrive_heap_off);
      fence_sys();
      red_add_release_sys(cnt + slot, static_cast<unsigned long long>(n));
    }
    __syncthreads();  // cleared before the next rows are counted
  };
  // Every warp of a CTA makes the same number of rounds (a round = one entry per warp), so the CTA can meet at a barrier
  // between rounds. In sorted order the counts are published every kPublishRounds rounds instead of once at the end:
  // the CTAs walk the send list together, so a receiver's tiles complete in list order while the dispatch is still
  // running, which is what lets its gated GEMM start early.
  constexpr int kPublishRounds = 8;
  const long long round_stride = static_cast<long long>(gridDim.x) * wpb;
  int round = 0;
  for (long long base = static_cast<long long>(blockIdx.x) * wpb; base < n_work; base += round_stride) {
    const long long wi = base + warp;
    if (wi < n_work) {
      int t, jbeg, nj;
      if (SORTED) { const int tj = a.send_list[wi]; t = tj / a.K; jbeg = tj % a.K; nj = 1; }
      else { t = static_cast<int>(wi); jbeg = 0; nj = a.K; }
      unsigned char* out_row[NJ];  // where each slot's row starts on its receiver (null: nothing to send for the slot)
      float scale[NJ];
      int row_of[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        out_row[j] = nullptr; scale[j] = 1.0f; row_of[j] = 0;
        if (j < nj) {
          const long long tj = static_cast<long long>(t) * a.K + jbeg + j;
          const int e = a.topk_idx[tj];
          if (e < 0 || e >= E) {  // not an expert: nothing is indexed with it; the step is flagged and the entry skipped
            if (first) report_failure(a.status, kStatusBadArg, kSiteExpertId, static_cast<unsigned long long>(tj), static_cast<unsigned long long>(static_cast<unsigned int>(e)), static_cast<unsigned long long>(E));
            continue;
          }
          int row;
          if (a.compute_rows) {
            row = a.send_base[e] + a.block_base[static_cast<long long>(t / tpb) * E + e] + a.slot_in_block[tj];
            if (first) a.dest_row[tj] = row;
          } else {
            row = a.dest_row[tj];
          }
          row_of[j] = row;
          if (ROUNDED) out_row[j] = reinterpret_cast<unsigned char*>(a.local_rows + static_cast<long long>(row) * a.H);
          else out_row[j] = static_cast<unsigned char*>(a.peer_table[e / El]) + a.recv_heap_off + static_cast<long long>(row) * a.H * (FP8 ? 1 : 2);
          if (SCALED) scale[j] = a.row_scale[tj];
          if (first && counted) atomicAdd(&s_cnt[a.tile_rows > 0 ? (e / El) * a.num_tiles + min(row / a.tile_rows, a.num_tiles - 1) : e], 1);
        }
      }
      const uint4* src = reinterpret_cast<const uint4*>(a.x + static_cast<long long>(t) * a.H);
      if constexpr (DOT) {
        const uint4* sum_with = a.sum_with ? reinterpret_cast<const uint4*>(a.sum_with + static_cast<long long>(t) * a.H) : nullptr;
        uint4* grad_out = a.sum_with ? reinterpret_cast<uint4*>(a.grad_out + static_cast<long long>(t) * a.H) : nullptr;
        const long long to_y = a.y_heap_off - a.recv_heap_off;
        float dots[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) dots[j] = 0.0f;
        constexpr int U = KM <= 2 ? 2 : 1;
        const int rounds = chunks / 32, c_end = rounds * (part + 1) / wpr * 32;
        for (int c0 = rounds * part / wpr * 32 + lane; c0 < c_end; c0 += 32 * U) {
          uint4 v[U], w[U], y[NJ][U];   // every load of the pass is in flight before the first value is used
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c0 + 32 * u < c_end) {
              v[u] = __ldg(src + c0 + 32 * u);
              if (sum_with != nullptr) w[u] = __ldg(sum_with + c0 + 32 * u);
            }
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            if (j >= nj || out_row[j] == nullptr) continue;
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (c0 + 32 * u < c_end) y[j][u] = __ldcg(reinterpret_cast<const uint4*>(out_row[j] + to_y) + c0 + 32 * u);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (c0 + 32 * u >= c_end) break;
            float f[8];
            if (sum_with != nullptr) {
              unpack8(add8(v[u], w[u]), f);
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] *= gscale;
              v[u] = pack8(f);
              grad_out[c0 + 32 * u] = v[u];
            }
            unpack8(v[u], f);
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              if (j >= nj || out_row[j] == nullptr) continue;
              float h[8];
              unpack8(y[j][u], h);
#pragma unroll
              for (int i = 0; i < 8; ++i) { dots[j] = fmaf(f[i], h[i], dots[j]); h[i] = f[i] * scale[j]; }
              reinterpret_cast<uint4*>(out_row[j])[c0 + 32 * u] = pack8(h);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          if (j >= nj) break;
          float d = dots[j];
#pragma unroll
          for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
          if (wpr == 1) { if (lane == 0) a.dot_out[static_cast<long long>(t) * a.K + j] = d; }
          else if (lane == 0) s_dot[part][j] = d;
        }
        if (wpr > 1) {   // the CTA's warps share this row
          __syncthreads();
          if (part == 0 && lane < nj) {
            float d = 0.0f;
            for (int q = 0; q < wpr; ++q) d += s_dot[q][lane];
            a.dot_out[static_cast<long long>(t) * a.K + lane] = d;
          }
          __syncthreads();
        }
      } else if constexpr (!FP8) {
        // Four 16-byte chunks per lane in flight before the first store: the loop is bound by the
        // latency of the local loads otherwise.
        constexpr int U = 4;
        const int rounds = chunks / 32, c_end = rounds * (part + 1) / wpr * 32;   // H is a multiple of 256
        for (int c0 = rounds * part / wpr * 32 + lane; c0 < c_end; c0 += 32 * U) {
          uint4 v[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c0 + 32 * u < c_end) v[u] = __ldg(src + c0 + 32 * u);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = c0 + 32 * u;
            if (c >= c_end) break;
            if (ROUNDED) v[u] = through_e4m3(v[u]);   // every lane of the warp is here: rounds are whole
            float f[8];
            if (SCALED) unpack8(v[u], f);
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              if (j >= nj || out_row[j] == nullptr) continue;
              uint4* out = reinterpret_cast<uint4*>(out_row[j]) + c;
              if (SCALED) {
                float g[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) g[i] = f[i] * scale[j];
                *out = pack8(g);
              } else {
                *out = v[u];
              }
            }
          }
        }
      } else {
        // 16 elements per lane (one 16-byte store of e4m3); 8 consecutive lanes = 128 elements share
        // one scale (amax / 448). The row's scales leave as 16-byte stores after the payload: 4-byte
        // remote stores would each cost a packet of their own.
        const int sgroups = a.H / 128;
        const int chunks16 = a.H / 16;
        float* my_scales = s_scales + warp * kMaxScaleGroups;
        if (a.xq != nullptr) {
          // Rows were quantised once by quantise_rows_kernel: this entry copies bytes.
          const uint4* qsrc = reinterpret_cast<const uint4*>(a.xq + static_cast<long long>(t) * a.H);
          constexpr int U = 4;
          for (int c0 = lane; c0 < chunks16; c0 += 32 * U) {
            uint4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (c0 + 32 * u < chunks16) v[u] = __ldg(qsrc + c0 + 32 * u);
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int c = c0 + 32 * u;
              if (c >= chunks16) break;
#pragma unroll
              for (int j = 0; j < NJ; ++j) {
                if (j >= nj || out_row[j] == nullptr) continue;
                *(reinterpret_cast<uint4*>(out_row[j]) + c) = v[u];
              }
            }
          }
          for (int g = lane; g < sgroups; g += 32) my_scales[g] = __ldg(a.xq_scales + static_cast<long long>(t) * sgroups + g);
        } else {
          // The whole warp walks the row together (the shuffles in quantise16 need every lane); lanes past
          // the end of a short row carry zeros and store nothing. Two blocks of 512 elements are in flight
          // per pass (their loads are issued before either is reduced). Measured: neither more resident warps
          // (8, 16 or 24 per SM), nor requesting the next pass before reducing this one, nor packed arithmetic
          // moves this path off about 600 GB/s to one peer; a plain copy of already quantised rows reaches 624.
          constexpr int U = 2;
          const int rounds = (chunks16 + 31) / 32, c_end = min(chunks16, rounds * (part + 1) / wpr * 32);
          for (int c0 = rounds * part / wpr * 32; c0 < c_end; c0 += 32 * U) {
            uint4 raw[U][2];
            bool active[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int c = c0 + 32 * u + lane;
              active[u] = c < c_end;
              raw[u][0] = active[u] ? __ldg(src + 2 * c) : make_uint4(0, 0, 0, 0);
              raw[u][1] = active[u] ? __ldg(src + 2 * c + 1) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (c0 + 32 * u >= c_end) break;  // warp-uniform: the second block of the last pass may not exist
              const int c = c0 + 32 * u + lane;
              float sc;
              const uint4 q = quantise16(raw[u], sc);
              if (active[u] && (lane & 7) == 0) my_scales[c / 8] = sc;
#pragma unroll
              for (int j = 0; j < NJ; ++j) {
                if (j >= nj || !active[u] || out_row[j] == nullptr) continue;
                *(reinterpret_cast<uint4*>(out_row[j]) + c) = q;
              }
            }
          }
        }
        if (wpr > 1) __syncthreads(); else __syncwarp();   // the row's scales are complete (all warps of the CTA are in this round)
        // sgroups is a multiple of 2 (H % 256 == 0): pairs of scales always; quads when the row's scale block is 16-byte aligned.
        const bool quad = (sgroups & 3) == 0;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          if (part != 0 || j >= nj || out_row[j] == nullptr) continue;
          // the receiver's slab base is the row pointer minus the row's offset in the receive buffer
          float* srow = reinterpret_cast<float*>(out_row[j] - a.recv_heap_off - static_cast<long long>(row_of[j]) * a.H + a.scale_heap_off) + static_cast<long long>(row_of[j]) * sgroups;
          if (quad) {
            for (int g = lane * 4; g < sgroups; g += 128) *reinterpret_cast<float4*>(srow + g) = *reinterpret_cast<const float4*>(my_scales + g);
          } else {
            for (int g = lane * 2; g < sgroups; g += 64) *reinterpret_cast<float2*>(srow + g) = *reinterpret_cast<const float2*>(my_scales + g);
          }
        }
        if (wpr > 1) __syncthreads(); else __syncwarp();  // the next row reuses my_scales
      }
    }  // wi < n_work
    if (SORTED && counted && (++round % kPublishRounds) == 0 && base + round_stride < n_work) publish_counts();
  }
  if (counted) publish_counts();
}

// LOSS: the rows are also added to a.residual and squared on their way out. KM: most rows a token has, K <= KM. With 2 the kernel
// keeps 3 or 4 blocks on an SM, with 8 two, and walks no slots that are not there: under the GEMMs'
// power cap the issue slots of an SM are as short as its bandwidth.
template <bool LOSS, int KM>
__global__ void __launch_bounds__(kCommThreads, KM > 2 ? 2 : LOSS ? 3 : 4) combine_pull_kernel(const CombineArgs a) {
  __shared__ int s_ok;
  grid_dependency_wait();
  launch_dependents();
  const int El = a.num_experts / a.world;
  if (threadIdx.x == 0) s_ok = *reinterpret_cast<volatile unsigned long long*>(&a.status->abort) == 0ull;
  __syncthreads();
  const unsigned long long ready_epoch = a.epoch_dev ? *a.epoch_dev : a.ready_epoch;
  if (s_ok && ready_epoch != 0 && a.world > 1) {   // alone, the rows were written by earlier kernels of this stream
    if (a.signal && blockIdx.x == 0 && threadIdx.x < a.world) {
      // My rows are final (this kernel follows their producer): say so to every rank. Block 0 is always resident, so no rank's
      // wait below can keep this from happening.
      __threadfence_system();
      st_release_sys(reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(a.peer_table[threadIdx.x]) + a.ready_flags_heap_off) + a.rank, ready_epoch);
    }
    const unsigned long long* flags = reinterpret_cast<const unsigned long long*>(static_cast<unsigned char*>(a.peer_table[a.rank]) + a.ready_flags_heap_off);
    if (threadIdx.x < a.world && !wait_ge_bounded(flags + threadIdx.x, ready_epoch, a.status, kSiteCombineReady, threadIdx.x, a.timeout_ns)) s_ok = 0;
    __syncthreads();
  }
  if (!s_ok) {
    if (LOSS) route::last_block(a.ticket);   // the count of blocks stays whole
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int rounds = a.H / 256, segs = a.segments;   // rounds of 32 lanes x 8 elements
  float square = 0.0f;   // my share of sum((residual + out)^2)
  // A warp takes one of `segs` column ranges of a token's row.
  for (long long u = blockIdx.x * wpb + warp; u < static_cast<long long>(a.T) * segs; u += gridDim.x * wpb) {
    const int t = static_cast<int>(u / segs), seg = static_cast<int>(u % segs);
    const int c_end = rounds * (seg + 1) / segs * 32;
    const uint4* rows[KM];
    float w[KM];
#pragma unroll
    for (int j = 0; j < KM; ++j) {
      rows[j] = nullptr; w[j] = 0.0f;
      if (j < a.K) {
        const long long tj = static_cast<long long>(t) * a.K + j;
        const int e = a.topk_idx[tj];
        if (e < 0 || e >= a.num_experts) {  // flagged and left out of the sum (rows[j] stays null)
          if (lane == 0) report_failure(a.status, kStatusBadArg, kSiteExpertId, static_cast<unsigned long long>(tj), static_cast<unsigned long long>(static_cast<unsigned int>(e)), static_cast<unsigned long long>(a.num_experts));
          continue;
        }
        rows[j] = reinterpret_cast<const uint4*>(static_cast<unsigned char*>(a.peer_table[e / El]) + a.src_heap_off +
                                                 static_cast<long long>(a.dest_row[tj]) * a.H * 2);
        w[j] = a.weights ? a.weights[tj] : 1.0f;
      }
    }
    uint4* out = reinterpret_cast<uint4*>(a.out + static_cast<long long>(t) * a.H);
    constexpr int U = 2;  // two chunks x K rows of peer loads in flight per lane
    for (int c0 = rounds * seg / segs * 32 + lane; c0 < c_end; c0 += 32 * U) {
      uint4 v[U][KM], res[U];
      if (LOSS) {
        const uint4* h = reinterpret_cast<const uint4*>(a.residual + static_cast<long long>(t) * a.H);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (c0 + 32 * u < c_end) res[u] = __ldg(h + c0 + 32 * u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < KM; ++j)
          if (j < a.K && c0 + 32 * u < c_end) v[u][j] = rows[j] ? __ldcg(rows[j] + c0 + 32 * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + 32 * u;
        if (c >= c_end) break;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < KM; ++j) {
          if (j >= a.K) break;
          float f[8];
          unpack8(v[u][j], f);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = fmaf(w[j], f[i], acc[i]);
        }
        const uint4 o = pack8(acc);
        out[c] = o;
        if (LOSS) {
          float q[8];
          unpack8(add8(o, res[u]), q);
#pragma unroll
          for (int i = 0; i < 8; ++i) square = fmaf(q[i], q[i], square);
        }
      }
    }
  }
  if constexpr (LOSS) {
    // Block sums, then the last block adds them up in a fixed order.
    __shared__ float s_sum[kCommThreads / 32];
    square = warp_sum(square);
    if (lane == 0) s_sum[warp] = square;
    __syncthreads();
    if (threadIdx.x == 0) {
      float v = 0.0f;
      for (int i = 0; i < wpb; ++i) v += s_sum[i];
      a.loss_partials[blockIdx.x] = v;
    }
    if (!route::last_block(a.ticket)) return;
    float v = 0.0f;
    for (int i = threadIdx.x; i < gridDim.x; i += blockDim.x) v += __ldcg(a.loss_partials + i);
    v = warp_sum(v);
    if (lane == 0) s_sum[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      v = 0.0f;
      for (int i = 0; i < wpb; ++i) v += s_sum[i];
      *a.loss = v * a.loss_scale;
    }
  }
}

__global__ void wait_counters_kernel(const unsigned long long* counter, const unsigned long long* target, int n, DeviceStatus* st,
                                     unsigned long long timeout_ns) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) wait_ge_bounded(counter + i, target[i], st, kSiteRailArrive, i, timeout_ns);
}

}  // namespace

cudaError_t launch_dispatch_push(const DispatchArgs& a, int ctas, cudaStream_t stream) {
  if (a.K < 1 || a.K > kMaxK || a.H % 256 || a.world < 1 || a.num_experts % a.world || ctas < 1) return cudaErrorInvalidValue;
  if (a.fp8 && a.H / 128 > kMaxScaleGroups) return cudaErrorInvalidValue;
  if ((a.xq != nullptr) != (a.xq_scales != nullptr) || (a.xq != nullptr && !a.fp8)) return cudaErrorInvalidValue;
  const bool announces = a.entry_epoch != 0 && a.world > 1;   // the peers wait for my entry flag, rows or none
  if (a.T == 0 && !announces) return cudaSuccess;
  if (a.tile_rows < 0 || (a.tile_rows > 0 && a.num_tiles < 1)) return cudaErrorInvalidValue;
  if (a.local_rows != nullptr && (!a.fp8 || a.send_list != nullptr || a.row_scale != nullptr || a.world != 1)) return cudaErrorInvalidValue;
  if (a.dot_out != nullptr && (a.fp8 || a.send_list != nullptr || a.row_scale == nullptr)) return cudaErrorInvalidValue;
  if (a.sum_with != nullptr && (a.dot_out == nullptr || a.grad_out == nullptr || a.grad_loss == nullptr)) return cudaErrorInvalidValue;
  DispatchArgs b = a;
  b.warps_per_row = a.send_list == nullptr && a.T <= ctas ? kCommThreads / 32 : 1;
  // No more CTAs than there is work for (entries of the sorted list, rows per CTA otherwise).
  const long long work = a.send_list != nullptr ? static_cast<long long>(a.T) * a.K : static_cast<long long>(a.T) * b.warps_per_row;
  ctas = announce_blocks(static_cast<int>(std::min<long long>(ctas, (work + kCommThreads / 32 - 1) / (kCommThreads / 32))), announces);
  const size_t smem = sizeof(int) * (a.tile_rows > 0 ? static_cast<size_t>(a.world) * a.num_tiles : static_cast<size_t>(a.num_experts));
  if (smem > 200 * 1024) return cudaErrorInvalidValue;  // per-CTA histogram of destination tiles must fit in shared memory
  auto go = [&](auto kern) {
    cudaError_t e = allow_smem(kern, smem);
    if (e == cudaSuccess) e = launch_early(kern, dim3(ctas), kCommThreads, smem, stream, b);
    if (e == cudaSuccess) note_launch();
    return e;
  };
  const bool sorted = a.send_list != nullptr, scaled = a.row_scale != nullptr;
  const bool few = a.K <= 2 && !sorted && !a.fp8;
  if (a.dot_out != nullptr) return few ? go(dispatch_push_kernel<false, false, true, false, true, 2>) : go(dispatch_push_kernel<false, false, true, false, true>);
  if (a.local_rows != nullptr) return go(dispatch_push_kernel<false, false, false, true>);
  if (a.fp8) return sorted ? go(dispatch_push_kernel<true, true, false>) : go(dispatch_push_kernel<true, false, false>);
  if (sorted) return scaled ? go(dispatch_push_kernel<false, true, true>) : go(dispatch_push_kernel<false, true, false>);
  if (few) return scaled ? go(dispatch_push_kernel<false, false, true, false, false, 2>) : go(dispatch_push_kernel<false, false, false, false, false, 2>);
  return scaled ? go(dispatch_push_kernel<false, false, true>) : go(dispatch_push_kernel<false, false, false>);
}

cudaError_t launch_quantise_rows(const __nv_bfloat16* x, int T, int H, unsigned char* q, float* scales, int ctas, cudaStream_t stream) {
  if (H % 256 || H / 128 > kMaxScaleGroups || ctas < 1 || T < 0) return cudaErrorInvalidValue;
  if (T == 0) return cudaSuccess;
  quantise_rows_kernel<<<ctas, kCommThreads, 0, stream>>>(x, T, H, q, scales);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_combine_pull(const CombineArgs& a, int ctas, cudaStream_t stream) {
  if (a.K < 1 || a.K > kMaxK || a.H % 256 || a.world < 1 || a.num_experts % a.world || ctas < 1) return cudaErrorInvalidValue;
  if (a.residual != nullptr && (a.out == nullptr || a.loss_partials == nullptr || a.ticket == nullptr || a.loss == nullptr || ctas > kMaxLossPartials)) return cudaErrorInvalidValue;
  if (a.residual != nullptr) ctas = std::max(1, ctas * 3 / 4);   // a grid of four blocks per SM; three of this variant fit
  // Without tokens of my own: the peers still wait for my ready flag.
  ctas = announce_blocks(a.T > 0 ? ctas : 0, a.signal && a.world > 1 && (a.ready_epoch != 0 || a.epoch_dev != nullptr));
  if (ctas == 0) return cudaSuccess;
  CombineArgs b = a;
  // Few tokens: as many warps per row as fill the grid, down to one round of loads per warp.
  b.segments = static_cast<int>(std::clamp<long long>(static_cast<long long>(ctas) * (kCommThreads / 32) / std::max(a.T, 1), 1, a.H / 256));
  cudaError_t e = launch_early(a.K <= 2 ? (a.residual != nullptr ? combine_pull_kernel<true, 2> : combine_pull_kernel<false, 2>)
                                      : (a.residual != nullptr ? combine_pull_kernel<true, kMaxK> : combine_pull_kernel<false, kMaxK>),
                               dim3(ctas), kCommThreads, 0, stream, b);
  if (e == cudaSuccess) note_launch();
  return e;
}

cudaError_t launch_wait_counters(const unsigned long long* counter, const unsigned long long* target, int n, DeviceStatus* status,
                                 unsigned long long timeout_ns, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  wait_counters_kernel<<<(n + 63) / 64, 64, 0, stream>>>(counter, target, n, status, timeout_ns);
  note_launch();
  return cudaGetLastError();
}

}  // namespace fastb
