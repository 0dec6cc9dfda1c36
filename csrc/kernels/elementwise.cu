// Element-wise kernels of the expert MLP and the optimizer (memory-bound; 16-byte accesses).
#include <cuda_fp8.h>

#include "api.h"
#include "early_start.cuh"

namespace fastb {

namespace {

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

// gate_up rows are tiles of [128 gate | 128 up]; chunk c (8 features) of tile n sits at
// 256 n + 8 (c % 16) for the gate and 128 further for the up projection.
__global__ void swiglu_fwd_kernel(const uint4* __restrict__ gu, uint4* __restrict__ act, long long rows, int inter) {
  const int cpr = inter / 8;  // output chunks per row
  const long long total = rows * cpr;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / cpr;
    const int c = static_cast<int>(i % cpr);
    const long long base = r * (2 * cpr) + (c / 16) * 32 + (c % 16);
    float g[8], u[8], o[8];
    unpack8(gu[base], g);
    unpack8(gu[base + 16], u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = g[k] / (1.0f + __expf(-g[k])) * u[k];
    act[i] = pack8(o);
  }
}

__global__ void swiglu_bwd_kernel(const uint4* __restrict__ gu, const uint4* __restrict__ dact, uint4* __restrict__ dgu, long long rows, int inter,
                                  const int* __restrict__ rows_dev) {
  if (rows_dev) rows = min(rows, static_cast<long long>(*rows_dev));  // rows in use this step (device-side count)
  const int cpr = inter / 8;
  const long long total = rows * cpr;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / cpr;
    const int c = static_cast<int>(i % cpr);
    const long long base = r * (2 * cpr) + (c / 16) * 32 + (c % 16);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(gu[base], g);
    unpack8(gu[base + 16], u);
    unpack8(dact[i], d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float s = 1.0f / (1.0f + __expf(-g[k]));
      const float silu = g[k] * s;
      du[k] = d[k] * silu;
      dg[k] = d[k] * u[k] * (s + silu * (1.0f - s));
    }
    dgu[base] = pack8(dg);
    dgu[base + 16] = pack8(du);
  }
}

__global__ void dequant_fp8_kernel(const uint2* __restrict__ q, const float* __restrict__ scales, uint4* __restrict__ out, long long rows, int H,
                                   const int* __restrict__ rows_dev) {
  if (rows_dev) rows = min(rows, static_cast<long long>(*rows_dev));
  const int cpr = H / 8;
  const long long total = rows * cpr;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / cpr;
    const int c = static_cast<int>(i % cpr);
    const float sc = scales[r * (H / 128) + c / 16];
    const uint2 v = q[i];
    const unsigned char* b = reinterpret_cast<const unsigned char*>(&v);
    float f[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const __half_raw h = __nv_cvt_fp8_to_halfraw(b[k], __NV_E4M3);
      f[k] = __half2float(*reinterpret_cast<const __half*>(&h)) * sc;
    }
    out[i] = pack8(f);
  }
}

// A block takes kAdamChunk consecutive parameters of one tensor, four of them a thread at a time: fp32 accesses are 16 bytes,
// contiguous across the warp, bf16 accesses 8 bytes. Nothing is read twice, so every access is marked streaming. Bound by
// HBM (28 bytes a parameter): one short block per chunk, as many as there are, keeps the seven streams of all resident
// blocks within a narrow moving window: 6.9 TB/s over 0.94 G parameters. A grid of resident blocks that strides through
// the same arrays reaches 6.1, bulk copies through shared memory 6.4. All tensors of an optimizer step are one launch.
constexpr int kAdamThreads = 256, kAdamPerThread = 2, kAdamChunk = 4 * kAdamThreads * kAdamPerThread;
__global__ void __launch_bounds__(kAdamThreads) adamw_kernel(const __grid_constant__ AdamWArgs a) {
  int k = 0;
  unsigned int block = blockIdx.x;
  grid_dependency_wait();
  launch_dependents();
  while (block >= a.t[k].blocks) block -= a.t[k++].blocks;
  const AdamWTensor& t = a.t[k];
  const long long n4 = t.n / 4, base = static_cast<long long>(block) * (kAdamChunk / 4) + threadIdx.x;
  uint2* param = reinterpret_cast<uint2*>(t.param);
  float4 *master = reinterpret_cast<float4*>(t.master), *m = reinterpret_cast<float4*>(t.m), *v = reinterpret_cast<float4*>(t.v);
  const uint2* grad = reinterpret_cast<const uint2*>(t.grad);
  constexpr int U = kAdamPerThread;
  float4 w[U], mm[U], vv[U];
  uint2 g[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + u * kAdamThreads;
    if (i < n4) { g[u] = __ldcs(grad + i); w[u] = __ldcs(master + i); mm[u] = __ldcs(m + i); vv[u] = __ldcs(v + i); }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + u * kAdamThreads;
    if (i >= n4) break;
    const float2 g01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g[u].x));
    const float2 g23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g[u].y));
    const float gk[4] = {g01.x * a.gscale, g01.y * a.gscale, g23.x * a.gscale, g23.y * a.gscale};
    float* wp = reinterpret_cast<float*>(&w[u]);
    float* mp = reinterpret_cast<float*>(&mm[u]);
    float* vp = reinterpret_cast<float*>(&vv[u]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      mp[q] = a.b1 * mp[q] + (1.0f - a.b1) * gk[q];
      vp[q] = a.b2 * vp[q] + (1.0f - a.b2) * gk[q] * gk[q];
      const float upd = (mp[q] * t.c1) / (sqrtf(vp[q] * t.c2) + a.eps);
      wp[q] = wp[q] - a.lr * (upd + a.wd * wp[q]);
    }
    __stcs(master + i, w[u]);
    __stcs(m + i, mm[u]);
    __stcs(v + i, vv[u]);
    uint2 pb;
    *reinterpret_cast<__nv_bfloat162*>(&pb.x) = __floats2bfloat162_rn(wp[0], wp[1]);
    *reinterpret_cast<__nv_bfloat162*>(&pb.y) = __floats2bfloat162_rn(wp[2], wp[3]);
    __stcs(param + i, pb);
  }
}

// sum((a + b)^2) over n8 chunks of 8 bf16: per-block partial sums, then one block folds them in a
// fixed order (deterministic).
__global__ void sumsq_add_partial_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, long long n8, float* __restrict__ partial) {
  float acc = 0.0f;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n8; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8], y[8];
    unpack8(a[i], x);
    unpack8(b[i], y);
#pragma unroll
    for (int k = 0; k < 8; ++k) { const float o = __bfloat162float(__float2bfloat16_rn(x[k] + y[k])); acc = fmaf(o, o, acc); }
  }
  __shared__ float s[32];
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? s[threadIdx.x] : 0.0f;
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
  }
}
__global__ void fold_partials_kernel(const float* __restrict__ partial, int n, float scale, float* __restrict__ out) {
  __shared__ float s[32];
  float acc = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += partial[i];
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? s[threadIdx.x] : 0.0f;
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) *out = v * scale;
  }
}
// grad = (a + b) * (*gscale) * factor, as bf16.
__global__ void scaled_sum_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, long long n8, const float* __restrict__ gscale, float factor,
                                  uint4* __restrict__ out) {
  const float g = (*gscale) * factor;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n8; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8], y[8], o[8];
    unpack8(a[i], x);
    unpack8(b[i], y);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = __bfloat162float(__float2bfloat16_rn(x[k] + y[k])) * g;
    out[i] = pack8(o);
  }
}

// ---- ids grouped by value, positions in order: a counting sort the embedding gradient is fed from -----------
// The sort's work is independent of the data (heavy duplicates cost the same as none). Blocks of kIdxBlock tokens:
//   1. per-block histogram of the ids (counts) and, per token, its rank among the block's earlier tokens with
//      the same id (position order, so the grouping is stable and the later summation order is fixed);
//   2. per id, the running sum over blocks (where a block's tokens of that id start inside the id's run);
//   3. exclusive scan over the ids (where each id's run starts);
//   4. scatter: sorted_ids / perm; embedding_rows_kernel reads start and perm.
constexpr int kIdxBlock = 256;

__global__ void __launch_bounds__(kIdxBlock) emb_block_hist_kernel(const long long* __restrict__ ids, long long T, int V, int* __restrict__ hist,
                                                                   int* __restrict__ rank_in_block) {
  __shared__ long long s_id[kIdxBlock];
  const long long p = blockIdx.x * static_cast<long long>(kIdxBlock) + threadIdx.x;
  long long id = -1;
  if (p < T) { id = ids[p]; if (id < 0 || id >= V) id = -1; }  // out-of-range ids take no part (F.embedding would have refused them)
  s_id[threadIdx.x] = id;
  __syncthreads();
  if (id < 0) { if (p < T) rank_in_block[p] = -1; return; }
  int r = 0;
  for (int j = 0; j < static_cast<int>(threadIdx.x); ++j) r += s_id[j] == id ? 1 : 0;
  rank_in_block[p] = r;
  atomicAdd(hist + static_cast<long long>(blockIdx.x) * V + id, 1);
}

__global__ void emb_scan_blocks_kernel(int* __restrict__ hist, int blocks, int V, int* __restrict__ total) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  int run = 0;
  // Eight independent loads in flight per round (the running sum is the only serial part).
  for (int b0 = 0; b0 < blocks; b0 += 8) {
    int c[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) c[u] = b0 + u < blocks ? hist[static_cast<long long>(b0 + u) * V + v] : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b0 + u < blocks) { hist[static_cast<long long>(b0 + u) * V + v] = run; run += c[u]; }  // counts become offsets inside the id's run
  }
  total[v] = run;
}

// Single block: start[v] = sum of total[< v]; start[V] = number of tokens that took part. Tiles of 4096 ids, each
// warp 128 of them with coalesced 16-byte accesses; all tiles of a batch are requested before the first is summed (eight
// dependent passes over 32000 ids took 25 us).
__global__ void __launch_bounds__(1024) emb_scan_ids_kernel(const int* __restrict__ total, int V, int* __restrict__ start) {
  constexpr int N = 8;                       // tiles of a batch
  __shared__ int s_warp[N][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry = 0;
  for (int v0 = 0; v0 < V; v0 += 4096 * N) {
    int x[N][4], incl[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int v = v0 + 4096 * n + 4 * static_cast<int>(threadIdx.x);
      if (v + 3 < V) {
        const int4 q = __ldg(reinterpret_cast<const int4*>(total + v));   // v is a multiple of 4
        x[n][0] = q.x; x[n][1] = q.y; x[n][2] = q.z; x[n][3] = q.w;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) x[n][u] = v + u < V ? __ldg(total + v + u) : 0;
      }
    }
    __syncthreads();   // the previous batch has read s_warp
#pragma unroll
    for (int n = 0; n < N; ++n) {
      incl[n] = x[n][0] + x[n][1] + x[n][2] + x[n][3];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl[n], o); if (lane >= o) incl[n] += y; }
      if (lane == 31) s_warp[n][warp] = incl[n];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int w = s_warp[n][lane];
      const int before = static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(lane < warp ? w : 0))), all = static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(w)));
      int at = carry + before + incl[n] - (x[n][0] + x[n][1] + x[n][2] + x[n][3]);
      const int v = v0 + 4096 * n + 4 * static_cast<int>(threadIdx.x);
#pragma unroll
      for (int u = 0; u < 4; ++u) { if (v + u < V) start[v + u] = at; at += x[n][u]; }
      carry += all;
    }
  }
  if (threadIdx.x == 0) start[V] = carry;
}

__global__ void emb_scatter_kernel(const long long* __restrict__ ids, const int* __restrict__ rank_in_block, const int* __restrict__ hist,
                                   const int* __restrict__ start, long long T, int V, long long* __restrict__ sorted_ids, long long* __restrict__ perm) {
  const long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (p >= T) return;
  const int r = rank_in_block[p];
  if (r < 0) return;
  const long long id = ids[p];
  const long long slot = start[id] + hist[(p / kIdxBlock) * V + id] + r;
  sorted_ids[slot] = id;
  perm[slot] = p;
}

// ---- the whole gradient of an embedding table ------------------------------------------------------------------
// A warp per table row, after the counting sort: every row is written once, its sum or zeros (cleared beforehand by a kernel of
// its own, the table cost one more pass of writes: 91 us for 32000 x 4096), in position order: evenly spread ids are bound by HBM.
// A warp reads its row's positions once and takes two of them at a time, 512 columns at once. A row with more than kEmbAlone positions is summed
// by its block's eight warps, 256 columns each and sixteen positions' loads ahead; by one warp, one load ahead, it was a chain. us with the
// sort, spread evenly, one warp per row with one load ahead -> eight loads ahead in shared rows -> this: 32768 ids on 32000 x 4096
// 189 -> 197 -> 169, 65536 on 32000 x 2048 174 -> 183 -> 159, 8192 on 32000 x 4096 113 -> 114 -> 107; 32768 skewed (one of them 27 %) on
// 32000 x 4096 67200 -> 3800 -> 3200.
constexpr int kEmbAlone = 16;
__global__ void __launch_bounds__(256) embedding_rows_kernel(const int* __restrict__ start, const long long* __restrict__ perm, const uint4* __restrict__ grad_out, uint4* __restrict__ grad_table, int V, int H) {
  const long long v0 = blockIdx.x * 8ll;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunks = H / 8;
  const int bound = v0 + lane <= V && lane <= 8 ? __ldg(start + v0 + lane) : 0;   // lane i: where row v0 + i starts
  const int next = __shfl_down_sync(0xffffffffu, bound, 1);
  const unsigned shared = __ballot_sync(0xffffffffu, lane < 8 && v0 + lane < V && next - bound > kEmbAlone);
  const int begin = __shfl_sync(0xffffffffu, bound, warp), end = __shfl_sync(0xffffffffu, next, warp);
  if (v0 + warp < V && !(shared >> warp & 1)) {
    uint4* out = grad_table + (v0 + warp) * chunks;
    const int n = end - begin;
    const long long pos = lane < n ? __ldg(perm + begin + lane) : 0;
    constexpr int U = 2;   // chunks in flight per row
    for (int first_c = 0; first_c < chunks; first_c += 32 * U) {
      const int c0 = first_c + lane;
      float acc[U][8] = {};
      const auto add = [&](int j, auto depth) {   // `depth` positions' loads ahead, added one after the other
        constexpr int J = decltype(depth)::value;
        uint4 x[J][U];
#pragma unroll
        for (int d = 0; d < J; ++d) {
          const uint4* row = grad_out + static_cast<long long>(__shfl_sync(0xffffffffu, pos, j + d)) * chunks;
#pragma unroll
          for (int u = 0; u < U; ++u) x[d][u] = c0 + 32 * u < chunks ? __ldg(row + c0 + 32 * u) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int d = 0; d < J; ++d)
#pragma unroll
          for (int u = 0; u < U; ++u) {
            float f[8];
            unpack8(x[d][u], f);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[u][k] += f[k];
          }
      };
      int j = 0;
      for (; j + 2 <= n; j += 2) add(j, std::integral_constant<int, 2>());
      if (j < n) add(j, std::integral_constant<int, 1>());
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c0 + 32 * u < chunks) __stcs(out + c0 + 32 * u, pack8(acc[u]));
    }
  }
  for (unsigned left = shared; left; left &= left - 1) {
    const int i = __ffs(left) - 1, first = __shfl_sync(0xffffffffu, bound, i), last = __shfl_sync(0xffffffffu, next, i);
    for (int c = threadIdx.x; c < chunks; c += 256) {
      float acc[8] = {};
      const auto add = [&](int j, auto depth) {
        constexpr int J = decltype(depth)::value;
        uint4 x[J];
#pragma unroll
        for (int d = 0; d < J; ++d) x[d] = __ldg(grad_out + __ldg(perm + j + d) * chunks + c);
#pragma unroll
        for (int d = 0; d < J; ++d) {
          float f[8];
          unpack8(x[d], f);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] += f[k];
        }
      };
      int j = first;
      for (; j + 16 <= last; j += 16) add(j, std::integral_constant<int, 16>());
      for (; j + 4 <= last; j += 4) add(j, std::integral_constant<int, 4>());
      for (; j < last; ++j) add(j, std::integral_constant<int, 1>());
      __stcs(grad_table + (v0 + i) * chunks + c, pack8(acc));
    }
  }
}

// Few tokens: the whole table gradient in one pass, every row written once. Of each 2^bits rows a block has one, and another one in
// the next 2^bits (frequent ids, neighbours or a power of two apart, fall to different blocks). A block files the positions that
// name its rows, in position order; its warps clear the rows that none names and share the others' columns, 512 at a time, four
// positions' loads ahead. Bound by the writes, and where one id has hundreds of positions by the reads that a warp has in flight.
// Against a memset and a warp per position that searched all others for its id (T * T / 32 comparisons) and summed them
// alone, on a table of 32000 x 4096: 4096 ids spread evenly 91 -> 62 us, skewed (one of them 27 %) 8411 -> 363, all the same 30590 ->
// 1200, 64 ids 48 -> 46. In blocks: 512, 1024, 2048 took 71, 68, 62 us there and 25, 22.5, 25 on 32000 x 1024 (the ids are read by
// each block): 2048 from 128 MB of table on.
constexpr int kEmbTokens = 4096, kEmbWarps = 8;
__device__ __forceinline__ int emb_mix(int low, int local, int bits) { return (low ^ local ^ local >> bits) & ((1 << bits) - 1); }   // its own inverse in low
__global__ void __launch_bounds__(32 * kEmbWarps, 4) embedding_few_kernel(const long long* __restrict__ ids, const uint4* __restrict__ grad_out, uint4* __restrict__ grad_table, int T, int V, int H, int bits) {
  constexpr int R = kEmbTokens / (32 * kEmbWarps), U = 2;
  __shared__ int s_row[kEmbTokens];              // of the block's own rows: which one, and the position that names it
  __shared__ unsigned short s_pos[kEmbTokens];
  __shared__ unsigned s_named[32];                  // a bit per own row (modulo 1024): clear means that no position names it
  __shared__ int s_count[kEmbWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunks = H / 8, own = static_cast<int>(blockIdx.x);
  if (threadIdx.x < 32) s_named[threadIdx.x] = 0;
  grid_dependency_wait();
  launch_dependents();
  const int part = (T + 32 * kEmbWarps - 1) / (32 * kEmbWarps) * 32, first = warp * part;
  int row[R], n = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int p = first + 32 * r + lane;
    const long long id = 32 * r < part && p < T ? __ldg(ids + p) : -1;   // ids outside [0, V) take no part
    row[r] = id >= 0 && id < V && emb_mix(static_cast<int>(id), static_cast<int>(id) >> bits, bits) == own ? static_cast<int>(id) >> bits : -1;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) n += __popc(__ballot_sync(0xffffffffu, row[r] >= 0));
  if (lane == 0) s_count[warp] = n;
  __syncthreads();
  int at = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kEmbWarps; ++w) {
    at += w < warp ? s_count[w] : 0;
    total += s_count[w];
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const unsigned m = __ballot_sync(0xffffffffu, row[r] >= 0);
    if (row[r] >= 0) {
      const int k = at + __popc(m & ((1u << lane) - 1));
      s_row[k] = row[r];
      s_pos[k] = static_cast<unsigned short>(first + 32 * r + lane);
      atomicOr(&s_named[row[r] >> 5 & 31], 1u << (row[r] & 31));
    }
    at += __popc(m);
  }
  __syncthreads();
  const int rows = ((V - 1) >> bits) + 1;
  const auto named = [&](int local) { return (s_named[local >> 5 & 31] >> (local & 31) & 1) != 0; };
  const auto row_of = [&](int local) { return (static_cast<long long>(local) << bits) + emb_mix(own, local, bits); };
  for (int local = warp; local < rows; local += kEmbWarps)
    if (row_of(local) < V && !named(local)) {
      uint4* out = grad_table + row_of(local) * chunks;
#pragma unroll 4
      for (int c = lane; c < chunks; c += 32) out[c] = make_uint4(0, 0, 0, 0);
    }
  int turn = 0;
  for (int local = 0; total && local < rows; ++local) {
    if (!named(local) || row_of(local) >= V) continue;
    uint4* out = grad_table + row_of(local) * chunks;
    for (int first_c = 0; first_c < chunks; first_c += 32 * U) {
      if (turn++ % kEmbWarps != warp) continue;
      int c[U];   // past the end: the last one again, not written
#pragma unroll
      for (int u = 0; u < U; ++u) c[u] = min(first_c + 32 * u + lane, chunks - 1);
      float acc[U][8] = {};
      for (int q0 = 0; q0 < total; q0 += 32) {
        unsigned m = __ballot_sync(0xffffffffu, q0 + lane < total && s_row[min(q0 + lane, total - 1)] == local);
        const auto add = [&](auto depth) {   // `depth` positions' loads ahead, added one after the other
          constexpr int J = decltype(depth)::value;
          uint4 v[J][U];
#pragma unroll
          for (int j = 0; j < J; ++j) {
            const uint4* from = grad_out + static_cast<long long>(s_pos[q0 + __ffs(m) - 1]) * chunks;
            m &= m - 1;
#pragma unroll
            for (int u = 0; u < U; ++u) v[j][u] = __ldg(from + c[u]);
          }
#pragma unroll
          for (int j = 0; j < J; ++j)
#pragma unroll
            for (int u = 0; u < U; ++u) {
              float f[8];
              unpack8(v[j][u], f);
#pragma unroll
              for (int k = 0; k < 8; ++k) acc[u][k] += f[k];
            }
        };
        while (__popc(m) >= 4) add(std::integral_constant<int, 4>());
        while (m) add(std::integral_constant<int, 1>());
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (first_c + 32 * u + lane < chunks) out[c[u]] = pack8(acc[u]);
    }
  }
}

int grid_for(long long items) { return static_cast<int>(std::min<long long>((items + 255) / 256, 148 * 8)); }

}  // namespace

cudaError_t launch_swiglu_fwd(const __nv_bfloat16* gate_up, __nv_bfloat16* act, long long rows, int inter, cudaStream_t stream) {
  if (inter % 128) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  swiglu_fwd_kernel<<<grid_for(rows * inter / 8), 256, 0, stream>>>(reinterpret_cast<const uint4*>(gate_up), reinterpret_cast<uint4*>(act), rows, inter);
  note_launch();
  return cudaGetLastError();
}
cudaError_t launch_swiglu_bwd(const __nv_bfloat16* gate_up, const __nv_bfloat16* d_act, __nv_bfloat16* d_gate_up, long long rows, int inter,
                              const int* rows_dev, cudaStream_t stream) {
  if (inter % 128) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  swiglu_bwd_kernel<<<grid_for(rows * inter / 8), 256, 0, stream>>>(reinterpret_cast<const uint4*>(gate_up), reinterpret_cast<const uint4*>(d_act),
                                                                  reinterpret_cast<uint4*>(d_gate_up), rows, inter, rows_dev);
  note_launch();
  return cudaGetLastError();
}
cudaError_t launch_sumsq_add(const __nv_bfloat16* a, const __nv_bfloat16* b, long long n, float scale, float* partial, int partial_len, float* out,
                             cudaStream_t stream) {
  if (n % 8 || partial_len < 1) return cudaErrorInvalidValue;
  const int blocks = std::min(partial_len, grid_for(n / 8));
  sumsq_add_partial_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const uint4*>(a), reinterpret_cast<const uint4*>(b), n / 8, partial);
  fold_partials_kernel<<<1, 1024, 0, stream>>>(partial, blocks, scale, out);
  note_launch(2);
  return cudaGetLastError();
}
cudaError_t launch_scaled_sum(const __nv_bfloat16* a, const __nv_bfloat16* b, long long n, const float* gscale, float factor, __nv_bfloat16* out,
                              cudaStream_t stream) {
  if (n % 8) return cudaErrorInvalidValue;
  if (n == 0) return cudaSuccess;
  scaled_sum_kernel<<<grid_for(n / 8), 256, 0, stream>>>(reinterpret_cast<const uint4*>(a), reinterpret_cast<const uint4*>(b), n / 8, gscale, factor,
                                                       reinterpret_cast<uint4*>(out));
  note_launch();
  return cudaGetLastError();
}
cudaError_t launch_embedding_index(const long long* ids, long long T, int V, int* hist, int* rank_in_block, int* total, int* start, long long* sorted_ids,
                                   long long* perm, cudaStream_t stream) {
  if (T <= 0 || V <= 0) return cudaErrorInvalidValue;
  const int blocks = static_cast<int>((T + kIdxBlock - 1) / kIdxBlock);
  cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(int) * static_cast<size_t>(blocks) * V, stream);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(sorted_ids, 0xFF, sizeof(long long) * static_cast<size_t>(T), stream);  // -1: slots that stay unused are skipped downstream
  if (e != cudaSuccess) return e;
  emb_block_hist_kernel<<<blocks, kIdxBlock, 0, stream>>>(ids, T, V, hist, rank_in_block);
  emb_scan_blocks_kernel<<<(V + 255) / 256, 256, 0, stream>>>(hist, blocks, V, total);
  emb_scan_ids_kernel<<<1, 1024, 0, stream>>>(total, V, start);
  emb_scatter_kernel<<<blocks, kIdxBlock, 0, stream>>>(ids, rank_in_block, hist, start, T, V, sorted_ids, perm);
  note_launch(4);
  return cudaGetLastError();
}
int embedding_index_block() { return kIdxBlock; }
cudaError_t launch_embedding_rows(const int* start, const long long* perm, const __nv_bfloat16* grad_out, __nv_bfloat16* grad_table, int V, int H, cudaStream_t stream) {
  if (H % 8) return cudaErrorInvalidValue;
  embedding_rows_kernel<<<static_cast<unsigned>((V + 7ll) / 8), 256, 0, stream>>>(start, perm, reinterpret_cast<const uint4*>(grad_out), reinterpret_cast<uint4*>(grad_table), V, H);
  note_launch();
  return cudaGetLastError();
}
cudaError_t launch_embedding_few(const long long* ids, const __nv_bfloat16* grad_out, __nv_bfloat16* grad_table, int T, int V, int H, cudaStream_t stream) {
  if (H % 8 || T > kEmbTokens) return cudaErrorInvalidValue;
  if (V == 0 || H == 0) return cudaSuccess;
  const int bits = static_cast<long long>(V) * H >= 1ll << 26 ? 11 : 10;
  const cudaError_t e = launch_early(embedding_few_kernel, dim3(1 << bits), 32 * kEmbWarps, 0, stream, ids, reinterpret_cast<const uint4*>(grad_out), reinterpret_cast<uint4*>(grad_table), T, V, H, bits);
  note_launch();
  return e;
}
cudaError_t launch_dequant_fp8(const unsigned char* q, const float* scales, __nv_bfloat16* out, long long rows, int H, const int* rows_dev,
                               cudaStream_t stream) {
  if (H % 128) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  dequant_fp8_kernel<<<grid_for(rows * H / 8), 256, 0, stream>>>(reinterpret_cast<const uint2*>(q), scales, reinterpret_cast<uint4*>(out), rows, H, rows_dev);
  note_launch();
  return cudaGetLastError();
}
cudaError_t launch_adamw(AdamWArgs args, cudaStream_t stream) {
  if (args.count < 0 || args.count > kAdamWTensors) return cudaErrorInvalidValue;
  long long blocks = 0;
  for (int k = 0; k < args.count; ++k) {
    AdamWTensor& t = args.t[k];
    if (t.n < 0 || t.n % 8) return cudaErrorInvalidValue;
    t.blocks = static_cast<unsigned int>((t.n + kAdamChunk - 1) / kAdamChunk);
    blocks += t.blocks;
  }
  if (blocks == 0) return cudaSuccess;
  if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
  const cudaError_t e = launch_early(adamw_kernel, dim3(static_cast<unsigned>(blocks)), kAdamThreads, 0, stream, args);
  note_launch();
  return e;
}

}  // namespace fastb
