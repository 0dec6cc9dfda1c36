// Router front end fused into one pass over the activations:
//   norm_gate_route : RMSNorm(h) -> hn, router logits hn . gate^T, softmax-over-top-k weights, the
//                     expert choice and the per-block histogram / stable ranks that the split scan
//                     consumes (what route_topk produces from ready-made logits);
//   norm_gate_bwd   : the matching backward: gradients of the selected logits from the weight
//                     gradients, d(hn) = grad of the MoE input + sum_j dlogit_j * gate[e_j], the gate
//                     and norm-weight gradients (block partials in shared memory, then fp32 atomics)
//                     and the RMSNorm backward to d(h).
// The reference has no router; in a stock stack these are a layer-norm kernel, a small library
// GEMM, top-k, gather, softmax and their backward kernels with the activations re-read each time.
// Limits: num_experts <= 32 (one logit per lane), hidden % 256 == 0, and the gate matrix (forward)
// or the gate matrix plus the fp32 gradient accumulators (backward) must fit in shared memory.
#include <algorithm>

#include "early_start.cuh"
#include "route_rank.cuh"
#include "route_splits.cuh"

namespace fastb {

namespace {

constexpr int kTokensPerBlock = kRouteTokensPerBlock;
constexpr int kGateThreads = 512;   // forward: 16 warps per block
constexpr int kGateBwdThreads = 512;            // backward: at most 16 warps, a thread per 8 columns
constexpr int kGateBwdMaxChunksPerThread = 2;  // backward: hidden <= 2 * 512 * 8 = 8192

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
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Dynamic shared memory: gate [E][H] bf16, norm weight [H] bf16, then what block_stable_ranks needs.
// Blocks walk groups of 16 TPW tokens, a warp takes TPW of them at a time (with two, every gate chunk is read and unpacked
// once for both rows). The block that finishes the last group of a routing block (128 tokens) ranks its entries. With one
// block per routing block, 4096 tokens kept 32 SMs busy (117 us) and 32768 tokens made two waves, one of them half
// empty (379 us); bound by the rows' way in and out of HBM otherwise.
// tickets: [0] blocks done, [1 + routing block] groups done; zero before and after.
template <int EMAX, int TPW>
__global__ void __launch_bounds__(kGateThreads) norm_gate_route_kernel(const NormGateArgs a, const SplitsArgs sp, const int with_splits, unsigned int* tickets) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_ranks;
  const int E = a.num_experts, H = a.H, K = a.K;
  uint4* s_gate = reinterpret_cast<uint4*>(smem);                            // [E][H / 8]
  uint4* s_nw = s_gate + static_cast<size_t>(E) * (H / 8);                  // [H / 8]
  int* s_eid = reinterpret_cast<int*>(s_nw + H / 8);                        // [kTokensPerBlock * K]
  const int chunks = H / 8;
  grid_dependency_wait();
  launch_dependents();
  for (int i = threadIdx.x; i < E * chunks; i += blockDim.x) s_gate[i] = __ldg(reinterpret_cast<const uint4*>(a.gate) + i);
  for (int i = threadIdx.x; i < chunks; i += blockDim.x) s_nw[i] = __ldg(reinterpret_cast<const uint4*>(a.norm_w) + i);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kGroup = kGateThreads / 32 * TPW;
  static_assert(kTokensPerBlock % kGroup == 0, "a group lies in one routing block");
  // Logits of one token are spread over the lanes' partial sums: reduce, publish, choose the top k.
  auto finish = [&](int t, const float (&acc)[EMAX]) {
    float raw = -INFINITY;  // lane e ends up with logit e
#pragma unroll
    for (int e = 0; e < EMAX; ++e) {
      if (e >= E) break;
      const float v = warp_sum(acc[e]);
      if (lane == e) raw = v;
    }
    if (lane < E) a.logits[static_cast<long long>(t) * E + lane] = raw;
    if (raw != raw) raw = -INFINITY;  // NaN counts as -inf: the selection stays total
    float sel = lane < E ? raw + (a.bias ? a.bias[lane] : 0.0f) : -INFINITY;
    if (sel != sel) sel = -INFINITY;
    int my_e;
    float my_w;
    const float sel1[1] = {sel}, raw1[1] = {lane < E ? raw : -INFINITY};
    route::warp_topk<1>(sel1, raw1, E, K, my_e, my_w);
    if (lane < K) {
      a.topk_idx[static_cast<long long>(t) * K + lane] = my_e;
      a.topk_w[static_cast<long long>(t) * K + lane] = my_w;
    }
  };
  for (int t0 = blockIdx.x * kGroup; t0 < a.T; t0 += gridDim.x * kGroup) {
    const int ta = t0 + warp * TPW;
    if (ta < a.T) {
      const uint4* row[TPW];
      bool live[TPW];
#pragma unroll
      for (int j = 0; j < TPW; ++j) {
        live[j] = ta + j < a.T;
        row[j] = reinterpret_cast<const uint4*>(a.h + static_cast<long long>(live[j] ? ta + j : ta) * H);  // a dead second token re-reads the first
      }
      float ss[TPW], r[TPW];
#pragma unroll
      for (int j = 0; j < TPW; ++j) ss[j] = 0.0f;
      constexpr int U = 4;
      for (int c0 = lane; c0 < chunks; c0 += 32 * U) {
        uint4 v[U][TPW];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < TPW; ++j) v[u][j] = c0 + 32 * u < chunks ? __ldg(row[j] + c0 + 32 * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < TPW; ++j) {
            float f[8];
            unpack8(v[u][j], f);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss[j] = fmaf(f[i], f[i], ss[j]);
          }
      }
#pragma unroll
      for (int j = 0; j < TPW; ++j) {
        r[j] = rsqrtf(warp_sum(ss[j]) / static_cast<float>(H) + a.eps);
        if (lane == 0 && live[j]) a.rstd[ta + j] = r[j];
      }
      // second pass over the rows (in L1 or L2): normalised rows out, logits accumulated against the gate rows
      float acc[TPW][EMAX];
#pragma unroll
      for (int j = 0; j < TPW; ++j)
#pragma unroll
        for (int e = 0; e < EMAX; ++e) acc[j][e] = 0.0f;
      uint4 nx[TPW];
#pragma unroll
      for (int j = 0; j < TPW; ++j) nx[j] = __ldg(row[j] + lane);
      for (int c = lane; c < chunks; c += 32) {
        uint4 cur[TPW];
#pragma unroll
        for (int j = 0; j < TPW; ++j) {
          cur[j] = nx[j];
          if (c + 32 < chunks) nx[j] = __ldg(row[j] + c + 32);
        }
        float w[8], y[TPW][8];
        unpack8(s_nw[c], w);
#pragma unroll
        for (int j = 0; j < TPW; ++j) {
          float f[8];
          unpack8(cur[j], f);
#pragma unroll
          for (int i = 0; i < 8; ++i) y[j][i] = bf16_round(f[i] * r[j] * w[i]);  // normalised and scaled in fp32, rounded once
          if (live[j]) reinterpret_cast<uint4*>(a.hn + static_cast<long long>(ta + j) * H)[c] = pack8(y[j]);
        }
#pragma unroll
        for (int e = 0; e < EMAX; ++e) {
          if (e >= E) break;
          float g[8];
          unpack8(s_gate[static_cast<size_t>(e) * chunks + c], g);
#pragma unroll
          for (int j = 0; j < TPW; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[j][e] = fmaf(y[j][i], g[i], acc[j][e]);
        }
      }
#pragma unroll
      for (int j = 0; j < TPW; ++j)
        if (live[j]) finish(ta + j, acc[j]);
    }
    const int rb = t0 / kTokensPerBlock, rows = min(kTokensPerBlock, a.T - rb * kTokensPerBlock), groups = (rows + kGroup - 1) / kGroup;
    __syncthreads();
    if (threadIdx.x == 0) { __threadfence(); s_ranks = atomicInc(tickets + 1 + rb, groups - 1) == static_cast<unsigned>(groups - 1); __threadfence(); }
    __syncthreads();
    if (s_ranks) {
      const long long first = static_cast<long long>(rb) * kTokensPerBlock * K;
      for (int i = threadIdx.x; i < kTokensPerBlock * K; i += blockDim.x) s_eid[i] = i < rows * K ? __ldcg(a.topk_idx + first + i) : -1;
      __syncthreads();
      route::block_stable_ranks(s_eid, reinterpret_cast<unsigned short*>(s_eid + kTokensPerBlock * K), E, K, a.slot_in_block + first, a.block_cnt + static_cast<long long>(rb) * E);
    }
  }
  if (with_splits && route::last_block(tickets)) route::splits_block(sp, reinterpret_cast<int*>(smem));
}

// Dynamic shared memory: gate [E][H] bf16, norm weight [H] bf16, then fp32 accumulators d_gate [E][H], d_nw [H].
// A block walks its tokens two at a time (one where a thread owns two chunks) and every thread owns the same 16-byte column chunks for all of them, so the
// gradient partials in shared memory are updated with plain read-modify-writes (no two threads ever touch the same word);
// the row-wide sums the RMSNorm backward needs are one block reduction per step. Bound by latency: rows are requested
// a step ahead, and the tokens' few scalars are turned into logit gradients for 32 tokens at a time (read token by token,
// they alone cost a dependent trip to L2 each: 3.6 us a token, 807 us for 32768). Narrow rows run in narrow blocks, several
// per SM. Each block leaves its partial sums; fold_gate_grads_kernel adds them up in a fixed order.
constexpr int kGateBwdBatch = 32;
template <int C>
__global__ void __launch_bounds__(kGateBwdThreads) norm_gate_bwd_kernel(const NormGateBwdArgs a) {
  constexpr int B = C == 1 ? 2 : 1;   // tokens per step
  constexpr int kMaxK = 8;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float s_part[2][B][kGateBwdThreads / 32];
  __shared__ float s_dl[kGateBwdBatch][kMaxK], s_rstd[kGateBwdBatch];
  __shared__ int s_ex[kGateBwdBatch][kMaxK];
  const int E = a.num_experts, H = a.H, K = a.K, nt = blockDim.x, nwarps = blockDim.x >> 5;
  const int chunks = H / 8;
  uint4* s_gate = reinterpret_cast<uint4*>(smem);
  uint4* s_nw = s_gate + static_cast<size_t>(E) * chunks;
  float* s_dgate = reinterpret_cast<float*>(s_nw + chunks);  // [E][H]
  float* s_dnw = s_dgate + static_cast<size_t>(E) * H;       // [H]
  grid_dependency_wait();
  launch_dependents();
  for (int i = threadIdx.x; i < E * chunks; i += nt) s_gate[i] = __ldg(reinterpret_cast<const uint4*>(a.gate) + i);
  for (int i = threadIdx.x; i < chunks; i += nt) s_nw[i] = __ldg(reinterpret_cast<const uint4*>(a.norm_w) + i);
  for (int i = threadIdx.x; i < (E + 1) * H; i += nt) s_dgate[i] = 0.0f;  // d_gate and d_nw are contiguous
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Every block has an equal share of the tokens (no second, partly filled wave).
  const int per = (a.T + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int t0 = blockIdx.x * per;
  const int n_tok = max(0, min(per, a.T - t0));
  const int nc = (chunks - static_cast<int>(threadIdx.x) + nt - 1) / nt;   // my chunks are threadIdx.x + nt * i, i < nc <= C
  uint4 nx[B][C], ng[B][C];
  auto request = [&](int lt) {
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const long long t = t0 + min(lt + b, n_tok - 1);
      const uint4* hrow = reinterpret_cast<const uint4*>(a.h + t * H);
      const uint4* grow = reinterpret_cast<const uint4*>(a.grad_hn + t * H);
#pragma unroll
      for (int i = 0; i < C; ++i)
        if (i < nc) { nx[b][i] = __ldg(hrow + threadIdx.x + nt * i); ng[b][i] = __ldg(grow + threadIdx.x + nt * i); }
    }
  };
  if (n_tok > 0) request(0);
  for (int lt = 0; lt < n_tok; lt += B) {
    if (lt % kGateBwdBatch == 0) {
      // gradients of the selected logits of the next tokens: w = softmax(l_sel)  =>  dl_j = w_j (gw_j - sum_i w_i gw_i)
      __syncthreads();
      for (int q = threadIdx.x; q < kGateBwdBatch; q += nt) {
        if (lt + q < n_tok) {
          const long long tj = static_cast<long long>(t0 + lt + q) * K;
          float w[kMaxK], gw[kMaxK], dotw = 0.0f;
#pragma unroll
          for (int j = 0; j < kMaxK; ++j)
            if (j < K) { w[j] = __ldg(a.topk_w + tj + j); gw[j] = __ldg(a.grad_w + tj + j); dotw = fmaf(w[j], gw[j], dotw); }
#pragma unroll
          for (int j = 0; j < kMaxK; ++j)
            if (j < K) {
              const int e = __ldg(a.topk_idx + tj + j);
              const bool in_range = e >= 0 && e < E;
              s_dl[q][j] = in_range ? w[j] * (gw[j] - dotw) : 0.0f;
              s_ex[q][j] = in_range ? e : 0;
            }
          s_rstd[q] = __ldg(a.rstd + t0 + lt + q);
        } else {
          for (int j = 0; j < K; ++j) { s_dl[q][j] = 0.0f; s_ex[q][j] = 0; }
          s_rstd[q] = 0.0f;   // a token past the end adds nothing
        }
      }
      __syncthreads();
    }
    uint4 cx[B][C], cg[B][C];
#pragma unroll
    for (int b = 0; b < B; ++b)
#pragma unroll
      for (int i = 0; i < C; ++i) { cx[b][i] = nx[b][i]; cg[b][i] = ng[b][i]; }
    if (lt + B < n_tok) request(lt + B);
    // pass 1 over my chunks: s = sum(dxhat * xhat), the gate / norm-weight gradient partials; keeps
    // dxhat = d(hn) * w of my chunks for pass 2
    float s[B], kdx[B][C][8];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      s[b] = 0.0f;
      const int q = (lt + b) % kGateBwdBatch;   // B divides the batch
      const float rstd = s_rstd[q];
#pragma unroll
      for (int ci = 0; ci < C; ++ci) {
        if (ci >= nc) break;
        const int c = threadIdx.x + nt * ci;
        float x[8], w[8], g[8], xh[8], hn[8];
        unpack8(cx[b][ci], x);
        unpack8(s_nw[c], w);
        unpack8(cg[b][ci], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) { xh[i] = x[i] * rstd; hn[i] = bf16_round(xh[i] * w[i]); }  // hn as the forward pass rounded it
        for (int j = 0; j < K; ++j) {
          const float dl = s_dl[q][j];
          const int ex = s_ex[q][j];
          float v[8];
          unpack8(s_gate[static_cast<size_t>(ex) * chunks + c], v);
          // a chunk's first four accumulators sit in the row's first half, the other four in its second
          // half: a warp's 16-byte accesses are then contiguous (no two-way bank conflict)
          float4* dg = reinterpret_cast<float4*>(s_dgate + static_cast<size_t>(ex) * H) + c;
          float4 d0 = dg[0], d1 = dg[chunks];
          d0.x = fmaf(dl, hn[0], d0.x); d0.y = fmaf(dl, hn[1], d0.y); d0.z = fmaf(dl, hn[2], d0.z); d0.w = fmaf(dl, hn[3], d0.w);
          d1.x = fmaf(dl, hn[4], d1.x); d1.y = fmaf(dl, hn[5], d1.y); d1.z = fmaf(dl, hn[6], d1.z); d1.w = fmaf(dl, hn[7], d1.w);
          dg[0] = d0; dg[chunks] = d1;
#pragma unroll
          for (int i = 0; i < 8; ++i) g[i] = fmaf(dl, v[i], g[i]);
        }
        float4* dn = reinterpret_cast<float4*>(s_dnw) + c;
        float4 n0 = dn[0], n1 = dn[chunks];
        n0.x = fmaf(g[0], xh[0], n0.x); n0.y = fmaf(g[1], xh[1], n0.y); n0.z = fmaf(g[2], xh[2], n0.z); n0.w = fmaf(g[3], xh[3], n0.w);
        n1.x = fmaf(g[4], xh[4], n1.x); n1.y = fmaf(g[5], xh[5], n1.y); n1.z = fmaf(g[6], xh[6], n1.z); n1.w = fmaf(g[7], xh[7], n1.w);
        dn[0] = n0; dn[chunks] = n1;
#pragma unroll
        for (int i = 0; i < 8; ++i) { kdx[b][ci][i] = g[i] * w[i]; s[b] = fmaf(kdx[b][ci][i], xh[i], s[b]); }
      }
    }
    const int buf = (lt / B) & 1;   // two buffers: the next step's partials never overwrite sums still being read
#pragma unroll
    for (int b = 0; b < B; ++b) {
      s[b] = warp_sum(s[b]);
      if (lane == 0) s_part[buf][b][warp] = s[b];
    }
    __syncthreads();
    // pass 2, from registers: d(h) = rstd * (dxhat - xhat * s) (+ the gradient that reaches h past the norm)
#pragma unroll
    for (int b = 0; b < B; ++b) {
      if (lt + b >= n_tok) break;
      float tot = 0.0f;
      for (int i = 0; i < nwarps; ++i) tot += s_part[buf][b][i];
      tot /= static_cast<float>(H);
      const float rstd = s_rstd[(lt + b) % kGateBwdBatch];
      const long long t = t0 + lt + b;
      uint4* orow = reinterpret_cast<uint4*>(a.grad_h + t * H);
#pragma unroll
      for (int ci = 0; ci < C; ++ci) {
        if (ci >= nc) break;
        float x[8], o[8];
        unpack8(cx[b][ci], x);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rstd * (kdx[b][ci][i] - x[i] * rstd * tot);
        if (a.residual != nullptr) {
          float q[8];
          unpack8(__ldg(reinterpret_cast<const uint4*>(a.residual + t * H) + threadIdx.x + nt * ci), q);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = bf16_round(o[i]) + q[i];   // the sum of two bf16 gradients
        }
        orow[threadIdx.x + nt * ci] = pack8(o);
      }
    }
  }
  __syncthreads();
  float* mine = a.partials + static_cast<size_t>(blockIdx.x) * (E + 1) * H;
  for (int i = threadIdx.x; i < (E + 1) * H / 4; i += nt) reinterpret_cast<float4*>(mine)[i] = reinterpret_cast<const float4*>(s_dgate)[i];
}

// Sums the blocks' partials: d_gate and d_norm_w as bf16, or added to fp32. Rows of d_gate and d_nw are contiguous ((E + 1) rows of
// H); the half-row split of the accumulators is undone on the way out. A block takes 128 float4 columns, its eight rows of
// threads an eighth of the partials each.
__global__ void __launch_bounds__(1024) fold_gate_grads_kernel(const float* __restrict__ partials, int blocks, int E, int H, __nv_bfloat16* __restrict__ d_gate, __nv_bfloat16* __restrict__ d_nw,
                                                               float* __restrict__ f_gate, float* __restrict__ f_nw) {
  __shared__ float4 s[8][128];
  const int x = threadIdx.x & 127, y = threadIdx.x >> 7, n4 = (E + 1) * H / 4, i = blockIdx.x * 128 + x;
  float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  grid_dependency_wait();
  launch_dependents();
  if (i < n4)
    for (int b = y; b < blocks; b += 8) {
      const float4 p = __ldcs(reinterpret_cast<const float4*>(partials) + static_cast<size_t>(b) * n4 + i);
      v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
    }
  s[y][x] = v;
  __syncthreads();
  if (y != 0 || i >= n4) return;
  for (int k = 1; k < 8; ++k) { v.x += s[k][x].x; v.y += s[k][x].y; v.z += s[k][x].z; v.w += s[k][x].w; }
  const int row = i / (H / 4), p = i % (H / 4);               // float4 position in the row
  const int half = p / (H / 8), q = p % (H / 8);              // accumulators 4 half .. 4 half + 3 of chunk q
  const size_t col = static_cast<size_t>(row < E ? row : 0) * H + q * 8 + half * 4;
  if (d_gate != nullptr) {
    uint2 o;
    *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>((row < E ? d_gate : d_nw) + col) = o;
  } else {
    float* f = (row < E ? f_gate : f_nw) + col;
    f[0] += v.x; f[1] += v.y; f[2] += v.z; f[3] += v.w;
  }
}

}  // namespace

size_t norm_gate_smem_bytes(int E, int H, int K, bool backward) {
  const size_t base = (static_cast<size_t>(E) + 1) * H * 2;
  return backward ? base + (static_cast<size_t>(E) + 1) * H * 4 : base + route::rank_smem_bytes(E, K);
}

int norm_gate_tickets(int T) { return 1 + (T + kTokensPerBlock - 1) / kTokensPerBlock; }

cudaError_t launch_norm_gate_route(const NormGateArgs& a, const SplitsArgs* sp, unsigned int* tickets, cudaStream_t stream) {
  if (a.num_experts < 1 || a.num_experts > 32 || a.K < 1 || a.K > a.num_experts || a.K > 32 || a.H % 256) return cudaErrorInvalidValue;
  if (tickets == nullptr || (sp != nullptr && (sp->num_experts != a.num_experts || sp->block_cnt != a.block_cnt))) return cudaErrorInvalidValue;
  const size_t smem = std::max(norm_gate_smem_bytes(a.num_experts, a.H, a.K, false), sp ? route::splits_smem_bytes(sp->world, a.num_experts) : size_t{0});
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  if (a.T == 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  auto go = [&](auto kern, int tokens_per_group) {
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    int per_sm = 1;
    if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kGateThreads, smem);
    if (err != cudaSuccess) return err;
    const int blocks = std::min((a.T + tokens_per_group - 1) / tokens_per_group, sms * std::max(per_sm, 1));
    err = launch_early(kern, dim3(blocks), kGateThreads, smem, stream, a, sp ? *sp : SplitsArgs{}, sp ? 1 : 0, tickets);
    note_launch();
    return err;
  };
  // Two tokens a warp save a quarter of the arithmetic; below two groups of 32 per SM the tokens are better spread out.
  const bool two = a.T >= 64 * sms;
  constexpr int one_group = kGateThreads / 32;
  if (a.num_experts <= 8) return two ? go(norm_gate_route_kernel<8, 2>, 2 * one_group) : go(norm_gate_route_kernel<8, 1>, one_group);
  if (a.num_experts <= 16) return two ? go(norm_gate_route_kernel<16, 2>, 2 * one_group) : go(norm_gate_route_kernel<16, 1>, one_group);
  return go(norm_gate_route_kernel<32, 1>, one_group);
}

int norm_gate_bwd_blocks(int T, int H, int E, int sms) {
  const int threads = std::min(kGateBwdThreads, (H / 8 + 31) / 32 * 32);
  const int fit = static_cast<int>(std::max<size_t>(1, (220 * 1024) / norm_gate_smem_bytes(E, H, 1, true)));
  const int per_sm = std::min({fit, kGateBwdThreads / threads, 4});
  return std::max(1, std::min(sms * per_sm, (T + 7) / 8));   // at least eight tokens per block: each leaves (E + 1) x H partial sums
}

cudaError_t launch_norm_gate_bwd(const NormGateBwdArgs& a, int blocks, cudaStream_t stream) {
  if (a.num_experts < 1 || a.num_experts > 32 || a.K < 1 || a.K > 8 || a.H % 256 || a.H > kGateBwdMaxChunksPerThread * kGateBwdThreads * 8) return cudaErrorInvalidValue;
  if (a.partials == nullptr || blocks < 1 || ((a.d_gate_bf16 != nullptr) == (a.d_gate != nullptr))) return cudaErrorInvalidValue;
  const size_t smem = norm_gate_smem_bytes(a.num_experts, a.H, a.K, true);
  if (smem > 220 * 1024) return cudaErrorInvalidValue;
  if (a.T <= 0) return cudaSuccess;
  const int threads = std::min(kGateBwdThreads, (a.H / 8 + 31) / 32 * 32);
  auto* kern = a.H / 8 > kGateBwdThreads ? norm_gate_bwd_kernel<2> : norm_gate_bwd_kernel<1>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  e = launch_early(kern, dim3(blocks), threads, smem, stream, a);
  if (e != cudaSuccess) return e;
  e = launch_early(fold_gate_grads_kernel, dim3(((a.num_experts + 1) * a.H / 4 + 127) / 128), 1024, 0, stream, a.partials, blocks, a.num_experts, a.H, a.d_gate_bf16, a.d_norm_w_bf16, a.d_gate, a.d_norm_w);
  note_launch(2);
  return e;
}

}  // namespace fastb
