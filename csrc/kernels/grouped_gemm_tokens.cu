// Grouped bf16 GEMM with the weights as operand A and the tokens as operand B: out[token, feature] is computed as
// W x X^T tile by tile, 256 features (M) by up to 256 or 512 tokens (N, in one or two accumulators), on CTA pairs (tcgen05.mma.cta_group::2).
//
//   kForward : out[rows of g, N]  = x[rows of g, K]  * W_g[N, K]^T     (A K-major)      store, or SwiGLU of gate and up
//   kDgrad   : out[rows of g, K]  = dy[rows of g, N] * W_g[N, K]       (A MN-major)     store, or SwiGLU backward
//
// Why the tokens are N. A tile of M = 256 costs the same whatever is in it, and an expert's tokens rarely fill a multiple
// of 256: 625 tokens took three 256-row tiles, 23 % of the work on padding; a decode step of one token did
// the work of 256. N is free in steps of 16, so a tile is as wide as the tokens it holds (in steps of 32, the rows of a
// TMA store). The second loss was the last wave: 32 weight tiles of the down projection on 74 pairs, or 384 on 74, leave
// half of a wave idle; what does not fill whole waves is cut into equal shares of the reduction (TokSplit), whose fp32
// partial sums are exchanged through L2.
// What bounds it: up to about 200 tokens per expert the weights' bytes (HBM), above that the tensor pipe.
// Measured before (tokens as M, 256-row tiles) and after, us, both forward projections of 8 experts of 4096 x 14336: 1 token
// 179 -> 137, 64 tokens 521 -> 465 (2.8 GB of weights: 6.1 TB/s), 625 tokens per expert 1518 -> 1321; at full 256-token
// tiles equal within 2 %.
//
// Each CTA of a pair loads its 128 features of A and its half of the tokens of B; the leader issues one M = 256 MMA per 16-wide
// k step; a CTA's accumulator is [128 features (TMEM lanes)] x [n tokens (columns)], the transpose of what is stored. The
// epilogue reads it in 16 x 256-bit fragments (a thread holds pairs of tokens of a feature), packs the pairs to bf16 and
// lets stmatrix.trans write [token][64 features] boxes in shared memory, which leave by TMA stores of 64 x 32; the saved
// gate|up tiles of the SwiGLU backward come in by TMA loads and ldmatrix.trans. Shared memory is what the epilogue must spare:
// the operand tiles' way in and out takes 128 bytes a cycle already, all that there is. Written value by value (2-byte
// stores, half-filled wavefronts) the same epilogue slowed the SwiGLU backward from 743 to 896 us.
// SwiGLU wants gate and up of a feature in one thread: the A tile is fetched through a 5-D tensor map as [16 gate rows | 16 up
// rows] x 4, so that the two 16-lane halves of a warp's fragments are gate and up of the same features.
//
// Wide tiles (SUB = 2, 512 tokens, both accumulators of 256 columns). Seconds of full tiles run at the power cap, and what a
// 256 x 256 tile spends beside the products is operand traffic: 64 KiB from L2 per block of 64 k, and both operands read from shared memory
// for every product, which with the loads' writes fills its 128 bytes a cycle (pipe "active" cycles were 9 % above the products').
// With 512 tokens a block is 96 KiB for twice the products, and operand A is read once for two of them (the collector buffer): L2 to SM
// traffic -25 %, active cycles 4 % above the products'. 8 experts x 8192 rows, seconds at the cap, TFLOP/s, 256 -> 512: reduction of 14336
// 1255 -> 1335; of 28672 1182 -> 1330; 4096 with the SwiGLU backward 1145 -> 1180. The price is that no accumulator is free while a tile
// is multiplied: what the epilogue needs of tensor memory stands still. So it reads both accumulators into registers (eight warps, with the
// registers of the others; 104 to 156 bytes a thread of them are spilled, 128 values beside a step of 32), one a little earlier than the
// other, and stores from there. The SwiGLU forward, 4 to 6 thousand
// cycles of special-function work before its second accumulator is free, gains nothing (reduction of 4096: 1390 -> 1365) but for groups that
// one wide tile holds and one of 256 does not. Which calls take wide tiles: ops/gemm.py.
//
// Barriers as in grouped_gemm_pair.cu. Every wait is bounded. No load is multicast.
#include "gemm_epilogue_tma.cuh"
#include "early_start.cuh"
#include "token_walker.h"

namespace fastb {

namespace {

using namespace ptx;
using namespace gemm;

constexpr int kPairM = 256, kHalfM = 128;
constexpr int kMaxStages = 10;
constexpr int kAccStages = 2;
constexpr int kTmemCols = 512;
constexpr int kABytes = kHalfM * BK * 2;          // 16 KiB
__host__ __device__ constexpr int stage_bytes(int tile_n) { return kABytes + tile_n / 2 * BK * 2; }   // B: half of the widest tile's tokens
// Warps: TMA, MMA, then four epilogue warps; for wide tiles two groups of four from warp 4 on, whose registers (they hold
// accumulators) come from the first four.
__host__ __device__ constexpr int first_epilogue_warp(int sub) { return sub == 1 ? 2 : 4; }
__host__ __device__ constexpr int threads_for(int sub) { return 32 * first_epilogue_warp(sub) + 128 * sub; }
constexpr int kLaunchRegs = 168, kOtherRegs = 72, kEpilogueRegs = 216;   // a thread, wide tiles
static_assert(kOtherRegs + 2 * kEpilogueRegs <= 3 * kLaunchRegs && threads_for(2) * kLaunchRegs <= 65536, "what the epilogue takes, the others have given");
constexpr int kStepTokens = 32;                   // tokens per epilogue step = rows of a TMA store
constexpr int kBox = kStepTokens * 128;           // 4 KiB: 32 tokens x 64 features

struct __align__(8) TokCtl {
  uint64_t full[kMaxStages], empty[kMaxStages], acc_full[kAccStages], acc_empty[kAccStages], epi_load[2], meet;
  uint32_t tmem_base;
  int abort_flag, last_arrived, widest, share_weights;
  int base[kTokPrefix + 1];                         // tiles of the groups before entry i
};
__host__ __device__ constexpr int epi_boxes(GemmEpilogue e) { return e == GemmEpilogue::kStore ? 2 : e == GemmEpilogue::kSwiGLU ? 3 : 4; }
constexpr int kSmemLimit = 227 * 1024;
constexpr int other_bytes(GemmEpilogue e) { return 2 * epi_boxes(e) * kBox + 1024 + static_cast<int>(sizeof(TokCtl)); }
// Operand stages that fit. Tiles of up to 256 tokens: 6 of 32 KiB. Where few tokens meet the weights, the loop is bound by
// HBM and wants weight bytes in flight: tiles of up to 64 tokens leave room for 10 stages of 20 KiB.
constexpr int stages_for(GemmEpilogue e, int tile_n) {
  const int n = (kSmemLimit - other_bytes(e)) / stage_bytes(tile_n);
  return n < kMaxStages ? n : kMaxStages;
}
constexpr int smem_bytes(GemmEpilogue e, int tile_n) { return stages_for(e, tile_n) * stage_bytes(tile_n) + other_bytes(e); }
static_assert(stages_for(GemmEpilogue::kSwiGLUBwd, kTokAccN) == 6 && stages_for(GemmEpilogue::kSwiGLU, 64) == 10, "stages at both ends of the range");
static_assert(stages_for(GemmEpilogue::kSwiGLUBwd, 2 * kTokAccN) == 4, "stages of wide tiles");
static_assert(kAccStages * kTokAccN <= kTmemCols, "two accumulators of 256 columns: of two tiles in turn, or both of a wide tile");
static_assert(kTokPartialFloats == kHalfM * kTokAccN, "a partial is one CTA's accumulator");

__device__ __forceinline__ void tma_load_5d_pair(void* smem_dst, const CUtensorMap* map, int x0, int x1, int x2, int x3, int x4, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(x4)
      : "memory");
}

// 16 lanes x 32 columns of fp32: thread T gets, for the 8-column block j, r[4 j + {0, 1}] = lane T / 4, columns 8 j + 2 (T % 4)
// + {0, 1}, and r[4 j + {2, 3}] = the same columns of lane T / 4 + 8.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
        "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Four 8 x 8 bf16 matrices; thread i names row i % 8 of matrix i / 8. Transposed: register m of thread T holds rows 2 (T % 4) +
// {0, 1} of column T / 4 of matrix m.
__device__ __forceinline__ void stmatrix_trans(uint32_t smem, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(smem), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void ldmatrix_trans(uint32_t smem, uint32_t (&v)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(smem) : "memory");
}
// Row address of this thread for 16 tokens from 16 jj on (matrices: features 0-7 and 8-15 of the first 8 tokens, then of the other 8)
// at feature chunk `chunk` (8 features each) of a swizzled box of [32 tokens][64 features].
__device__ __forceinline__ uint32_t box_row(uint32_t box, int lane, int jj, int chunk) {
  const int t = jj * 16 + ((lane >> 4) << 3) + (lane & 7), ch = chunk + ((lane >> 3) & 1);
  return box + t * 128 + ((ch ^ (t & 7)) << 4);
}
__device__ __forceinline__ float as_f(uint32_t x) { return __uint_as_float(x); }

// Tokens of a tile of n that accumulator `sub` holds.
__device__ __forceinline__ int acc_n(int n, int sub) { return sub == 0 ? min(n, kTokAccN) : max(n - kTokAccN, 0); }

template <GemmMode MODE, GemmEpilogue EPI, int SUB>
__global__ void __launch_bounds__(threads_for(SUB), 1)
grouped_gemm_tokens_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ TokMapsX map_x, const __grid_constant__ CUtensorMap map_c,
                           const __grid_constant__ CUtensorMap map_c2,
                           const TokGemmArgs p) {
  constexpr bool A_MN = MODE == GemmMode::kDgrad;
  constexpr int kRing = epi_boxes(EPI) * kBox;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int stages = p.stages, stage_size = stage_bytes(p.tile_n);
  uint8_t* ring = tiles + stages * stage_size;
  TokCtl* ctl = reinterpret_cast<TokCtl*>(ring + 2 * kRing);
  if (!p.early) grid_dependency_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = static_cast<int>(cluster_cta_rank());  // 0 = leader
  const bool leader = cta == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&ctl->full[s], 1); mbar_init(&ctl->empty[s], 1); }
    for (int a = 0; a < kAccStages; ++a) { mbar_init(&ctl->acc_full[a], 1); mbar_init(&ctl->acc_empty[a], 2 * 4 * SUB); mbar_init(&ctl->epi_load[a], 1); }
    mbar_init(&ctl->meet, 4 * SUB);
    ctl->abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&map_w);
    for (int j = 0; j < kTokBoxes; ++j) prefetch_tmap(&map_x.box[j]);
    prefetch_tmap(&map_c);
    if (EPI != GemmEpilogue::kStore) prefetch_tmap(&map_c2);
  }
  if (warp == 1) { tmem_alloc_pair(&ctl->tmem_base, kTmemCols); tmem_relinquish_pair(); }
  const int per_entry = tok_per_entry(p.num_groups);
  if (warp == 2) {
    // Prefix sums of the tile counts over the groups, the widest tile, and whether any group has several token tiles.
    int run = 0, widest = 0, most = 0;
    const int entries = div_up(p.num_groups, per_entry);
    for (int e0 = 0; e0 < entries; e0 += 32) {
      int mine = 0;
      for (int q = (e0 + lane) * per_entry; q < min((e0 + lane + 1) * per_entry, p.num_groups); ++q) {
        const int rows = tok_rows(p, q);
        mine += tok_group_tiles(p, q);
        widest = max(widest, tok_tile_size(rows, p.tile_n));
        most = max(most, tok_tiles(rows, p.tile_n));
      }
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
      if (e0 + lane < entries) ctl->base[e0 + lane + 1] = run + incl;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    widest = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(widest)));
    most = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(most)));
    if (lane == 0) { ctl->base[0] = 0; ctl->widest = widest; ctl->share_weights = most > 1; }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything arrives on them remotely
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abort_flag = &ctl->abort_flag;

  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const TokSplit split = TokSplit::make(ctl->base[div_up(p.num_groups, per_entry)], p.red_blocks, pairs, ctl->widest, ctl->share_weights != 0);
  TokSegments segs(split, pair);
  TokTiles<TokGemmArgs> walk{p, ctl->base, per_entry};
  TokSegment sg;
  auto give_registers = [] {
    if constexpr (SUB == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
  };
  if (warp == 0) {
    give_registers();
    // ---------------- TMA producer (both CTAs, each for its own halves) ----------------
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      int gated = -1;
      // The first stages' weights do not depend on the kernel before this one: with p.early they are on their way before it has ended.
      bool first = true;
      while (ok && segs.next(sg)) {
        const TokTile tc = walk.locate(sg.tile);
        const int n0 = acc_n(tc.n, 0), half = n0 >> 1, x_row = tc.row0 + cta * half;         // my tokens of the first accumulator
        const int half2 = (tc.n - n0) >> 1, x_row2 = tc.row0 + n0 + cta * half2;             // ... and of a second
        const int feat0 = tc.m * kPairM + cta * kHalfM;
        const uint32_t bytes = 2u * (kABytes + static_cast<uint32_t>(half + half2) * 128u);
        // Where the token panels of a band are a good part of the L2 (p.back_tiles) and a group has several bands, every other
        // wave walks the reduction backwards, from the panel ends that the wave before left in L2: 1093 -> 1132 TFLOP/s at a reduction of
        // 14336 and 985 -> 997 at 28672 over 8192 rows of a training step. Where the tokens stay in L2 anyway there is nothing to win.
        const bool back = sg.parts == 1 && tok_tiles(tok_rows(p, tc.g), p.tile_n) > p.back_tiles && (((sg.tile - split.cut_tiles) / pairs) & 1);
        const int k_step = back ? -BK : BK, blocks = sg.kb1 - sg.kb0;
        int k = back ? (p.red_blocks - 1) * BK : sg.kb0 * BK;   // column of the operands that comes next
        auto load_w = [&](int at, int st) {
          uint8_t* sa = tiles + st * stage_size;
          const uint32_t full_leader = map_to_cta(smem_u32(&ctl->full[st]), 0);
          if (leader) mbar_arrive_expect_tx(&ctl->full[st], bytes);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < kHalfM / 64; ++j)
              tma_load_2d_pair(sa + j * (BK * 128), &map_w, feat0 + j * 64, tc.g * p.w_rows_per_group + at, full_leader);
          } else if (EPI == GemmEpilogue::kSwiGLU) {
            tma_load_5d_pair(sa, &map_w, at, 0, 0, cta * 4, tc.g * p.m_tiles + tc.m, full_leader);
          } else {
            tma_load_2d_pair(sa, &map_w, at, tc.g * p.w_rows_per_group + feat0, full_leader);
          }
        };
        const int early = first ? min(blocks, stages) : 0;   // blocks whose weights are requested now
        for (int i = 0; i < early; ++i) load_w(k + i * k_step, i);
        if (first) { grid_dependency_wait(); first = false; }
        if (p.gate_counter != nullptr) {
          // Arrival gate: per group, or (gate_tile_rows > 0) per tile of that many rows of the grouped matrix that this one touches.
          const int lo = p.gate_tile_rows > 0 ? tc.row0 / p.gate_tile_rows : tc.g, hi = p.gate_tile_rows > 0 ? (tc.row0 + tc.n - 1) / p.gate_tile_rows : tc.g;
          for (int q = lo; ok && q <= hi; ++q) {
            const int slot = min(q, p.gate_slots - 1);
            if (slot == gated) continue;
            if (!(ok = wait_ge_bounded(p.gate_counter + slot, p.gate_target[slot], p.status, kSiteRailArrive, slot, p.timeout_ns))) { *abort_flag = 1; break; }
            asm volatile("fence.proxy.async.global;" ::: "memory");
            gated = slot;
          }
          if (!ok) break;
        }
        for (int i = 0; i < blocks; ++i, k += k_step) {
          if (i >= early) {
            if (!(ok = mbar_wait_bounded(&ctl->empty[s], ph ^ 1, abort_flag, p.status, 100 + s, p.timeout_ns))) break;
            load_w(k, s);
          }
          uint8_t* sb = tiles + s * stage_size + kABytes;
          const uint32_t full_leader = map_to_cta(smem_u32(&ctl->full[s]), 0);
          // As few loads as half has bits set. What this thread does per block bounds the loop of narrow tiles: in boxes of 32
          // rows (four loads for 224 tokens instead of three) projections over 625 tokens per group took 5 % longer.
          auto load_x = [&](uint8_t* to, int rows, int row) {
            int at = 0;
#pragma unroll
            for (int j = kTokBoxes - 1; j >= 0; --j)
              if (rows & (16 << j)) { tma_load_2d_pair(to + at * 128, &map_x.box[j], k, row + at, full_leader); at += 16 << j; }
          };
          load_x(sb, half, x_row);
          if (SUB == 2) load_x(sb + kTokAccN / 2 * 128, half2, x_row2);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    give_registers();
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (leader && elect_one()) {
      int s = 0;
      uint32_t ph = 0, acc_it = 0;
      bool ok = true;
      while (ok && segs.next(sg)) {
        const TokTile tc = walk.locate(sg.tile);
        const bool both = SUB == 2 && tc.n > kTokAccN;
        const uint32_t it0 = acc_it;
        acc_it += both ? 2 : 1;
        const uint32_t idesc0 = make_idesc_bf16(kPairM, acc_n(tc.n, 0), A_MN, false), idesc1 = make_idesc_bf16(kPairM, acc_n(tc.n, 1), A_MN, false);
        const uint32_t d0 = tmem_base + it0 % kAccStages * kTokAccN, d1 = tmem_base + (it0 + 1) % kAccStages * kTokAccN;
        auto claim = [&](int sub) {               // the epilogue has read the accumulator's last tile
          const int a = (it0 + sub) % kAccStages;
          ok = mbar_wait_bounded(&ctl->acc_empty[a], (((it0 + sub) / kAccStages) & 1) ^ 1, abort_flag, p.status, 200 + a, p.timeout_ns);
          tc_fence_after_sync();
        };
        // One block: operand A times the tokens of the first accumulator, of the second, or of both (operand A is then read once per k step).
        enum { kFirst, kSecond, kBoth };
        auto multiply = [&](int which, bool fresh) {
          const uint32_t sa = smem_u32(tiles + s * stage_size), sb = sa + kABytes, sb1 = sb + kTokAccN / 2 * 128;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, BK * 128, 1024) : make_smem_desc(sa + k * 32, 16, 1024);
            const uint32_t add = (!fresh || k != 0) ? 1u : 0u;
            if (SUB == 2 && which == kBoth) {
              mma_bf16_ss_pair_fill_a(d0, da, make_smem_desc(sb + k * 32, 16, 1024), idesc0, add);
              mma_bf16_ss_pair_last_a(d1, da, make_smem_desc(sb1 + k * 32, 16, 1024), idesc1, add);
            } else if (SUB == 1 || which == kFirst) {
              mma_bf16_ss_pair(d0, da, make_smem_desc(sb + k * 32, 16, 1024), idesc0, add);
            } else {
              mma_bf16_ss_pair(d1, da, make_smem_desc(sb1 + k * 32, 16, 1024), idesc1, add);
            }
          }
        };
        claim(0);
        if (!ok) break;
        for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
          if (!(ok = mbar_wait_bounded(&ctl->full[s], ph, abort_flag, p.status, 300 + s, p.timeout_ns))) break;
          tc_fence_after_sync();
          const bool head = kb == sg.kb0, tail = kb + 1 == sg.kb1;
          if (both && !head && !tail) {
            multiply(kBoth, false);
          } else {
            // The first block and the last go to one accumulator after the other: the first is full that much earlier, and the next tile can run
            // in it that much longer before it needs the second. Longer ends hide more of the epilogue but lose the saving of kBoth and hold
            // stages: two blocks at either end were equal, eight 5 % slower.
            multiply(kFirst, head);
            if (tail) mma_commit_pair(&ctl->acc_full[it0 % kAccStages], 0x3);
            if (both) {
              if (head) { claim(1); if (!ok) break; }
              multiply(kSecond, head);
            }
          }
          mma_commit_pair(&ctl->empty[s], 0x3);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        if (both) mma_commit_pair(&ctl->acc_full[(it0 + 1) % kAccStages], 0x3);
      }
    }
  } else if (warp < first_epilogue_warp(SUB)) {
    give_registers();
  } else {
    if constexpr (SUB == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
    // ---------------- epilogue (both CTAs, each for its 128 features) ----------------
    // A wide tile has two groups of four warps, which take the 32-token steps in turn: a group owns half of the ring, and one group
    // converts while the other's stores and loads are under way.
    const int quarter = warp & 3, group = (warp - first_epilogue_warp(SUB)) >> 2;
    const int et = (threadIdx.x - 32 * first_epilogue_warp(SUB)) & 127;   // 0..127 in the group
    const bool issuer = et == 0;
    const int first_step = SUB == 1 ? 0 : group;
    grid_dependency_wait();   // what is written below may still be read by earlier kernels
    launch_dependents();
    // The other arrival counters are cleared for the next launch; this launch's are back at zero once all parts have arrived.
    if (blockIdx.x == 0 && group == 0)
      for (int i = et; i < p.num_counters; i += 128) p.counters_next[i] = 0u;
    uint32_t acc_it = 0, ring_n = 0, load_ph = 0u;   // load_ph: one parity bit per half of the ring
    bool ok = true;
    // All epilogue warps, twice per part of a tile (phases 0 and 1 of the barrier). Two groups wait with a limit: one of them may have given up.
    auto meet = [&](uint32_t phase) {
      if (SUB == 1) { epi_bar(); return; }
      __syncwarp();
      if (!ok) return;
      if (lane == 0) mbar_arrive(&ctl->meet);
      ok = mbar_wait_bounded(&ctl->meet, phase, abort_flag, p.status, 600 + phase, p.timeout_ns);
    };
    while (ok && segs.next(sg)) {
      const TokTile tc = walk.locate(sg.tile);
      const int accs = SUB == 2 && tc.n > kTokAccN ? 2 : 1;    // accumulators that the tile fills
      const uint32_t it0 = acc_it;
      acc_it += accs;
      auto steps_of = [&](int sub) { return acc_n(tc.n, sub) / kStepTokens; };
      auto acc_row = [&](int sub) { return tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + (it0 + sub) % kAccStages * kTokAccN; };
      auto wait_acc = [&](int sub) {
        const int a = (it0 + sub) % kAccStages;
        ok = mbar_wait_bounded(&ctl->acc_full[a], ((it0 + sub) / kAccStages) & 1, abort_flag, p.status, 400 + a, p.timeout_ns);
        tc_fence_after_sync();
      };
      auto release_acc = [&](int sub) {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl->acc_empty[(it0 + sub) % kAccStages]), 0));
      };
      const size_t part_step = static_cast<size_t>(sg.pair_step) * SUB * kTokPartialFloats;   // from there on, in float4s: four partials per pair
      if (sg.parts > 1) {
        // Part of a tile: leave my sums (values in the order in which the same thread of another CTA holds them), and go on only
        // if all other parts are there already.
        for (int sub = 0; sub < accs; ++sub) {
          wait_acc(sub);
          if (!ok) break;
          float4* out = reinterpret_cast<float4*>(p.partials + ((static_cast<size_t>(pair * 2 + (sg.part == 0 ? 1 : 0)) * 2 + cta) * SUB + sub) * kTokPartialFloats) + et;
          const uint32_t t_row = acc_row(sub);
          for (int st = first_step; st < steps_of(sub); st += SUB) {
            uint32_t r[32];
            tmem_ld_16x32(t_row + st * kStepTokens, r);
            tmem_ld_16x32(t_row + (16u << 16) + st * kStepTokens, r + 16);
            tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 8; ++q)
              __stcg(out + static_cast<size_t>(st * 8 + q) * kHalfM, make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3])));
          }
          release_acc(sub);
        }
        __threadfence();
        meet(0);
        if (ok && issuer && group == 0) ctl->last_arrived = atomicInc(p.counters + sg.tile * 2 + cta, static_cast<unsigned>(sg.parts - 1)) == static_cast<unsigned>(sg.parts - 1);
        meet(1);
        if (!ok) break;
        if (!ctl->last_arrived) continue;
        __threadfence();
      }
      const int feat0 = tc.m * kPairM + cta * kHalfM;          // my 128 features
      auto row_of = [&](int sub, int st) { return tc.row0 + sub * kTokAccN + st * kStepTokens; };
      // 32 tokens of my features, (r[0..15]: lanes 0-15 of the warp, r[16..31]: lanes 16-31): from tensor memory, or the parts in
      // the order of the reduction.
      auto load_acc = [&](int sub, int st, uint32_t (&r)[32]) {
        if (sg.parts == 1) {
          tmem_ld_16x32(acc_row(sub) + st * kStepTokens, r);
          tmem_ld_16x32(acc_row(sub) + (16u << 16) + st * kStepTokens, r + 16);
          tmem_wait_ld();
          return;
        }
        const float* parts0 = p.partials + (static_cast<size_t>(cta) * SUB + sub) * kTokPartialFloats;
        const float4* first = reinterpret_cast<const float4*>(parts0 + static_cast<size_t>(sg.first_pair * 2 + 1) * 2 * SUB * kTokPartialFloats) + et;
        const float4* more = reinterpret_cast<const float4*>(parts0 + static_cast<size_t>((sg.first_pair + sg.pair_step) * 2) * 2 * SUB * kTokPartialFloats) + et;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 v = __ldcg(first + static_cast<size_t>(st * 8 + q) * kHalfM);
          r[4 * q] = __float_as_uint(v.x); r[4 * q + 1] = __float_as_uint(v.y); r[4 * q + 2] = __float_as_uint(v.z); r[4 * q + 3] = __float_as_uint(v.w);
        }
        for (int j = 1; j < sg.parts; ++j, more += part_step) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 v = __ldcg(more + static_cast<size_t>(st * 8 + q) * kHalfM);
            r[4 * q] = __float_as_uint(as_f(r[4 * q]) + v.x); r[4 * q + 1] = __float_as_uint(as_f(r[4 * q + 1]) + v.y);
            r[4 * q + 2] = __float_as_uint(as_f(r[4 * q + 2]) + v.z); r[4 * q + 3] = __float_as_uint(as_f(r[4 * q + 3]) + v.w);
          }
        }
      };
      auto to_bf16 = [](const uint32_t (&r)[32], uint32_t* h) {
#pragma unroll
        for (int i = 0; i < 16; ++i) h[i] = pack_bf16(as_f(r[2 * i]), as_f(r[2 * i + 1]));
      };
      // 16 features x 32 tokens (8 bf16 pairs a thread) -> a box, at feature chunk `chunk`.
      auto put = [&](uint32_t box, int chunk, const uint32_t* h) {
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) stmatrix_trans(box_row(box, lane, jj, chunk), h[4 * jj], h[4 * jj + 1], h[4 * jj + 2], h[4 * jj + 3]);
      };
      auto acquire = [&]() {
        if (issuer) bulk_wait_read<SUB == 1 ? 1 : 0>();   // the stores that read this half of the ring are done with it
        group_bar(group);
        return ring + (SUB == 1 ? ring_n & 1u : group) * kRing;
      };
      auto load_gu = [&](int sub, int st) {                    // issuer only: gate and up of my 128 features, saved by the forward pass
        uint8_t* b = ring + (st & 1) * kRing;
        mbar_arrive_expect_tx(&ctl->epi_load[st & 1], 4 * kBox);
#pragma unroll
        for (int q = 0; q < 4; ++q) tma_load_2d(b + q * kBox, &map_c2, 2 * feat0 + q * 64, row_of(sub, st), &ctl->epi_load[st & 1]);
      };
      auto begin_gu = [&](int sub) {
        if (!issuer) return;
        bulk_wait_read<0>();
        if (first_step < steps_of(sub)) load_gu(sub, first_step);
        if (SUB == 1 && steps_of(sub) > 1) load_gu(sub, 1);
      };
      // One step of 32 tokens on its way out: h are its values as bf16 (plain store; SwiGLU backward, whose d(act) the unfused path
      // stores as bf16 too), r its fp32 values (SwiGLU: gate in r[0..15], up in r[16..31]).
      auto emit_bf16 = [&](int sub, int st, const uint32_t* h) {
        const int y = row_of(sub, st);
        if (EPI == GemmEpilogue::kStore) {
          uint8_t* b = acquire();
          const uint32_t sb = smem_u32(b) + (quarter >> 1) * kBox;
          put(sb, (quarter & 1) * 4, h);
          put(sb, (quarter & 1) * 4 + 2, h + 8);
          fence_proxy_async_smem();
          group_bar(group);
          if (issuer) {
            tma_store_2d(&map_c, b, feat0, y);
            tma_store_2d(&map_c, b + kBox, feat0 + 64, y);
            bulk_commit();
          }
          ++ring_n;
          return;
        }
        uint8_t* b = ring + (st & 1) * kRing;
        if (!(ok = mbar_wait_bounded(&ctl->epi_load[st & 1], (load_ph >> (st & 1)) & 1u, abort_flag, p.status, 500, p.timeout_ns))) return;
        load_ph ^= 1u << (st & 1);
        const uint32_t gb = smem_u32(b + (quarter >> 1) * kBox), ub = gb + 2 * kBox;
        uint32_t gv[4][4], uv[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int chunk = (quarter & 1) * 4 + (e >> 1) * 2;
          ldmatrix_trans(box_row(gb, lane, e & 1, chunk), gv[e]);
          ldmatrix_trans(box_row(ub, lane, e & 1, chunk), uv[e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 g2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gv[e][q])), u2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&uv[e][q]));
            const uint32_t da2 = h[4 * e + q];
            float dg[2], du[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float g = i ? g2.y : g2.x, u = i ? u2.y : u2.x;
              const float da = as_f(i ? da2 & 0xFFFF0000u : da2 << 16);
              const float sgm = sigmoid(g);
              const float sl = g * sgm;
              du[i] = da * sl;
              dg[i] = da * u * (sgm + sl * (1.0f - sgm));
            }
            gv[e][q] = pack_bf16(dg[0], dg[1]);
            uv[e][q] = pack_bf16(du[0], du[1]);
          }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int chunk = (quarter & 1) * 4 + (e >> 1) * 2;
          stmatrix_trans(box_row(gb, lane, e & 1, chunk), gv[e][0], gv[e][1], gv[e][2], gv[e][3]);
          stmatrix_trans(box_row(ub, lane, e & 1, chunk), uv[e][0], uv[e][1], uv[e][2], uv[e][3]);
        }
        fence_proxy_async_smem();
        group_bar(group);
        if (issuer) {
#pragma unroll
          for (int q = 0; q < 4; ++q) tma_store_2d(&map_c, b + q * kBox, 2 * feat0 + q * 64, y);
          bulk_commit();
          if (st + 2 < steps_of(sub)) { bulk_wait_read<0>(); load_gu(sub, st + 2); }
        }
      };
      auto emit_swiglu = [&](int sub, int st, const uint32_t (&r)[32]) {
        const int y = row_of(sub, st);
        uint8_t* b = acquire();
        const uint32_t sb = smem_u32(b);
        uint32_t h[16];
        if (p.keep_gate_up) {
          to_bf16(r, h);
          put(sb + kBox, quarter * 2, h);
          put(sb + 2 * kBox, quarter * 2, h + 8);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = pack_bf16(silu(as_f(r[2 * i])) * as_f(r[16 + 2 * i]), silu(as_f(r[2 * i + 1])) * as_f(r[17 + 2 * i]));
        put(sb, quarter * 2, h);
        fence_proxy_async_smem();
        group_bar(group);
        if (issuer) {
          tma_store_2d(&map_c, b, feat0 / 2, y);
          if (p.keep_gate_up) {
            tma_store_2d(&map_c2, b + kBox, tc.m * kPairM + cta * 64, y);
            tma_store_2d(&map_c2, b + 2 * kBox, tc.m * kPairM + kHalfM + cta * 64, y);
          }
          bulk_commit();
        }
        ++ring_n;
      };
      if constexpr (SUB == 1) {
        if (EPI == GemmEpilogue::kSwiGLUBwd) begin_gu(0);       // the saved tiles arrive while the MMAs still run
        if (sg.parts == 1) wait_acc(0);
        for (int st = 0; ok && st < steps_of(0); ++st) {
          uint32_t r[32];
          load_acc(0, st, r);
          if constexpr (EPI == GemmEpilogue::kSwiGLU) emit_swiglu(0, st, r);
          else { uint32_t h[16]; to_bf16(r, h); emit_bf16(0, st, h); }
        }
        if (!ok) break;
        if (sg.parts == 1) release_acc(0);
      } else {
        // The next tile's first accumulator can be multiplied one block ahead of the second (the first and the last block of a tile, see the MMA
        // issuer), so what the tensor pipe waits for is the reading of the second: values move to registers first and leave from there while
        // the next tile is on its way.
        constexpr int kMine = kTokAccN / kStepTokens / SUB;      // steps of a group
        if constexpr (EPI == GemmEpilogue::kSwiGLU) {
          uint32_t keep[kMine][32];                              // the first accumulator; a second leaves straight from tensor memory
          if (sg.parts == 1) {
            wait_acc(0);
            if (!ok) break;
#pragma unroll
            for (int i = 0; i < kMine; ++i) {                    // all of it, whatever part is used
              tmem_ld_16x32(acc_row(0) + (first_step + SUB * i) * kStepTokens, keep[i]);
              tmem_ld_16x32(acc_row(0) + (16u << 16) + (first_step + SUB * i) * kStepTokens, keep[i] + 16);
            }
            tmem_wait_ld();
            release_acc(0);
            if (accs == 2) wait_acc(1);
            if (!ok) break;
          }
          if (accs == 2) {
#pragma unroll 1
            for (int st = first_step; st < steps_of(1); st += SUB) {
              uint32_t r[32];
              load_acc(1, st, r);
              emit_swiglu(1, st, r);
            }
            if (sg.parts == 1) release_acc(1);
          }
#pragma unroll 1
          for (int st = first_step; st < steps_of(0); st += SUB) {
            if (sg.parts > 1) load_acc(0, st, keep[0]);
            emit_swiglu(0, st, keep[0]);
#pragma unroll
            for (int i = 0; i + 1 < kMine; ++i)
#pragma unroll
              for (int q = 0; q < 32; ++q) keep[i][q] = keep[i + 1][q];
          }
        } else {
          uint32_t keep[SUB * kMine][16];
          if (EPI == GemmEpilogue::kSwiGLUBwd) begin_gu(0);
#pragma unroll
          for (int sub = 0; sub < SUB; ++sub) {
            if (sub >= accs) break;
            if (sg.parts == 1) {
              wait_acc(sub);
              if (!ok) break;
#pragma unroll
              for (int i = 0; i < kMine; i += 2) {
                uint32_t r[2][32];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                  tmem_ld_16x32(acc_row(sub) + (first_step + SUB * (i + q)) * kStepTokens, r[q]);
                  tmem_ld_16x32(acc_row(sub) + (16u << 16) + (first_step + SUB * (i + q)) * kStepTokens, r[q] + 16);
                }
                tmem_wait_ld();
                to_bf16(r[0], keep[sub * kMine + i]);
                to_bf16(r[1], keep[sub * kMine + i + 1]);
              }
              release_acc(sub);
            } else {
#pragma unroll
              for (int i = 0; i < kMine; ++i)
                if (first_step + SUB * i < steps_of(sub)) {
                  uint32_t r[32];
                  load_acc(sub, first_step + SUB * i, r);
                  to_bf16(r, keep[sub * kMine + i]);
                }
            }
          }
          if (!ok) break;
          // One copy of the code that stores a step: unrolled, the SwiGLU backward's eight copies did not fit the instruction cache and took
          // twice as long. The registers move up instead.
#pragma unroll 1
          for (int sub = 0; ok && sub < accs; ++sub) {
            if (EPI == GemmEpilogue::kSwiGLUBwd && sub > 0) begin_gu(sub);
#pragma unroll 1
            for (int i = 0; ok && i < kMine; ++i) {
              if (first_step + SUB * i < steps_of(sub)) emit_bf16(sub, first_step + SUB * i, keep[0]);
#pragma unroll
              for (int j = 0; j + 1 < SUB * kMine; ++j)
#pragma unroll
                for (int q = 0; q < 16; ++q) keep[j][q] = keep[j + 1][q];
            }
          }
          if (!ok) break;
        }
      }
    }
    if (issuer) bulk_wait_all();  // every bulk store of this CTA has landed before anything is torn down
  }
  // ---------------- teardown: nobody frees tensor memory while the pair still uses it ----------------
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc_pair(tmem_base, kTmemCols); }
}

template <GemmMode MODE, GemmEpilogue EPI, int SUB>
cudaError_t launch_sub(const TokGemmMaps& m, TokGemmArgs args, int ctas, cudaStream_t stream) {
  auto kern = grouped_gemm_tokens_kernel<MODE, EPI, SUB>;
  args.stages = stages_for(EPI, args.tile_n);
  const int smem = smem_bytes(EPI, args.tile_n);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas & ~1);
  cfg.blockDim = dim3(threads_for(SUB));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1] = early_start_attribute();
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, kern, *m.w, *m.x, *m.c, m.c2 ? *m.c2 : *m.c, args);
  if (e == cudaSuccess) note_launch();
  return e;
}
template <GemmMode MODE, GemmEpilogue EPI>
cudaError_t launch(const TokGemmMaps& m, const TokGemmArgs& args, int ctas, cudaStream_t stream) {
  return args.tile_n > kTokAccN ? launch_sub<MODE, EPI, 2>(m, args, ctas, stream) : launch_sub<MODE, EPI, 1>(m, args, ctas, stream);
}

}  // namespace

cudaError_t launch_grouped_gemm_tokens(GemmMode mode, GemmEpilogue epi, const TokGemmMaps& maps, const TokGemmArgs& args, int ctas, cudaStream_t stream) {
  if (ctas < 2 || args.num_groups < 1 || args.m_tiles < 1 || args.red_blocks < 1 || args.band_tiles < 1) return cudaErrorInvalidValue;
  if (args.tile_n != 64 && args.tile_n != 128 && args.tile_n != kTokAccN && args.tile_n != 2 * kTokAccN) return cudaErrorInvalidValue;
  if ((args.granule != 32 && args.granule != 64) || args.partials == nullptr || args.counters == nullptr || args.counters_next == nullptr) return cudaErrorInvalidValue;
  if (args.num_counters < tok_counters(ctas)) return cudaErrorInvalidValue;
  if (mode == GemmMode::kForward && epi == GemmEpilogue::kStore) return launch<GemmMode::kForward, GemmEpilogue::kStore>(maps, args, ctas, stream);
  if (mode == GemmMode::kForward && epi == GemmEpilogue::kSwiGLU && (args.keep_gate_up != 0) == (maps.c2 != nullptr))
    return launch<GemmMode::kForward, GemmEpilogue::kSwiGLU>(maps, args, ctas, stream);
  if (mode == GemmMode::kDgrad && epi == GemmEpilogue::kStore) return launch<GemmMode::kDgrad, GemmEpilogue::kStore>(maps, args, ctas, stream);
  if (mode == GemmMode::kDgrad && epi == GemmEpilogue::kSwiGLUBwd && maps.c2 != nullptr) return launch<GemmMode::kDgrad, GemmEpilogue::kSwiGLUBwd>(maps, args, ctas, stream);
  return cudaErrorInvalidValue;
}

}  // namespace fastb
