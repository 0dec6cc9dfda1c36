// Work split of the grouped GEMM whose N dimension is the tokens (grouped_gemm_tokens.cu): which tiles there are, in which
// order, and which part of the reduction of which tile a CTA pair does. Plain arithmetic: the native self-check
// (csrc/sched/selfcheck.cc) walks it on the host over random groups.
#pragma once

#if defined(__CUDACC__)
#define FASTB_HD __host__ __device__
#else
#define FASTB_HD
#endif

namespace fastb {
namespace gemm {

constexpr int kTokAccN = 256;       // most tokens of one accumulator: a tile has one, or two with one read of the weights (tile_n 512)

FASTB_HD constexpr int ceil_to(int x, int q) { return (x + q - 1) / q * q; }
FASTB_HD constexpr int div_up(int a, int b) { return (a + b - 1) / b; }

// Token tiles of a group whose tokens are taken up to `rows` (real rows rounded up to the granule, a multiple of 32): as few
// as hold them, their widths as even as multiples of 32 allow. 1056 tokens are 3 tiles of 224 and 2 of 192, not 4 of 224 and one
// of 160: tiles that run side by side then advance at about one pace and keep sharing operand panels.
FASTB_HD inline int tok_tiles(int rows, int tile_n) { return div_up(rows, tile_n); }
FASTB_HD inline int tok_tile_size(int rows, int tile_n) {   // the widest
  const int t = tok_tiles(rows, tile_n);
  return t > 0 ? ceil_to(div_up(rows, t), 32) : 0;
}
struct TokSpan { int begin, n; };
FASTB_HD inline TokSpan tok_span(int rows, int tile_n, int i) {
  const int t = tok_tiles(rows, tile_n), units = rows / 32, base = units / t, extra = units - base * t;
  return TokSpan{32 * (i * base + (i < extra ? i : extra)), 32 * (base + (i < extra ? 1 : 0))};
}

// How `tiles` tiles of kb_tile reduction blocks are spread over `pairs` CTA pairs. Whole tiles go round robin; where the last
// wave would be partly idle, its tiles are cut along the reduction. A pair that does a part of a tile leaves fp32 partial
// sums, and the pair that arrives last adds them up. Two ways of cutting:
//   stream (no two tiles share weights, i.e. every group fits one token tile): the last full wave and the rest are one sequence
//       of reduction blocks, cut into equal shares wherever the cut falls. Every pair then works equally long. The weights are
//       read once whatever the order, and the tokens stay in L2.
//   parts  (tiles share weights): the rest is cut into as many equal parts as there are pairs for it, part by part: pairs that
//       run side by side stay at the same depth of the reduction and share operand panels in L2. Cut as a stream, a
//       reduction of 28672 over 4096 tokens fell from 1.5 to 1.2 PFLOP/s: each pair fetched panels of its own.
// When a cut pays, in cycles of an SM. A block of n tokens takes 256 + n (its products read 128 rows of operand A and n / 2 of B from shared
// memory); where no tiles share weights, the tiles that are under way also share HBM, which gives one of them a block about every 8 (rest
// tiles: 8 * rest). So the last wave costs kb_tile blocks of max(256 + n, 8 * rest) as it is, and of max((256 + n) * rest / pairs, 8 * rest)
// when cut. The exchange costs, per step of 32 tokens, 800 to leave the sums, 600 to store and 550 per part to read (L2 to an SM: 64 bytes a
// cycle), and 2000 to meet. Counting only idle blocks against 2 + n / 16 blocks, as before, cut weight-bound
// waves for nothing: us before -> after, forward W2 / data gradient of W13 of 8 experts of 4096 x 14336 at 200 tokens 174 -> 159 / 351 -> 289, 512
// tokens 221 -> 188 / 459 -> 347; forward W13 / W2 of 1024 x 3584 at 16 tokens 35 -> 29 / 24 -> 21, 512 tokens 47 -> 37 / 35 -> 29.
FASTB_HD inline int tok_block_cycles(int n) { return kTokAccN + (n < kTokAccN ? n : kTokAccN) + (n > kTokAccN ? 2 * (n - kTokAccN) : 0); }
FASTB_HD inline int tok_exchange_cycles(int n, int parts) {
  return 2000 + div_up(n, n > kTokAccN ? 64 : 32) * (1400 + 550 * parts);   // wide tiles: two groups of warps share the steps
}
struct TokSplit {
  int pairs, kb_tile;
  int whole_tiles;     // tiles done whole: the i-th of them, tile cut_tiles + i, by pair i % pairs
  int cut_tiles;       // the first tiles, done in parts, before the whole ones: their exchange then hides behind the others
  int shares;          // stream: pairs that take a share; parts: parts per tile
  bool stream;
  FASTB_HD static TokSplit make(int tiles, int kb_tile, int pairs, int widest_n, bool share_weights) {
    TokSplit s{pairs, kb_tile, tiles, 0, 1, !share_weights};
    const int rest = tiles % pairs, block = tok_block_cycles(widest_n);
    if (rest == 0 || kb_tile < 2) return s;
    if (share_weights) {
      int most = pairs / rest < kb_tile / 4 ? pairs / rest : kb_tile / 4;
      most = most < 8 ? most : 8;
      int best = 1, best_cycles = kb_tile * block;
      for (int n = 2; n <= most; ++n) {
        const int c = div_up(kb_tile, n) * block + tok_exchange_cycles(widest_n, n);
        if (c < best_cycles) { best = n; best_cycles = c; }
      }
      if (best > 1) { s.whole_tiles = tiles - rest; s.cut_tiles = rest; s.shares = best; }
      return s;
    }
    const int full = tiles / pairs, hbm = 8 * rest, even = div_up(block * rest, pairs);
    const int alone = block > hbm ? block : hbm, cut = even > hbm ? even : hbm;
    if (static_cast<long long>(kb_tile) * (alone - cut) <= tok_exchange_cycles(widest_n, pairs / (full > 0 ? rest + pairs : rest) + 1)) return s;
    s.whole_tiles = full > 1 ? (full - 1) * pairs : 0;
    s.cut_tiles = tiles - s.whole_tiles;
    const long long units = static_cast<long long>(s.cut_tiles) * kb_tile;
    s.shares = units / 4 < pairs ? static_cast<int>(units / 4 > 0 ? units / 4 : 1) : pairs;  // a share is at least four blocks
    return s;
  }
  FASTB_HD long long cut_units() const { return static_cast<long long>(cut_tiles) * kb_tile; }
  FASTB_HD int share_begin(int p) const { return static_cast<int>(cut_units() * p / shares); }
  // The pair whose share holds unit u: the largest p with share_begin(p) <= u.
  FASTB_HD int share_of(int u) const { return static_cast<int>(((static_cast<long long>(u) + 1) * shares - 1) / cut_units()); }
};

// One pair's segments in order: tile, first block, end block, number of parts of the tile, my part, and the pairs that do the
// parts: first_pair + j * pair_step for part j.
struct TokSegment { int tile, kb0, kb1, parts, part, first_pair, pair_step; };
struct TokSegments {
  TokSplit s;
  int pair, next_whole, u, u_end;
  FASTB_HD TokSegments(const TokSplit& split, int pair_) : s(split), pair(pair_), next_whole(pair_), u(0), u_end(0) {
    if (s.cut_tiles == 0) return;
    if (!s.stream) u_end = pair < s.cut_tiles * s.shares ? 1 : 0;
    else if (pair < s.shares) { u = s.share_begin(pair); u_end = s.share_begin(pair + 1); }
  }
  FASTB_HD bool next(TokSegment& g) {
    if (u >= u_end) {
      if (next_whole >= s.whole_tiles) return false;
      g = TokSegment{s.cut_tiles + next_whole, 0, s.kb_tile, 1, 0, pair, 1};
      next_whole += s.pairs;
      return true;
    }
    if (!s.stream) {
      const int t = pair % s.cut_tiles, j = pair / s.cut_tiles;
      g = TokSegment{t, static_cast<int>(static_cast<long long>(s.kb_tile) * j / s.shares), static_cast<int>(static_cast<long long>(s.kb_tile) * (j + 1) / s.shares),
                     s.shares, j, t, s.cut_tiles};
      u = u_end;
      return true;
    }
    const int t = u / s.kb_tile, kb0 = u - t * s.kb_tile;
    const int left = s.kb_tile - kb0, kb1 = kb0 + (u_end - u < left ? u_end - u : left);
    const int lo = s.share_of(t * s.kb_tile), hi = s.share_of((t + 1) * s.kb_tile - 1);
    g = TokSegment{t, kb0, kb1, hi - lo + 1, pair - lo, lo, 1};
    u += kb1 - kb0;
    return true;
  }
};

// Place of tile `local` inside its group: bands of `band` token tiles, token tiles fastest inside a band, so that the
// tiles that run together cover a squarish patch and share their operand panels in L2.
// How many: as the reduction grows, fewer, so that the token panels of a band take at most half of the L2 while the weights
// stream past them; at most 16: every further one saves a reading of the weights. What this saves is the power that moving operands costs,
// and with it clock. 8 experts of 8192, 4096 and 2048 rows of a training step, seconds at the power cap, TFLOP/s at bands of 16, 8, 4
// tiles: reduction of 4096 1280, 1262, 1152; 1265, 1254, 1163; 1276, 1235, 1146; of 14336 1103, 1134, 1073; 1155, 1137, 1123; 1189,
// 1182, 1124; of 28672 981, 1010, 1007; 1052, 1040, 1073; 1098, 1100, 1063. On normal random rows 16 tiles are ahead by 3-5 % at 8192 rows;
// DRAM reads of a reduction of 4096 over 8192 rows at bands of 4, 8, 16, 32 tiles: 2.2, 1.1, 0.7, 1.7 GB an expert.
// Where the weights of a group stay in L2 from band to band nothing is saved by more than 8: 2 experts of 2048 x 4096 and 8192 rows,
// bands of 16 and 8, us: forward 184 -> 182.5, its SwiGLU 191 -> 189.5, data gradient of 4096 186 -> 183.
constexpr int kTokBandBytes = 60 << 20, kTokBandTiles = 16;
FASTB_HD inline int tok_band_tiles(int red_len, int m_tiles) {
  const long long fit = kTokBandBytes / (2ll * red_len * kTokAccN);
  const int most = 512ll * red_len * m_tiles <= kTokBandBytes / 2 ? kTokBandTiles / 2 : kTokBandTiles;
  return fit < 1 ? 1 : fit > most ? most : static_cast<int>(fit);
}
// From how many token tiles of a group on alternating the direction of the reduction pays (grouped_gemm_tokens.cu).
FASTB_HD inline int tok_back_tiles(int red_len, int band_tiles, int tile_n = kTokAccN) {
  return 2ll * red_len * tile_n * band_tiles > kTokBandBytes / 2 ? band_tiles : 1 << 30;
}
// Token tiles of a band of wide tiles (512 tokens). Same operands, 8192 rows, TFLOP/s at 2, 4, 8 and 16 tiles: reduction of 4096 (SwiGLU
// backward) 1151, 1180, 1176, 1117; of 14336 1320, 1342, 1333, 1275; of 28672 1313, 1330, 1305, 1172.
constexpr int kTokWideBandTiles = 4;
// The band of a launch: by the rules above, or of the rows that its caller wants.
FASTB_HD inline int tok_band(int band_rows, int red_len, int m_tiles, int tile_n) {
  const int tile = tile_n > kTokAccN ? tile_n : kTokAccN;
  if (band_rows > 0) return band_rows < tile ? 1 : band_rows / tile;
  return tile_n > kTokAccN ? kTokWideBandTiles : tok_band_tiles(red_len, m_tiles);
}
struct TokPlace { int m, t; };
FASTB_HD inline TokPlace tok_place(int local, int m_tiles, int t_tiles, int band_tiles) {
  const int per_band = band_tiles * m_tiles, band = local / per_band, rem = local - band * per_band;
  const int t0 = band * band_tiles, left = t_tiles - t0, cur = left < band_tiles ? left : band_tiles;
  return TokPlace{rem / cur, t0 + rem % cur};
}

// Rows of group q that are worked on: the real ones, up to a multiple of the granule. Args: TokGemmArgs, or on the host anything with its
// group_off, group_rows, granule, tile_n, m_tiles and band_tiles.
template <class Args>
FASTB_HD inline int tok_rows(const Args& p, int q) { return p.group_rows ? ceil_to(p.group_rows[q], p.granule) : p.group_off[q + 1] - p.group_off[q]; }
template <class Args>
FASTB_HD inline int tok_group_tiles(const Args& p, int q) { return tok_tiles(tok_rows(p, q), p.tile_n) * p.m_tiles; }

// Prefix of the tile counts: entry i holds the tiles of the groups before group i * tok_per_entry (several groups an entry
// when there are more than kTokPrefix).
constexpr int kTokPrefix = 256;
FASTB_HD constexpr int tok_per_entry(int groups) { return div_up(groups, kTokPrefix); }

// Tiles in order, group by group; `locate` wants non-decreasing tile numbers.
struct TokTile { int g, m, row0, n; };            // first row of the tile in the grouped matrix, rows = columns of the MMA
template <class Args>
struct TokTiles {
  const Args& p;
  const int* base;
  int per_entry, entry = 0, g = 0, g_base = 0;
  FASTB_HD TokTile locate(int tile) {
    if (tile >= base[entry + 1]) {
      while (tile >= base[entry + 1]) ++entry;
      g = entry * per_entry; g_base = base[entry];
    }
    int rows = tok_rows(p, g);
    while (tile >= g_base + tok_tiles(rows, p.tile_n) * p.m_tiles) { g_base += tok_tiles(rows, p.tile_n) * p.m_tiles; rows = tok_rows(p, ++g); }
    const TokPlace at = tok_place(tile - g_base, p.m_tiles, tok_tiles(rows, p.tile_n), p.band_tiles);
    const TokSpan span = tok_span(rows, p.tile_n, at.t);
    return TokTile{g, at.m, p.group_off[g] + span.begin, span.n};
  }
};

}  // namespace gemm
}  // namespace fastb
