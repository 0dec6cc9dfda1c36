// Tile enumeration of the grouped GEMM kernels, usable from host code (the native self-check walks
// it exhaustively) and from the kernels.
#pragma once

#if defined(__CUDACC__)
#define FASTB_HD __host__ __device__
#else
#define FASTB_HD
#endif

namespace fastb {
namespace gemm {

constexpr int kWalkBK = 64;  // reduction step of the kernels (BK)

struct TileCoord {
  int g, m_idx, n_idx;   // group, tile row inside the group (of the fixed dim for wgrad), tile column
  int row0;              // first row of the group in the grouped matrix
  int red_blocks;        // BK steps of the reduction
};

// Walks the tile space group by group; inside a group, in bands of kBandRows rows: all column tiles
// of a band are visited (m fastest inside the band) before the next band starts. The tiles that
// run at the same time then form a roughly square patch of the output, which minimises the
// operand bytes a wave pulls from DRAM (a wave of p x q tiles reads p A-panels and q B-panels).
// TILE_M is 128 (one CTA) or 256 (CTA pair). `locate` must be called with non-decreasing tile
// indices (each role of a CTA steps its own walker by the grid stride).
// For weight gradients that is 16 tiles: 8 experts of 8192 rows of a training step, seconds at the power cap, TFLOP/s at bands of 4, 8
// and 16 tiles, down projection 1193, 1284, 1292, gate|up 1258, 1269, 1265; at 4096 rows 1208, 1290, 1316 and 1320, 1292, 1299.
constexpr int kDefaultBandRows = 4096;
// Weight gradients: whether every other wave walks the reduction (the group's rows) backwards, from the panel ends that the wave before
// left in L2. It pays where a band's panels are more than a quarter of the 126 MB L2, i.e. above 4096 rows in the default
// band. 8 experts of 8192 rows of a training step, seconds at the power cap, always forwards -> this: 1240 -> 1292 TFLOP/s (down
// projection), 1198 -> 1262 (gate|up). On normal random rows, forwards against every other wave backwards: 6144 rows 1309, 1326 and
// 1252, 1256; 5120 rows 1331, 1336 and 1271, 1270; 4096 rows 1350, 1337 and 1291, 1285; 3072 rows 1344, 1333 and 1318, 1305.
constexpr long long kBackBandBytes = 32ll << 20;
FASTB_HD inline bool wgrad_back(int red_blocks, int band_rows) {
  return 2ll * red_blocks * kWalkBK * (band_rows > 0 ? band_rows : kDefaultBandRows) > kBackBandBytes;
}
template <int TILE_M>
struct TileWalker {
  const int* off; int G, tiles_n, fixed_m, red_len; bool wgrad; int band_rows;
  const int* rows = nullptr;  // wgrad, optional: real rows per group; the reduction stops at the block that holds the last of them
  int g = 0, base = 0;
  FASTB_HD bool locate(int tile, TileCoord& c) {
    while (g < G) {
      const int r0 = off[g], r1 = off[g + 1];
      const int mt = wgrad ? fixed_m : (r1 - r0) / TILE_M;
      const int cnt = mt * tiles_n;
      if (tile < base + cnt) {
        const int local = tile - base;
        const int want = (band_rows > 0 ? band_rows : kDefaultBandRows) / TILE_M;
        const int kBand = want > 1 ? want : 1;
        const int band = local / (kBand * tiles_n), rem = local % (kBand * tiles_n);
        const int m0 = band * kBand, left = mt - m0, cur = kBand < left ? kBand : left;
        c.g = g; c.n_idx = rem / cur; c.m_idx = m0 + rem % cur; c.row0 = r0;
        c.red_blocks = !wgrad ? red_len / kWalkBK : rows ? (rows[g] + kWalkBK - 1) / kWalkBK : (r1 - r0) / kWalkBK;
        return true;
      }
      base += cnt; ++g;
    }
    return false;
  }
};

}  // namespace gemm
}  // namespace fastb
