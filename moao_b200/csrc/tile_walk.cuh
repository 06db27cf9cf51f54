// Order in which a tensor-core product visits the 128 (or 256) x 256 tiles of C
// that are written, shared by the kernels that must agree on it.
#ifndef MOAO_TILE_WALK_CUH
#define MOAO_TILE_WALK_CUH

#include <algorithm>

namespace moao {

constexpr int kWalkTileN = 256;          // columns of C per tile
constexpr int kBandRows = 2048;          // rows of C per band of the tile order
constexpr int kMaxBands = 64;

// Walk over the tiles of C that are written (decode_tile).
struct TileWalk {
  int lower;               // 1: only C(r, c) with r + diag_off >= c
  int diag_off;
  int tile_m;              // rows of C per tile (128, or 256 for CTA pairs)
  int tiles_m, tiles_n;
  int total_tiles;         // tiles that intersect the written part of C
  int band;                // row tiles per band of the tile order
  int band_start[kMaxBands + 1];  // tiles before each band
};

// First row tile of column tile nt that reaches the written (lower) part.
__device__ __forceinline__ int first_mt(const TileWalk& p, int nt) {
  if (!p.lower) return 0;
  const int num = nt * kWalkTileN - p.diag_off - (p.tile_m - 1);
  return num <= 0 ? 0 : (num + p.tile_m - 1) / p.tile_m;
}

// v-th tile of the walk over the tiles that are written. The row tiles are
// taken in bands of p.band (about 2,048 rows); a band is walked column by
// column and each column down the band's rows. A wave of the persistent grid
// then covers a block of roughly 2,048 rows by 2,300 columns of C, whose A rows
// and B rows stay in L2 while its tiles run (a column-major walk over all rows
// streams every A row through L2 in every wave).
__device__ __forceinline__ void decode_tile(const TileWalk& p, int v, int* mt, int* nt) {
  int b = 0;
  while (b + 1 < kMaxBands && p.band_start[b + 1] <= v && b + 1 < (p.tiles_m + p.band - 1) / p.band)
    ++b;
  v -= p.band_start[b];
  const int r0 = b * p.band, r1 = min(r0 + p.band, p.tiles_m), h = r1 - r0;
  // columns whose first written row tile is at or above r0 hold all h tiles of the band
  int full = p.tiles_n;
  if (p.lower) {
    const int num = r0 * p.tile_m + p.diag_off + p.tile_m - 1;
    full = num < 0 ? 0 : min(p.tiles_n, num / kWalkTileN + 1);
  }
  if (v < full * h) {
    *nt = v / h;
    *mt = r0 + v % h;
    return;
  }
  v -= full * h;
  for (int c = full; c < p.tiles_n; ++c) {
    const int f = max(r0, first_mt(p, c));
    const int cnt = max(0, r1 - f);
    if (v < cnt || c == p.tiles_n - 1) {
      *nt = c;
      *mt = f + v;
      return;
    }
    v -= cnt;
  }
  *nt = p.tiles_n - 1;
  *mt = r0;
}

// Tile counts and band offsets of the walk over an M x N result's written tiles;
// returns the number of tiles.
inline long fill_walk(TileWalk* p, long M, long N, int lower, int diag_off, int tile_m) {
  p->lower = lower;
  p->diag_off = diag_off;
  p->tile_m = tile_m;
  p->tiles_m = (int)((M + tile_m - 1) / tile_m);
  p->tiles_n = (int)((N + kWalkTileN - 1) / kWalkTileN);
  p->band = std::max(kBandRows / tile_m, (p->tiles_m + kMaxBands - 1) / kMaxBands);
  const int nbands = (p->tiles_m + p->band - 1) / p->band;
  long total = 0;
  for (int b = 0; b < nbands; ++b) {
    p->band_start[b] = (int)total;
    const long r0 = (long)b * p->band, r1 = std::min<long>(r0 + p->band, p->tiles_m);
    for (int nt = 0; nt < p->tiles_n; ++nt) {
      long first = 0;
      if (lower) {
        const long num = (long)nt * kWalkTileN - diag_off - (tile_m - 1);
        first = num <= 0 ? 0 : (num + tile_m - 1) / tile_m;
      }
      total += std::max(0L, r1 - std::max(r0, first));
    }
  }
  for (int b = nbands; b <= kMaxBands; ++b) p->band_start[b] = (int)total;
  p->total_tiles = (int)total;
  return total;
}

}  // namespace moao

#endif  // MOAO_TILE_WALK_CUH
