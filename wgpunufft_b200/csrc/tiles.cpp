// Spreading tiles of a plan and point count: their sides, the records of a part
// and how many parts there can be (which sizes the padded tiles' scratch).
#include <algorithm>
#include <limits>

#include "spread.h"
#include "tc_spread.h"

namespace b200nufft {

namespace {

// Records of one spreading subproblem, at most.
constexpr int32_t kPartCap = 4096;
// Padded tile bytes a spreading CTA may hold, so that two fit on an SM.
constexpr int64_t kTileBytesTarget = 100 * 1024;

int64_t pow2_ceil(int64_t v) {
  int64_t p = 1;
  while (p < v) p <<= 1;
  return p;
}

// Fine cells per point up to which 3D f64 plans spread in registers. Sparser
// tiles leave a CTA per SM waiting for its few records and its write-out, where
// two CTAs of the shared-memory kernel overlap. 256^3 cells, uniform, us per
// transform, registers against shared memory: w 7, 1/64 point per cell 1443 / 1627,
// 1/512 1323 / 1119; w 10, 1/192 1932 / 2654, 1/1536 1750 / 1397. (Scattered
// points: the line is the earlier of that and a 180 x 140 x 200 grid.)
int64_t reg64_cells_per_point(int w) {
  switch (w) {
    case 6: return 128;
    case 8: return 64;
    case 9: return 96;
    case 10:
    case 11: return 768;
    case 12:
    case 13: return 1536;
    default: return 256;  // 5, 7
  }
}

}  // namespace

int64_t reg64_least_points(const GridParams& grid) {
  const int64_t per_point = reg64_cells_per_point(grid.width);
  return (grid.fine_count + per_point - 1) / per_point;
}

TileShape tile_shape(const GridParams& grid, bool f64, bool tensor_cores, const b200nufft_tuning& tuning,
                     int64_t points) {
  TileShape s{};
  const int dim = grid.dimensions, w = grid.width;
  points = std::max<int64_t>(points, 0);
  int64_t tile[3] = {1, 1, 1};
  if (dim == 1) tile[0] = 1024;
  // 2D f32 register runs (w <= 7) slide along the rows of 64 x 64 tiles:
  // a thread's range of consecutive records then spans more starts of a row.
  const bool runs2d = dim == 2 && !f64 && 2 * w * w * 4 < 400;
  if (dim == 2) tile[0] = tile[1] = runs2d ? 64 : 32;
  if (dim == 3) tile[0] = tile[1] = tile[2] = 16;
  if (tuning.tile > 0) {
    for (int a = 0; a < dim; ++a) tile[a] = tuning.tile;
  }
  for (int a = 0; a < dim; ++a) tile[a] = std::min(tile[a], pow2_ceil(grid.fine[a]));
  const bool regs64 = dim == 3 && f64 && w >= kReg64MinWidth && w <= kReg64MaxWidth &&
                      points >= reg64_least_points(grid);
  auto padded_bytes = [&]() {
    int64_t cells = 1;
    for (int a = 0; a < dim; ++a) cells *= tile[a] + w - 1;
    return cells * 16;
  };
  if (regs64) {
    // Tiles spread in registers have the one shape that fills them.
    tile[0] = kReg64Planes - w + 1;
    tile[1] = 8 * reg64_blocks_y(w) - w + 1;
    tile[2] = 8 * reg64_blocks_z(w) - w + 1;
  } else if (tensor_cores) {
    // The tensor-core spreader's own shape: 16 cells x 22 - w rows.
    tile[0] = kTcTileX;
    tile[1] = tc_tile_rows(w);
  } else {
    while (padded_bytes() > kTileBytesTarget) {
      int largest = dim - 1;
      for (int a = dim - 1; a >= 0; --a) {
        if (tile[a] > tile[largest]) largest = a;
      }
      if (tile[largest] == 1) break;
      tile[largest] /= 2;
    }
  }
  s.regs64 = regs64 ? 1 : 0;
  s.tile_count = 1;
  s.padded_cells = 1;
  s.rows = 1;
  int64_t tiles_per_bin = 1;
  for (int a = 0; a < 3; ++a) {
    s.tile[a] = static_cast<int32_t>(tile[a]);
    s.pad[a] = a < dim ? static_cast<int32_t>(tile[a] + w - 1) : 1;
    s.ntiles[a] = a < dim ? static_cast<int32_t>((grid.fine[a] + tile[a] - 1) / tile[a]) : 1;
    if (a >= dim) continue;
    s.tile_count *= s.ntiles[a];
    s.padded_cells *= s.pad[a];
    const int64_t side = int64_t(1) << grid.axis[a].shift;
    // Tiles that a bin can meet, and bins that a tile can: tiles of no whole
    // number of bins (or bins of no whole number of tiles) share some.
    if (tile[a] % side != 0) tiles_per_bin *= side % tile[a] == 0 ? side / tile[a] : (side + tile[a] - 2) / tile[a] + 1;
    if (a > 0) s.rows *= tile[a] % side == 0 ? tile[a] / side : (side % tile[a] == 0 ? 1 : (tile[a] + side - 2) / side + 1);
  }
  // Parts of a few thousand records at most, fewer for small point sets so that
  // about four CTAs per SM have work. On one-cell bins holding eight or more
  // points per cell, consecutive records share their start: parts sized for
  // one CTA per SM give every thread runs several times longer, and the
  // warps' flushes, which would otherwise all land on the same few windows,
  // fall on more cells and come less often.
  // (Register runs are taken in 1D, and in 2D while the 2 w^2 accumulators
  // fit: spread_run in spread.cu.)
  const bool runs = dim == 1 || (dim == 2 && 2 * w * w * (f64 ? 8 : 4) < 400);
  bool one_cell_bins = true;
  for (int a = 0; a < dim; ++a) one_cell_bins = one_cell_bins && grid.axis[a].shift == 0;
  const bool crowded = runs && one_cell_bins && points >= 8 * grid.fine_count;
  // 3D parts stay within the 2048 records that crowded tiles bucket in shared
  // memory, 2D f64 parts of w >= kStrip64MinWidth within those that the strips
  // order (kStripMaxRecords); 1D and 2D f32 parts take up to 16384 records, so that
  // a thread's register runs can reach 64 records in crowded tiles; other f64
  // parts kPartCap, the register tiles' too, whose padded cells are up to twice
  // as many.
  const bool strips64 = dim == 2 && f64 && w >= kStrip64MinWidth;
  s.cap_max = (dim == 3 && !regs64) || strips64 ? kStripMaxRecords : (f64 ? kPartCap : 16384);
  s.cap_ctas = tuning.ctas_per_sm * 148;
  s.cap_ctas_crowded = tuning.crowded_ctas_per_sm * 148;
  s.crowded_points = runs && one_cell_bins ? 8 * grid.fine_count : std::numeric_limits<int64_t>::max();
  const int64_t ctas = crowded ? s.cap_ctas_crowded : s.cap_ctas;
  const int64_t cap = (std::max<int64_t>(points, 1) + ctas - 1) / ctas;
  s.part_cap = static_cast<int32_t>(std::min<int64_t>(s.cap_max, std::max<int64_t>(256, (cap + 255) / 256 * 256)));
  // The device sizes the parts from the points within reach; the host bounds the
  // parts for any count up to `points`: valid / cap(valid) is at most most_ctas, or
  // points / cap_max once the cap saturates. A bin's records count in every tile
  // that the bin meets. The register tiles, which rarely are whole bins and whose
  // padded cells are large, size their parts from the records so counted
  // (cap_parts) instead: a part that passes over other tiles' records is longer, but
  // no scratch is kept for them.
  const int64_t most_ctas = std::max(s.cap_ctas, s.cap_ctas_crowded);
  // Crowded sets get up to twice as many register tiles' parts, so that these come
  // out no longer than others' for the records passed over (128^3 modes, w 10,
  // clustered, 1/16 point per cell: 2453 -> 2257 us per transform).
  const int64_t ctas_worth = regs64 ? std::min(std::max(most_ctas, points / 512), 2 * most_ctas) : most_ctas;
  const int64_t whole = std::max<int64_t>(ctas_worth, (points + s.cap_max - 1) / s.cap_max);
  s.cap_parts = regs64 ? whole : 0;
  // (A part but for a tile's last holds at least 256 records.)
  s.part_bound = s.tile_count + std::min((regs64 ? 1 : tiles_per_bin) * whole, tiles_per_bin * points / 256) + 1;
  return s;
}

}  // namespace b200nufft

extern "C" int b200nufft_internal_tile_shape(int32_t dimensions, int32_t f64, int32_t width, const int64_t* fine,
                                             const int64_t* bin_side, int64_t points, int64_t* out) {
  using namespace b200nufft;
  GridParams grid{};
  grid.dimensions = dimensions;
  grid.width = width;
  grid.fine_count = 1;
  for (int a = 0; a < dimensions; ++a) {
    grid.fine[a] = fine[a];
    grid.fine_count *= fine[a];
    while ((int64_t{1} << grid.axis[a].shift) < bin_side[a]) ++grid.axis[a].shift;
  }
  const b200nufft_tuning defaults{0, 4, 1, 16};
  const TileShape s = tile_shape(grid, f64 != 0, false, defaults, points);
  const int64_t values[] = {s.regs64, s.tile[0], s.tile[1], s.tile[2], s.tile_count, s.padded_cells, s.rows,
                            s.part_bound, s.cap_parts};
  std::copy(std::begin(values), std::end(values), out);
  return 0;
}
