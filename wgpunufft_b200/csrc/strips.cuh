// Type-1 spreading of tiles by small matrix products (mma.sync) over strips
// of support starts.
//
// A tile's support starts are cut into strips; the window sums of a chunk of 8
// points of one strip are products with the points as the contracted index,
// accumulated in a warp's registers over all consecutive chunks of the strip
// and added to the tile's fixed-point cells in shared memory once per strip.
// A point then costs its share of a few matrix instructions instead of w^d
// shared-memory atomics.
//
// A part's records are first ordered by (strip, x) with a stable counting sort
// in shared memory. Chunks are every 8 records from a strip's first; warp w
// takes the chunks that start in the w-th share of the order. So the order of
// all floating-point sums depends on the records alone, and the fixed-point
// tile makes the order of the warps irrelevant.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "device.h"
#include "mma.cuh"
#include "spread.h"

namespace b200nufft {

constexpr int kSpreadThreads = 256;
constexpr int kSpreadWarps = kSpreadThreads / 32;
constexpr int kStripMax = 96;           // strips of a tile, at most

// Last tile whose first part is at or below `part` (one warp). Sets of about
// one part per tile have it near tile `part`, which costs one load's latency
// (on every CTA's critical path); elsewhere the warp narrows the range 33-fold per
// load.
__device__ __forceinline__ int64_t part_tile(const uint32_t* part_start, int64_t tiles, uint32_t part) {
  const int lane = threadIdx.x & 31;
  int64_t low = 0, count = tiles;  // the tile lies in [low, low + count)
  int64_t near = static_cast<int64_t>(part) - 15;
  near = near > tiles - 32 ? tiles - 32 : near;
  near = near < 0 ? 0 : near;
  int64_t step = (count + 32) / 33;
  const int64_t far = (lane + 1) * step;
  const bool near_below = near + lane < tiles && part_start[near + lane] <= part;
  bool below = far < tiles && part_start[far] <= part;
  const int before = __popc(__ballot_sync(0xFFFFFFFFu, near_below));
  if (before > 0 && (before < 32 || near + 32 >= tiles)) return near + before - 1;
  while (count > 1) {
    const int passed = __popc(__ballot_sync(0xFFFFFFFFu, below));
    count = min(step, count - passed * step);
    low += passed * step;
    step = (count + 32) / 33;
    const int64_t probe = low + (lane + 1) * step;
    below = count > 1 && probe < low + count && part_start[probe] <= part;
  }
  return low;
}

// Shared memory of the strips beside the tile: records in strip order, first
// record of every strip, every strip's start cell (x | y << 8 | z << 16) and
// the warps' staged chunks.
struct StripShared {
  uint32_t* sorted;
  uint32_t* start;
  uint32_t* cell;
  float* stage;
};

// Bytes of strip_order's counters.
__host__ __device__ constexpr size_t strip_counter_bytes(int strips, int per_strip) {
  return sizeof(uint32_t) * kSpreadWarps * (static_cast<size_t>(strips) * per_strip + 1);
}

// Orders the part's records by key, stably: key_of(load_of(slot)) lies in
// [0, strips * per_strip), or is negative for a record to skip. Fills sh.sorted
// with slots and sh.start[0, strips]. `count` is scratch of
// strip_counter_bytes(strips, per_strip). The caller synchronizes.
template <typename LoadOf, typename KeyOf>
__device__ __forceinline__ void strip_order(const uint32_t* row_begin, const uint32_t* row_prefix, int rows,
                                            uint32_t record_begin, uint32_t record_end, int strips, int per_strip,
                                            uint32_t* count, const StripShared& sh, LoadOf load_of, KeyOf key_of) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = static_cast<int>(record_end - record_begin);
  const int keys = strips * per_strip, entries = (keys + 1) * kSpreadWarps;
  // Warp w takes w's eighth of the records, a lane every 32nd of it (eight at
  // most), whose slots and keys stay in registers. count[key * warps + warp];
  // the last key collects the skipped records.
  constexpr int kLaneRecords = kStripMaxRecords / kSpreadThreads;
  for (int c = tid; c < entries; c += kSpreadThreads) count[c] = 0u;
  const int per_warp = (n + kSpreadWarps - 1) / kSpreadWarps;
  const int warp_begin = min(n, per_warp * warp), warp_end = min(n, per_warp * (warp + 1));
  uint32_t slot[kLaneRecords];
  int key[kLaneRecords];
  {
    // Rows of the records (the last row starting at or before each).
    int row[kLaneRecords];
#pragma unroll
    for (int i = 0; i < kLaneRecords; ++i) row[i] = 0;
    for (int step = kMaxTileRows / 2; step > 0; step >>= 1) {
      if (step >= rows) continue;
#pragma unroll
      for (int i = 0; i < kLaneRecords; ++i) {
        const uint32_t r = record_begin + warp_begin + lane + 32 * i;
        const int probe = row[i] + step;
        if (probe < rows && row_prefix[probe] <= r) row[i] = probe;
      }
    }
    decltype(load_of(0u)) loaded[kLaneRecords];
#pragma unroll
    for (int i = 0; i < kLaneRecords; ++i) {
      const int r = warp_begin + lane + 32 * i;
      slot[i] = row_begin[row[i]] + (record_begin + r - row_prefix[row[i]]);
      if (r < warp_end) loaded[i] = load_of(slot[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kLaneRecords; ++i) {
      key[i] = -1;
      if (warp_begin + lane + 32 * i < warp_end) {
        const int k = key_of(loaded[i]);
        key[i] = k < 0 ? keys : k;
        atomicAdd(&count[key[i] * kSpreadWarps + warp], 1u);
      }
    }
  }
  __syncthreads();
  // Exclusive scan of the counters, key-major.
  uint32_t* block_sums = sh.sorted;
  const int per = (entries + kSpreadThreads - 1) / kSpreadThreads;
  const int e0 = min(entries, tid * per), e1 = min(entries, e0 + per);
  uint32_t sum = 0;
  for (int c = e0; c < e1; ++c) sum += count[c];
  block_sums[tid] = sum;
  __syncthreads();
  if (warp == 0) {
    constexpr int kPer = kSpreadThreads / 32;
    uint32_t v[kPer];
    uint32_t mine = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      v[k] = block_sums[lane * kPer + k];
      mine += v[k];
    }
    uint32_t x = mine;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, offset);
      if (lane >= offset) x += y;
    }
    uint32_t running = x - mine;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      block_sums[lane * kPer + k] = running;
      running += v[k];
    }
  }
  __syncthreads();
  uint32_t running = block_sums[tid];
  for (int c = e0; c < e1; ++c) {
    const uint32_t v = count[c];
    count[c] = running;
    running += v;
  }
  __syncthreads();
  for (int s = tid; s <= strips; s += kSpreadThreads) sh.start[s] = count[s * per_strip * kSpreadWarps];
  __syncthreads();
  // Stable scatter: equal keys of one step take consecutive places in lane order.
  const unsigned lower = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < kLaneRecords; ++i) {
    if (warp_begin + 32 * i < warp_end) {
      const unsigned same = __match_any_sync(0xFFFFFFFFu, key[i]);
      uint32_t* counter = &count[(key[i] < 0 ? 0 : key[i]) * kSpreadWarps + warp];
      const uint32_t place = key[i] < 0 ? 0u : *counter + __popc(same & lower);
      __syncwarp();
      if (key[i] >= 0) {
        sh.sorted[place] = slot[i];
        if ((same & lower) == 0u) *counter += __popc(same);
      }
      __syncwarp();
    }
  }
}

// A chunk: its strip, its first record in strip order, and the strip's end.
struct StripChunk {
  int strip, at, end;
};

// The chunk after `c`; past the last one, `at` is the number of records.
__device__ __forceinline__ void next_chunk(StripChunk& c, const uint32_t* start, int strips) {
  c.at += 8;
  if (c.at >= c.end) {
    c.at = c.end;
    while (c.at >= c.end && c.strip + 1 < strips) {
      ++c.strip;
      c.end = static_cast<int>(start[c.strip + 1]);
    }
  }
}

// The first chunk that starts at or after record `from`.
__device__ __forceinline__ StripChunk first_chunk(int from, const uint32_t* start, int strips) {
  int low = 0, high = strips - 1;  // last strip starting at or before `from`
  while (low < high) {
    const int mid = (low + high + 1) >> 1;
    if (static_cast<int>(start[mid]) <= from) low = mid; else high = mid - 1;
  }
  const int begin = static_cast<int>(start[low]);
  StripChunk c{low, begin + (from - begin + 7) / 8 * 8, static_cast<int>(start[low + 1])};
  if (c.at >= c.end) {
    c.at -= 8;
    next_chunk(c, start, strips);
  }
  return c;
}

// 3D f32 tiles holding enough points are spread as products of small
// matrices on the tensor cores. The tile's support starts are cut into strips of
// 8 x (9 - w) x (9 - w) cells (x, y, z), whose windows reach 8 + w - 1 planes
// of 8 x 8 cells (y, z). For 8 points of one strip, plane p receives
//   C_p[(y, re/im), z] += sum_k (c wy)[(y, re/im), k] (wx[p] wz)[k, z],
// one 16 x 8 x 8 product (mma m16n8k8) whose left operand all planes share.
// Both operands are split into tf32 high and low parts, and the three
// products hi lo, lo hi, hi hi accumulate from zero, smallest first; the
// chunk's sum joins the plane's f32 registers by a rounded add, so the tensor
// core's truncated accumulation never runs over more than 8 points. The
// registers reach the fixed-point tile when the strip changes: about ten
// shared-memory adds per start cell of the strip instead of w^3 per point.
constexpr int kStripX = 8;            // support starts of a strip along x
// Staged floats of a point: wx[16] - - wy[8] - - wz[8] re im - -: the axes'
// rows start in different banks modulo 8, the points' rows 8 banks apart.
constexpr int kStripStride = 40;
constexpr int kStripY = 18, kStripZ = 28, kStripValue = 36;
constexpr int kStripFloats = 8 * kStripStride;
// Start cells per record up to which a tile takes the strips (below that
// density the products of a strip's few points cost more than their w^3 adds).
__host__ __device__ constexpr int strip_cells_per_record(int w) { return w == 7 ? 5 : 8; }

// Adds a scaled sum to the tile's two words of a cell: v = 65536 h + l with
// |l| <= 32768, both rounded to integers by adding 1.5 x 2^23 (|v| < 2^38).
__device__ __forceinline__ void add_split(uint32_t* acc, int span, int part, int c, float h, float l) {
  atomicAdd(&acc[(2 * part) * span + c], __float_as_uint(l) - 0x4B400000u);
  atomicAdd(&acc[(2 * part + 1) * span + c], __float_as_uint(h) - 0x4B400000u);
}

template <int W>
__device__ void spread_strips3(const SpreadParams& sp, const PreparedWindow<3>* win3, const float2* sv,
                               const uint32_t* perm, const uint32_t* row_begin, const uint32_t* row_prefix,
                               int rows, const int* origin, uint32_t record_begin, uint32_t record_end,
                               uint32_t* acc, int span, int pitch0, int pitch01, const StripShared& sh,
                               float scale_lo, float scale_hi) {
  constexpr int S = 9 - W;
  constexpr int P = kStripX + W - 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = sp.tile[0], t1 = sp.tile[1], t2 = sp.tile[2];
  const int nx = (t0 + kStripX - 1) / kStripX, ny = (t1 + S - 1) / S, nz = (t2 + S - 1) / S;
  const int strips = nx * ny * nz;
  for (int s = tid; s < strips; s += kSpreadThreads) {
    const int yz = s / nx;
    sh.cell[s] = static_cast<uint32_t>((s - yz * nx) * kStripX | (yz % ny) * S << 8 | (yz / ny) * S << 16);
  }
  // The counters lie in the tile region, which is cleared afterwards.
  strip_order(
      row_begin, row_prefix, rows, record_begin, record_end, strips, kStripX, acc, sh,
      [&](uint32_t slot) { return __ldg(reinterpret_cast<const int4*>(win3 + slot)); },
      [&](const int4& start) {
        const int x = start.x - origin[0], y = start.y - origin[1], z = start.z - origin[2];
        const bool inside = start.x >= 0 && x >= 0 && x < t0 && y >= 0 && y < t1 && z >= 0 && z < t2;
        const int strip = x / kStripX + nx * (y / S + ny * (z / S));
        return inside ? strip * kStripX + x % kStripX : -1;
      });
  __syncthreads();
  {
    uint4* acc16 = reinterpret_cast<uint4*>(acc);
    for (int c = tid; c < span; c += kSpreadThreads) acc16[c] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();

  const int spread = static_cast<int>(sh.start[strips]);
  const int share = (spread + kSpreadWarps - 1) / kSpreadWarps;
  const int from = min(spread, share * warp), to = min(spread, share * (warp + 1));
  if (from >= to) return;
  StripChunk k0 = first_chunk(from, sh.start, strips);
  if (k0.at >= to) return;
  const int g = lane >> 2, t = lane & 3;  // fragment row / column group; also staged point g, role t
  float* st = sh.stage + warp * kStripFloats;
  float2 acc_p[P][2];  // plane p: (z = 2t, 2t + 1) of y = g, real and imaginary
#pragma unroll
  for (int p = 0; p < P; ++p) acc_p[p][0] = acc_p[p][1] = make_float2(0.0f, 0.0f);
  // Lane (g, t) stages axis t of point g (t < 3) or its strength (t = 3):
  // starts, offsets and point indexes are loaded two chunks ahead, the
  // strength one chunk ahead.
  const int32_t* words = reinterpret_cast<const int32_t*>(win3) + t;
  auto fetch = [&](const StripChunk& c, int32_t& first, int32_t& second) {
    const int at = c.at + g;
    if (c.at < to && at < c.end) {
      const uint32_t slot = sh.sorted[at];
      if (t < 3) {
        first = __ldg(words + static_cast<int64_t>(slot) * 8);
        second = __ldg(words + static_cast<int64_t>(slot) * 8 + 4);
      } else {
        first = static_cast<int32_t>(__ldg(perm + slot));
      }
    }
  };
  auto strength_of = [&](const StripChunk& c, int32_t point, float2& v) {
    if (t == 3 && c.at < to && c.at + g < c.end) v = __ldg(sv + static_cast<uint32_t>(point));
  };
  int32_t a0 = 0, b0 = 0, a1 = 0, b1 = 0;
  float2 c0 = make_float2(0.0f, 0.0f);
  StripChunk k1 = k0;
  next_chunk(k1, sh.start, strips);
  fetch(k0, a0, b0);
  fetch(k1, a1, b1);
  strength_of(k0, a0, c0);
  const int role_origin = t == 0 ? origin[0] : (t == 1 ? origin[1] : origin[2]);
  float* const rowp = st + g * kStripStride + (t == 0 ? 0 : (t == 1 ? kStripY : (t == 2 ? kStripZ : kStripValue)));
  const float* const p0 = st + t * kStripStride;
  const float* const p1 = p0 + 4 * kStripStride;
  int plane_lo = P, plane_hi = -1;
  for (;;) {
    const StripChunk now = k0;
    const int32_t start = a0, offset_bits = b0;
    const float2 c = c0;
    const int points = min(now.end - now.at, 8);
    // Advance the pipeline.
    strength_of(k1, a1, c0);
    k0 = k1;
    a0 = a1;
    b0 = b1;
    next_chunk(k1, sh.start, strips);
    fetch(k1, a1, b1);
    const uint32_t cell = sh.cell[now.strip];
    // Stage the chunk: rows of zeros with the weights at their place.
    {
      float4* st4 = reinterpret_cast<float4*>(st);
      __syncwarp();  // the previous chunk's rows are read
      st4[lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      st4[lane + 32] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (lane < kStripFloats / 4 - 64) st4[lane + 64] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      __syncwarp();
    }
    const int place = start - role_origin - static_cast<int>((cell >> (8 * t)) & 255u);
    if (g < points) {
      if (t < 3) {
        float w[W];
        horner32_window<W>(__int_as_float(offset_bits), sp.grid.horner32, w);
#pragma unroll
        for (int j = 0; j < W; ++j) rowp[place + j] = w[j];
      } else {
        *reinterpret_cast<float2*>(rowp) = make_float2((c.x * scale_lo) * scale_hi, (c.y * scale_lo) * scale_hi);
      }
    }
    const int lo = __shfl_sync(0xFFFFFFFFu, place, 0);
    const int hi = __shfl_sync(0xFFFFFFFFu, place, 4 * (points - 1)) + W - 1;
    __syncwarp();
    plane_lo = min(plane_lo, lo);
    plane_hi = max(plane_hi, hi);
    uint32_t ah[4], al[4];
    {
      const float y0 = p0[kStripY + g], y1 = p1[kStripY + g];
      const float2 q0 = *reinterpret_cast<const float2*>(p0 + kStripValue);
      const float2 q1 = *reinterpret_cast<const float2*>(p1 + kStripValue);
      split_tf32(q0.x * y0, ah[0], al[0]);
      split_tf32(q0.y * y0, ah[1], al[1]);
      split_tf32(q1.x * y1, ah[2], al[2]);
      split_tf32(q1.y * y1, ah[3], al[3]);
    }
    const float z0 = p0[kStripZ + g], z1 = p1[kStripZ + g];
#pragma unroll
    for (int q = 0; q < P; q += 2) {
      if (lo <= q + 1 && hi >= q) {
        const float2 x0 = *reinterpret_cast<const float2*>(p0 + q);
        const float2 x1 = *reinterpret_cast<const float2*>(p1 + q);
        float d[2][4];
        uint32_t bh[2][2], bl[2][2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          split_tf32((k == 0 ? x0.x : x0.y) * z0, bh[k][0], bl[k][0]);
          split_tf32((k == 0 ? x1.x : x1.y) * z1, bh[k][1], bl[k][1]);
          d[k][0] = d[k][1] = d[k][2] = d[k][3] = 0.0f;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) mma_tf32(d[k], ah, bl[k][0], bl[k][1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) mma_tf32(d[k], al, bh[k][0], bh[k][1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) mma_tf32(d[k], ah, bh[k][0], bh[k][1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (q + k < P) {
            acc_p[q + k][0] = __fadd2_rn(acc_p[q + k][0], make_float2(d[k][0], d[k][1]));
            acc_p[q + k][1] = __fadd2_rn(acc_p[q + k][1], make_float2(d[k][2], d[k][3]));
          }
        }
      }
    }
    const bool done = k0.at >= to;
    if (done || k0.strip != now.strip) {
      // The strip's planes to the tile: cell (x = p, y = g, z = 2t, 2t + 1).
      const int y = static_cast<int>((cell >> 8) & 255u) + g, z = static_cast<int>(cell >> 16) + 2 * t;
      const int base = static_cast<int>(cell & 255u) + y * pitch0 + z * pitch01;
      const bool in0 = y < sp.pad[1] && z < sp.pad[2], in1 = y < sp.pad[1] && z + 1 < sp.pad[2];
      constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23
      const float2 magic = make_float2(kMagic, kMagic), minus = make_float2(-kMagic, -kMagic);
      const float2 down = make_float2(1.0f / 65536.0f, 1.0f / 65536.0f), up = make_float2(-65536.0f, -65536.0f);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        if (p >= plane_lo && p <= plane_hi) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 h = __ffma2_rn(acc_p[p][i], down, magic);
            const float2 l = __fadd2_rn(__ffma2_rn(__fadd2_rn(h, minus), up, acc_p[p][i]), magic);
            if (in0) add_split(acc, span, i, base + p, h.x, l.x);
            if (in1) add_split(acc, span, i, base + p + pitch01, h.y, l.y);
            acc_p[p][i] = make_float2(0.0f, 0.0f);
          }
        }
      }
      if (done) return;
      plane_lo = P;
      plane_hi = -1;
    }
  }
}

// 2D f32 tiles: the bin rows of a tile are strips already, in x order up to
// the bins' width, as long as a row's windows reach at most 8 rows of cells
// (bins of at most 9 - w cells along y), so no order is built. A warp takes an
// equal range of consecutive records; for 8 points of one bin row,
//   C[(y, re/im), x] += sum_k (c wy)[(y, re/im), k] wx[k, x]
// is one 16 x 8 x 8 product per block of 8 columns that their windows reach,
// in split tf32 as for the 3D strips. A row's blocks reach the tile when the
// range leaves the row.
constexpr int kRowBlocks = 9;      // blocks of 8 columns: 64 starts and the window
constexpr int kRowMaxTile = 64;    // starts of a tile along x, at most
// The width that takes them, where a tile holds a record per two start cells:
// below w 7 the register runs of the per-point spreader are at least as fast
// (1024^2 modes, 2 points per cell, w 6: 294 us against 408; w 7: 527 against
// 492, crowded points 190 against 126; at 1/4 point per cell 185 against 197).
constexpr int kRowWidth = 7;
// Staged floats of a point: wx[8] wy[8] re im - -.
constexpr int kRowStride = 20;
constexpr int kRowFloats = 32 * kRowStride;

template <int W>
__device__ void spread_rows2(const SpreadParams& sp, const PreparedWindow<2>* win2, const float2* sv,
                             const uint32_t* perm, const uint32_t* row_begin, const uint32_t* row_prefix, int rows,
                             const int* origin, uint32_t record_begin, uint32_t record_end, uint32_t* acc, int padded,
                             float* stage, float scale_lo, float scale_hi) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  float* const st = stage + warp * kRowFloats;
  const uint32_t n = record_end - record_begin;
  const uint32_t share = (n + kSpreadWarps - 1) / kSpreadWarps;
  uint32_t at = record_begin + min(n, share * warp);
  const uint32_t to = record_begin + min(n, share * (warp + 1));
  if (at >= to) return;
  const int bin_first = origin[1] >> sp.grid.axis[1].shift;  // the tile's first bin row
  int row = 0;
  {
    int low = 0, high = rows - 1;  // last row starting at or before `at`
    while (low < high) {
      const int mid = (low + high + 1) >> 1;
      if (row_prefix[mid] <= at) low = mid; else high = mid - 1;
    }
    row = low;
  }
  float2 sum[kRowBlocks][2];  // columns 8 j + 2 t, + 1 of row g: real and imaginary parts
#pragma unroll
  for (int j = 0; j < kRowBlocks; ++j) sum[j][0] = sum[j][1] = make_float2(0.0f, 0.0f);
  int col_lo = kRowBlocks, col_hi = -1;
  // Lane = point of the chunk (up to 32 records of one row). The next chunk's
  // windows and point indexes are loaded one chunk ahead.
  struct Rows {
    int row;
    uint32_t at, end;
  };
  auto settle = [&](Rows& r) {  // the row holding record r.at
    while (r.row + 1 < rows && r.at >= row_prefix[r.row + 1]) ++r.row;
    r.end = min(min(r.at + 32u, row_prefix[r.row + 1]), to);
  };
  auto fetch = [&](const Rows& r, int4& win, uint32_t& point) {
    win.x = -1;
    if (r.at < to && r.at + lane < r.end) {
      const uint32_t slot = row_begin[r.row] + (r.at + lane - row_prefix[r.row]);
      win = __ldg(reinterpret_cast<const int4*>(win2 + slot));
      point = __ldg(perm + slot);
    }
  };
  Rows now{row, at, at};
  settle(now);
  int4 win0, win1;
  uint32_t q0 = 0, q1 = 0;
  fetch(now, win0, q0);
  float2 c0 = make_float2(0.0f, 0.0f);
  if (win0.x >= 0) c0 = __ldg(sv + q0);
  for (;;) {
    Rows next{now.row, now.end, now.end};
    if (next.at < to) settle(next);
    fetch(next, win1, q1);
    // Stage the chunk. Points outside the fold's reach or starting in another
    // tile weigh zero.
    const int y_first = max((bin_first + now.row) << sp.grid.axis[1].shift, origin[1]);  // first start of the row
    const int x = win0.x - origin[0], y = win0.y - origin[1];
    const bool inside = win0.x >= 0 && x >= 0 && x < sp.tile[0] && y >= 0 && y < sp.tile[1];
    float wx[W], wy[W];
    horner32_window<W>(__int_as_float(win0.z), sp.grid.horner32, wx);
    horner32_window<W>(__int_as_float(win0.w), sp.grid.horner32, wy);
    __syncwarp();  // the previous chunk's rows are read
    {
      float* const mine = st + lane * kRowStride;
      float row_x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) row_x[j] = j < W ? wx[j] : 0.0f;
      float4* const mine4 = reinterpret_cast<float4*>(mine);
      mine4[0] = make_float4(row_x[0], row_x[1], row_x[2], row_x[3]);
      mine4[1] = make_float4(row_x[4], row_x[5], row_x[6], row_x[7]);
      mine4[2] = mine4[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const int place = inside ? win0.y - y_first : 0;
#pragma unroll
      for (int j = 0; j < W; ++j) mine[8 + place + j] = wy[j];
      const float2 c = inside ? cscale(cscale(c0, scale_lo), scale_hi) : make_float2(0.0f, 0.0f);
      *reinterpret_cast<float2*>(mine + 16) = c;
    }
    __syncwarp();
    const int count = static_cast<int>(now.end - now.at);
    float2 c1 = make_float2(0.0f, 0.0f);
    if (win1.x >= 0) c1 = __ldg(sv + q1);
#pragma unroll 1
    for (int k = 0; k < count; k += 8) {
      // Columns of the eight points' windows.
      const bool member = inside && (lane >> 3) == (k >> 3);
      const int lo = __reduce_min_sync(0xFFFFFFFFu, member ? x : 0x7FFF) >> 3;
      const int hi = (__reduce_max_sync(0xFFFFFFFFu, member ? x : -W) + W - 1) >> 3;
      const int x0 = g - __shfl_sync(0xFFFFFFFFu, x, k + t), x1 = g - __shfl_sync(0xFFFFFFFFu, x, k + 4 + t);
      const float* const p0 = st + (k + t) * kRowStride;
      const float* const p1 = p0 + 4 * kRowStride;
      uint32_t ah[4], al[4];
      {
        const float y0 = p0[8 + g], y1 = p1[8 + g];
        const float2 v0 = *reinterpret_cast<const float2*>(p0 + 16);
        const float2 v1 = *reinterpret_cast<const float2*>(p1 + 16);
        split_tf32(v0.x * y0, ah[0], al[0]);
        split_tf32(v0.y * y0, ah[1], al[1]);
        split_tf32(v1.x * y1, ah[2], al[2]);
        split_tf32(v1.y * y1, ah[3], al[3]);
      }
      col_lo = min(col_lo, lo);
      col_hi = max(col_hi, hi);
      auto block = [&](int j) {  // j: a constant of the caller
        const unsigned i0 = static_cast<unsigned>(x0 + 8 * j), i1 = static_cast<unsigned>(x1 + 8 * j);
        uint32_t bh0, bl0, bh1, bl1;
        split_tf32(i0 < 8u ? p0[i0] : 0.0f, bh0, bl0);
        split_tf32(i1 < 8u ? p1[i1] : 0.0f, bh1, bl1);
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        mma_tf32(d, ah, bl0, bl1);
        mma_tf32(d, al, bh0, bh1);
        mma_tf32(d, ah, bh0, bh1);
        sum[j][0] = __fadd2_rn(sum[j][0], make_float2(d[0], d[1]));
        sum[j][1] = __fadd2_rn(sum[j][1], make_float2(d[2], d[3]));
      };
      // Blocks lo .. hi: a jump to the first, and on while there are more.
      switch (lo) {
#define B200NUFFT_ROW_BLOCK(J) \
  case J:                      \
    block(J);                  \
    if (hi <= J) break;        \
    [[fallthrough]];
        B200NUFFT_ROW_BLOCK(0)
        B200NUFFT_ROW_BLOCK(1)
        B200NUFFT_ROW_BLOCK(2)
        B200NUFFT_ROW_BLOCK(3)
        B200NUFFT_ROW_BLOCK(4)
        B200NUFFT_ROW_BLOCK(5)
        B200NUFFT_ROW_BLOCK(6)
        B200NUFFT_ROW_BLOCK(7)
#undef B200NUFFT_ROW_BLOCK
        case 8: block(8); break;
        default: break;  // no point of these in the tile
      }
    }
    const bool done = next.at >= to;
    if (done || next.row != now.row) {
      const int cy = y_first - origin[1] + g;
      constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23
      const float2 magic = make_float2(kMagic, kMagic), minus = make_float2(-kMagic, -kMagic);
      const float2 down = make_float2(1.0f / 65536.0f, 1.0f / 65536.0f), up = make_float2(-65536.0f, -65536.0f);
#pragma unroll
      for (int j = 0; j < kRowBlocks; ++j) {
        if (j >= col_lo && j <= col_hi) {
          const int cx = 8 * j + 2 * t, cell = cy * sp.pad[0] + cx;
          const bool in0 = cy < sp.pad[1] && cx < sp.pad[0], in1 = cy < sp.pad[1] && cx + 1 < sp.pad[0];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 h = __ffma2_rn(sum[j][i], down, magic);
            const float2 l = __fadd2_rn(__ffma2_rn(__fadd2_rn(h, minus), up, sum[j][i]), magic);
            if (in0) add_split(acc, padded, i, cell, h.x, l.x);
            if (in1) add_split(acc, padded, i, cell + 1, h.y, l.y);
            sum[j][i] = make_float2(0.0f, 0.0f);
          }
        }
      }
      col_lo = kRowBlocks;
      col_hi = -1;
    }
    if (done) return;
    now = next;
    win0 = win1;
    c0 = c1;
  }
}

// 2D f64 tiles: strips of 16 x S cells (x, y) reach YT x NT blocks of 8 x 8
// cells, and 4 points add
//   C[y, x] += sum_k (c wy)[y, k] wx[k, x]
// to each block in two m8n8k4 products (real and imaginary part) in f64, whose
// rounding is that of fused multiply-adds. Blocks of columns that no window of
// the chunk reaches are skipped.
constexpr int kStrip64X = 16;
template <int W>
struct Strip64 {
  static constexpr int YT = W <= 13 ? 2 : 3;       // blocks of rows
  static constexpr int S = 8 * YT - W + 1;         // support starts along y
  static constexpr int NT = (kStrip64X + W - 1 + 7) / 8;
  // Staged doubles of a point: wx[8 NT] wy[8 YT] re im; the pitch is 4 mod 16
  // doubles, so the four points of a product read different banks.
  static constexpr int kY = 8 * NT, kValue = kY + 8 * YT;
  static constexpr int kStride = (kValue + 2 + 11) / 16 * 16 + 4;
  static constexpr int kDoubles = 8 * kStride;
  // Horner rows (EsHornerTable::fit), each as its even taps, then its odd
  // ones, kTaps (even) of each.
  static constexpr int kRows = W + 3 < kMaxHornerCoefficients ? W + 3 : kMaxHornerCoefficients;
  static constexpr int kTaps = (W + 3) / 4 * 2;
};
// Fills the window's Horner table: per row the even taps, then the odd ones;
// leading rows that the fit dropped are zero. The caller synchronizes.
template <int W>
__device__ __forceinline__ void strip64_table(const GridParams& grid, double* table) {
  using L = Strip64<W>;
  for (int i = threadIdx.x; i < L::kRows * 2 * L::kTaps; i += kSpreadThreads) {
    const int tap = 2 * (i % L::kTaps) + (i / L::kTaps) % 2;
    const int r = i / (2 * L::kTaps) - (L::kRows - grid.horner_rows);
    table[i] = tap < W && r >= 0 ? grid.horner[r * W + tap] : 0.0;
  }
}
template <int W>
__host__ __device__ constexpr int strip64_count(int t0, int t1) {
  return ((t0 + kStrip64X - 1) / kStrip64X) * ((t1 + Strip64<W>::S - 1) / Strip64<W>::S);
}

template <int W>
__device__ void spread_strips2_f64(const SpreadParams& sp, const double2* points, const double2* sv,
                                   const uint32_t* perm, const uint32_t* row_begin, const uint32_t* row_prefix,
                                   int rows, const int* origin, uint32_t record_begin, uint32_t record_end,
                                   unsigned long long* acc, int padded, const StripShared& sh,
                                   const double* table, double scale_lo, double scale_hi) {
  using L = Strip64<W>;
  constexpr int S = L::S, YT = L::YT, NT = L::NT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = sp.tile[0], t1 = sp.tile[1];
  const int nx = (t0 + kStrip64X - 1) / kStrip64X, ny = (t1 + S - 1) / S;
  const int strips = nx * ny;
  for (int s = tid; s < strips; s += kSpreadThreads) {
    sh.cell[s] = static_cast<uint32_t>((s % nx) * kStrip64X | (s / nx) * S << 8);
  }
  auto start_of = [&](double x, int a, double& offset) {
    int32_t start;
    support_of64(x, sp.grid.axis64[a], sp.grid.half_width64, start, offset);
    return wrap_start(start, sp.grid.axis[a].length) - origin[a];
  };
  // The counters lie in the tile region, which is cleared afterwards.
  strip_order(
      row_begin, row_prefix, rows, record_begin, record_end, strips, kStrip64X, reinterpret_cast<uint32_t*>(acc),
      sh, [&](uint32_t slot) { return __ldg(points + slot); },
      [&](const double2& p) {
        if (!in_fold_reach64(p.x) || !in_fold_reach64(p.y)) return -1;
        double offset;
        const int x = start_of(p.x, 0, offset), y = start_of(p.y, 1, offset);
        if (x < 0 || x >= t0 || y < 0 || y >= t1) return -1;  // another tile owns it
        return (x / kStrip64X + nx * (y / S)) * kStrip64X + x % kStrip64X;
      });
  __syncthreads();
  {
    uint4* acc16 = reinterpret_cast<uint4*>(acc);
    for (int c = tid; c < padded; c += kSpreadThreads) acc16[c] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  const int spread = static_cast<int>(sh.start[strips]);
  const int share = (spread + kSpreadWarps - 1) / kSpreadWarps;
  const int from = min(spread, share * warp), to = min(spread, share * (warp + 1));
  if (from >= to) return;
  StripChunk k0 = first_chunk(from, sh.start, strips);
  if (k0.at >= to) return;
  const int g = lane >> 2, t = lane & 3;  // fragment row / column group
  double* const st = reinterpret_cast<double*>(sh.stage) + warp * L::kDoubles;
  double2 sum[YT][NT][2];  // block (rows y, columns x = 2t, 2t + 1), real and imaginary
#pragma unroll
  for (int i = 0; i < YT; ++i) {
#pragma unroll
    for (int j = 0; j < NT; ++j) sum[i][j][0] = sum[i][j][1] = make_double2(0.0, 0.0);
  }
  // Lane (g, t) stages half the taps of one axis of point g (axis t >> 1, the
  // even or odd taps), lane (g, 0) its strength too. Coordinates and point
  // indexes are loaded two chunks ahead, strengths one chunk ahead.
  const int axis = t >> 1;
  auto fetch = [&](const StripChunk& c, double& x, uint32_t& point) {
    const int at = c.at + g;
    if (c.at < to && at < c.end) {
      const uint32_t slot = sh.sorted[at];
      x = __ldg(reinterpret_cast<const double*>(points) + 2 * static_cast<int64_t>(slot) + axis);
      if (t == 0) point = __ldg(perm + slot);
    }
  };
  auto strength_of = [&](const StripChunk& c, uint32_t point, double2& v) {
    if (t == 0 && c.at < to && c.at + g < c.end) v = __ldg(sv + point);
  };
  double x0 = 0.0, x1 = 0.0;
  uint32_t q0 = 0, q1 = 0;
  double2 c0 = make_double2(0.0, 0.0);
  StripChunk k1 = k0;
  next_chunk(k1, sh.start, strips);
  fetch(k0, x0, q0);
  fetch(k1, x1, q1);
  strength_of(k0, q0, c0);
  int col_lo = NT, col_hi = -1;
  for (;;) {
    const StripChunk now = k0;
    const double x = x0;
    const double2 c = c0;
    const int count = min(now.end - now.at, 8);
    strength_of(k1, q1, c0);
    k0 = k1;
    x0 = x1;
    next_chunk(k1, sh.start, strips);
    fetch(k1, x1, q1);
    const uint32_t cell = sh.cell[now.strip];
    double offset;
    const int place = start_of(x, axis, offset) - static_cast<int>((cell >> (8 * axis)) & 255u);
    // Stage the chunk: rows of zeros with the weights at their place.
    __syncwarp();  // the previous chunk's rows are read
    for (int i = lane; i < L::kDoubles / 2; i += 32) reinterpret_cast<double2*>(st)[i] = make_double2(0.0, 0.0);
    __syncwarp();
    if (g < count) {
      double* const row = st + g * L::kStride + (axis == 0 ? 0 : L::kY) + place;
      const double local = 2.0 * offset + static_cast<double>(W - 1);
      const bool inside = fabs(local) <= 1.0;
      constexpr int kTaps = L::kTaps;
      double w[kTaps];
#pragma unroll
      for (int j = 0; j < kTaps; ++j) w[j] = 0.0;
      const double2* coefficients = reinterpret_cast<const double2*>(table) + (t & 1) * (kTaps / 2);
#pragma unroll
      for (int r = 0; r < L::kRows; ++r) {
#pragma unroll
        for (int j = 0; j < kTaps; j += 2) {
          const double2 pair = coefficients[r * kTaps + j / 2];
          w[j] = fma(w[j], local, pair.x);
          w[j + 1] = fma(w[j + 1], local, pair.y);
        }
      }
#pragma unroll
      for (int j = 0; j < kTaps; ++j) {
        if (2 * j + (t & 1) < W) row[2 * j + (t & 1)] = inside ? w[j] : 0.0;
      }
      if (t == 0) {
        *reinterpret_cast<double2*>(st + g * L::kStride + L::kValue) =
            make_double2((c.x * scale_lo) * scale_hi, (c.y * scale_lo) * scale_hi);
      }
    }
    const int lo = __shfl_sync(0xFFFFFFFFu, place, 0) >> 3;
    const int hi = (__shfl_sync(0xFFFFFFFFu, place, 4 * (count - 1)) + W - 1) >> 3;
    __syncwarp();
    col_lo = min(col_lo, lo);
    col_hi = max(col_hi, hi);
#pragma unroll
    for (int k = 0; k < 8; k += 4) {
      if (k >= count) break;
      const double* const p = st + (k + t) * L::kStride;
      const double2 v = *reinterpret_cast<const double2*>(p + L::kValue);
      double re[YT], im[YT];
#pragma unroll
      for (int i = 0; i < YT; ++i) {
        const double wy = p[L::kY + 8 * i + g];
        re[i] = v.x * wy;
        im[i] = v.y * wy;
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        if (j >= lo && j <= hi) {
          const double wx = p[8 * j + g];
#pragma unroll
          for (int i = 0; i < YT; ++i) {
            mma_f64(sum[i][j][0], re[i], wx);
            mma_f64(sum[i][j][1], im[i], wx);
          }
        }
      }
    }
    const bool done = k0.at >= to;
    if (done || k0.strip != now.strip) {
      // The strip's blocks to the tile.
      const int xs = static_cast<int>(cell & 255u), ys = static_cast<int>(cell >> 8);
      auto add = [&](int part, int at, double v) {
        atomicAdd(&acc[part * padded + at], static_cast<unsigned long long>(__double2ll_rn(v)));
      };
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        if (j >= col_lo && j <= col_hi) {
          const int cx = xs + 8 * j + 2 * t;
#pragma unroll
          for (int i = 0; i < YT; ++i) {
            const int cy = ys + 8 * i + g;
            const int at = cy * sp.pad[0] + cx;
            if (cy < sp.pad[1] && cx < sp.pad[0]) {
              add(0, at, sum[i][j][0].x);
              add(1, at, sum[i][j][1].x);
            }
            if (cy < sp.pad[1] && cx + 1 < sp.pad[0]) {
              add(0, at + 1, sum[i][j][0].y);
              add(1, at + 1, sum[i][j][1].y);
            }
            sum[i][j][0] = sum[i][j][1] = make_double2(0.0, 0.0);
          }
        }
      }
      if (done) return;
      col_lo = NT;
      col_hi = -1;
    }
  }
}

}  // namespace b200nufft
