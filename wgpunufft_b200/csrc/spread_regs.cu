// Type-1 spreading of 3D f64 tiles in registers.
//
// A CTA takes one part of one tile; the padded tile is 24 planes (x) of 8 YB x
// 8 ZB cells (y, z), and each of its 12 warps keeps two neighbouring planes as
// f64 accumulators of m8n8k4 products. For 4 points whose windows reach the
// warp's planes, each plane p receives
//   C_p[y, z] += sum_k (c wy)[y, k] (wx[p] wz)[k, z]
// (real and imaginary part). The points' weights are evaluated once per CTA, 32
// points at a time, into shared memory, the next 32 while these are
// multiplied. There is no shared-memory tile, no atomic and no fixed point: a
// cell's sum is the fused multiply-adds of the records in their order, so it
// repeats bit for bit, and a part's tile is written out from the registers
// (two neighbouring cells, a 32-byte sector, per lane).
//
// Bound: the f64 matrix rate, (w + 1) planes x 2 YB ZB products of 4 points, 4
// cycles each per SM, where tiles hold hundreds of points; below that the
// padded tiles' traffic and each CTA's start. Against a warp per record adding
// to a 64-bit fixed-point tile in shared memory (9 cycles per add of a warp),
// 128^3 cells, uniform: w 10 at 1/16 point per cell 665 -> 300 us, at 1 point
// 8.13 -> 2.34 ms; w 13 at 1 point 18.6 -> 2.82 ms; w 7 at 1/512 point 70 -> 89
// us.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.h"
#include "mma.cuh"
#include "spread.h"
#include "strips.cuh"

namespace b200nufft {

namespace {

constexpr int kThreads = 384;
constexpr int kBatch = 32;  // points staged at a time
constexpr int kPlanes = kReg64Planes;
static_assert(2 * kThreads / 32 == kPlanes, "two planes per warp");
static_assert(kThreads / 12 == kBatch, "12 threads evaluate a point's windows");

template <int W>
struct Regs {
  static constexpr int YB = reg64_blocks_y(W), ZB = reg64_blocks_z(W);
  // Staged doubles of a point: wx[24] wy[8 YB] wz[8 ZB] re im - -.
  static constexpr int kY = kPlanes, kZ = kY + 8 * YB, kValue = kZ + 8 * ZB, kStride = kValue + 4;
  static constexpr int kRows = W + 3;  // Horner rows (EsHornerTable::fit), w <= 13
};

template <int W>
__global__ void __launch_bounds__(kThreads, 1) spread_regs3_kernel(
    SpreadParams sp, const double* __restrict__ points, const double2* __restrict__ strengths, int64_t point_count,
    int batch, const uint32_t* __restrict__ perm, const uint32_t* __restrict__ offsets,
    const uint32_t* __restrict__ part_start, double2* __restrict__ scratch) {
  using R = Regs<W>;
  constexpr int YB = R::YB, ZB = R::ZB;
  __shared__ __align__(16) double stage[2][(kBatch + 1) * R::kStride];  // the last row: zeros
  __shared__ int place[2][3][kBatch];                                   // starts in the tile; negative: skipped
  __shared__ double table[R::kRows * W];
  __shared__ uint32_t row_begin[kMaxTileRows], row_prefix[kMaxTileRows + 1], warp_totals[kMaxTileRows / 32];
  __shared__ int list[kThreads / 32][kBatch + 4];
  __shared__ int64_t s_tile;
  const uint32_t part = blockIdx.x;
  if (part >= part_start[sp.tile_count]) return;
  const uint32_t part_cap = static_cast<uint32_t>(sp.part_cap_device != nullptr ? *sp.part_cap_device : sp.part_cap);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp == 0) {
    const int64_t found = part_tile(part_start, sp.tile_count, part);
    if (lane == 0) s_tile = found;
  }
  {
    const int missing = (R::kRows - sp.grid.horner_rows) * W;  // leading rows that vanish are dropped
    for (int i = tid; i < R::kRows * W; i += kThreads) table[i] = i >= missing ? sp.grid.horner[i - missing] : 0.0;
    for (int i = tid; i < R::kStride; i += kThreads) {
      stage[0][kBatch * R::kStride + i] = 0.0;
      stage[1][kBatch * R::kStride + i] = 0.0;
    }
  }
  __syncthreads();
  const int64_t tile = s_tile;
  int origin[3], bin_lo[3], rows_along[3], bin_hi0 = 0;
  {
    uint32_t rest = static_cast<uint32_t>(tile);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t tiles = static_cast<uint32_t>(sp.ntiles[a]), next = rest / tiles;
      origin[a] = static_cast<int>(rest - next * tiles) * sp.tile[a];
      rest = next;
      const int64_t last = min(static_cast<int64_t>(origin[a]) + sp.tile[a], sp.grid.fine[a]) - 1;
      bin_lo[a] = origin[a] >> sp.grid.axis[a].shift;
      const int hi = static_cast<int>(last >> sp.grid.axis[a].shift);
      rows_along[a] = hi - bin_lo[a] + 1;
      if (a == 0) bin_hi0 = hi;
    }
  }
  const int rows = rows_along[1] * rows_along[2];
  // Row slot ranges and their exclusive prefix.
  if (tid < kMaxTileRows) {
    uint32_t n = 0;
    if (tid < rows) {
      const int y = bin_lo[1] + tid % rows_along[1], z = bin_lo[2] + tid / rows_along[1];
      const uint64_t row = static_cast<uint64_t>(sp.grid.axis[0].bins) *
                           (y + static_cast<uint64_t>(sp.grid.axis[1].bins) * z);
      const uint32_t begin = offsets[row + bin_lo[0]];
      n = offsets[row + bin_hi0 + 1] - begin;
      row_begin[tid] = begin;
    }
    uint32_t x = n;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, offset);
      if (lane >= offset) x += y;
    }
    if (lane == 31) warp_totals[warp] = x;
    row_prefix[tid] = x - n;
  }
  __syncthreads();
  if (tid < kMaxTileRows) {
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += warp_totals[w];
    row_prefix[tid] += before;
    if (tid == kMaxTileRows - 1) row_prefix[kMaxTileRows] = before + warp_totals[warp];
  }
  __syncthreads();
  const uint32_t record_begin = (part - part_start[tile]) * part_cap;
  const uint32_t record_end = min(row_prefix[kMaxTileRows], record_begin + part_cap);
  const int batches = record_end > record_begin ? static_cast<int>((record_end - record_begin + kBatch - 1) / kBatch) : 0;
  const double2* const sv = strengths + static_cast<int64_t>(blockIdx.y) * point_count;

  // Twelve threads per staged point: axis `axis`, taps and cells of residue q
  // modulo 4. Coordinates and strengths are loaded a batch ahead of their
  // staging, point indexes two.
  const int p = tid / 12, role = tid % 12, axis = role >> 2, q = role & 3;
  auto slot_of = [&](int b) {  // slot of the thread's point in batch b; false past the part
    const uint32_t r = record_begin + static_cast<uint32_t>(b) * kBatch + p;
    if (r >= record_end) return int64_t{-1};
    int row = 0;
#pragma unroll
    for (int step = kMaxTileRows / 2; step > 0; step >>= 1) {
      if (row + step < rows && row_prefix[row + step] <= r) row += step;
    }
    return static_cast<int64_t>(row_begin[row] + (r - row_prefix[row]));
  };
  double x_next = 0.0;
  double2 c_next = make_double2(0.0, 0.0);
  uint32_t q_next = 0;
  bool has_next = false, has_q = false;
  auto load_point = [&](int b) {
    has_q = false;
    if (role != 0) return;
    const int64_t slot = slot_of(b);
    if (slot >= 0) {
      q_next = __ldg(perm + slot);
      has_q = true;
    }
  };
  auto load = [&](int b) {
    const int64_t slot = slot_of(b);
    has_next = slot >= 0;
    if (has_next) x_next = __ldg(points + slot * 3 + axis);
    if (role == 0) c_next = has_q ? __ldg(sv + q_next) : make_double2(0.0, 0.0);
  };
  auto fill = [&](int buffer) {
    double* const row = stage[buffer] + p * R::kStride;
    double* const mine = row + (axis == 0 ? 0 : (axis == 1 ? R::kY : R::kZ));
    const int cells = axis == 0 ? kPlanes : (axis == 1 ? 8 * YB : 8 * ZB);
    for (int j = q; j < cells; j += 4) mine[j] = 0.0;
    int start = -1;
    if (has_next && in_fold_reach64(x_next)) {
      int32_t first;
      double offset;
      support_of64(x_next, sp.grid.axis64[axis], sp.grid.half_width64, first, offset);
      const int local_start = wrap_start(first, sp.grid.axis[axis].length) - origin[axis];
      if (local_start >= 0 && local_start < sp.tile[axis]) {  // else another tile owns it
        start = local_start;
        constexpr int kTaps = (W + 3) / 4;
        const double local = 2.0 * offset + static_cast<double>(W - 1);
        const bool inside = fabs(local) <= 1.0;
        const int tap = (q - start) & 3;
        double w[kTaps];
#pragma unroll
        for (int j = 0; j < kTaps; ++j) w[j] = 0.0;
#pragma unroll
        for (int r = 0; r < R::kRows; ++r) {
#pragma unroll
          for (int j = 0; j < kTaps; ++j) w[j] = fma(w[j], local, table[r * W + min(tap + 4 * j, W - 1)]);
        }
#pragma unroll
        for (int j = 0; j < kTaps; ++j) {
          if (tap + 4 * j < W) mine[start + tap + 4 * j] = inside ? w[j] : 0.0;
        }
      }
    }
    if (q == 0) place[buffer][axis][p] = start;
    if (role == 0) *reinterpret_cast<double2*>(row + R::kValue) = c_next;
  };
  const int g = lane >> 2, t = lane & 3;
  const int plane = 2 * warp;
  double2 sum[2][YB][ZB][2];  // [plane][rows y][columns z = 2 t, 2 t + 1][real, imaginary]
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int i = 0; i < YB; ++i) {
#pragma unroll
      for (int j = 0; j < ZB; ++j) sum[k][i][j][0] = sum[k][i][j][1] = make_double2(0.0, 0.0);
    }
  }
  if (batches > 0) {
    load_point(0);
    load(0);
    load_point(1);
    fill(0);
    load(1);
    load_point(2);
  }
  for (int b = 0; b < batches; ++b) {
    __syncthreads();  // batch b is staged, and batch b - 1 is read
    if (b + 1 < batches) {
      fill((b + 1) & 1);
      load(b + 2);
      load_point(b + 3);
    }
    const double* const rows_of = stage[b & 1];
    // The points that reach the warp's planes, in their order.
    const int px = place[b & 1][0][lane];
    const bool hit = px >= 0 && place[b & 1][1][lane] >= 0 && place[b & 1][2][lane] >= 0 && px <= plane + 1 &&
                     px + W - 1 >= plane;
    const unsigned hits = __ballot_sync(0xFFFFFFFFu, hit);
    const int count = __popc(hits);
    __syncwarp();  // the previous list is read
    if (hit) list[warp][__popc(hits & ((1u << lane) - 1u))] = lane;
    if (lane < 4) list[warp][count + lane] = kBatch;  // the row of zeros
    __syncwarp();
    for (int s = 0; s < count; s += 4) {
      const double* const row = rows_of + list[warp][s + t] * R::kStride;
      const double2 wx = *reinterpret_cast<const double2*>(row + plane);
      const double2 c = *reinterpret_cast<const double2*>(row + R::kValue);
      double re[YB], im[YB];
#pragma unroll
      for (int i = 0; i < YB; ++i) {
        const double wy = row[R::kY + 8 * i + g];
        re[i] = c.x * wy;
        im[i] = c.y * wy;
      }
#pragma unroll
      for (int j = 0; j < ZB; ++j) {
        const double wz = row[R::kZ + 8 * j + g];
        const double w0 = wx.x * wz, w1 = wx.y * wz;
#pragma unroll
        for (int i = 0; i < YB; ++i) {
          mma_f64(sum[0][i][j][0], re[i], w0);
          mma_f64(sum[0][i][j][1], im[i], w0);
          mma_f64(sum[1][i][j][0], re[i], w1);
          mma_f64(sum[1][i][j][1], im[i], w1);
        }
      }
    }
  }
  double2* const out = scratch + (static_cast<int64_t>(part) * batch + blockIdx.y) * sp.padded_cells + plane;
#pragma unroll
  for (int i = 0; i < YB; ++i) {
#pragma unroll
    for (int j = 0; j < ZB; ++j) {
      const int y = 8 * i + g, z = 8 * j + 2 * t;
      double2* const at = out + sp.pad[0] * (y + sp.pad[1] * z);
      double2* const up = at + sp.pad[0] * sp.pad[1];
      at[0] = make_double2(sum[0][i][j][0].x, sum[0][i][j][1].x);
      at[1] = make_double2(sum[1][i][j][0].x, sum[1][i][j][1].x);
      up[0] = make_double2(sum[0][i][j][0].y, sum[0][i][j][1].y);
      up[1] = make_double2(sum[1][i][j][0].y, sum[1][i][j][1].y);
    }
  }
}

template <int W>
void launch(const SpreadParams& sp, const SpreadLaunch64& l, cudaStream_t stream) {
  const dim3 grid(static_cast<unsigned>(l.part_upper_bound), static_cast<unsigned>(l.batch));
  spread_regs3_kernel<W><<<grid, kThreads, 0, stream>>>(sp, l.points, l.strengths, l.point_count, l.batch, l.perm,
                                                        l.offsets, l.part_start, l.scratch);
  note_launch();
}

}  // namespace

void spread_regs64(const SpreadParams& sp, const SpreadLaunch64& l, cudaStream_t stream) {
  switch (sp.grid.width) {
    case 5: launch<5>(sp, l, stream); break;
    case 6: launch<6>(sp, l, stream); break;
    case 7: launch<7>(sp, l, stream); break;
    case 8: launch<8>(sp, l, stream); break;
    case 9: launch<9>(sp, l, stream); break;
    case 10: launch<10>(sp, l, stream); break;
    case 11: launch<11>(sp, l, stream); break;
    case 12: launch<12>(sp, l, stream); break;
    default: launch<13>(sp, l, stream); break;
  }
}

}  // namespace b200nufft
