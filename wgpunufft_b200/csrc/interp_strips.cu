// Type-2 interpolation by small matrix products (mma.sync): 2D and 3D plans
// whose points are ordered by strips of support starts.
//
// set_points orders the points by (z strip, y strip, x start), the strips a
// few cells wide (interp_strip_shifts). A warp takes 32 consecutive points and
// serves them in groups of one strip whose starts lie within kSpan cells of x.
// For a group, every plane z and every block of 4 columns,
//   T[point, x] = sum_y wy[point, y] G[z, y, x]
// is a product with the strip's rows as the contracted index (f32: 8 rows,
// m16n8k8 on tf32 high and low parts, smallest products first, from zero; f64:
// m8n8k4), whose right operand, the grid values, is loaded once for 32 points
// straight into fragments; each point then adds wx wz T to its sum. The
// gather of w^d cells per point becomes a few loads per point.
//
// A point's sum depends on its own window alone: rows and columns outside
// it weigh zero, blocks and rows are fixed by the grid, so the bits do not
// depend on the group, the batch or the other points.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.h"
#include "interp.h"
#include "mma.cuh"

namespace b200nufft {

namespace {

constexpr int kSpan = 16;  // x starts of a group, at most
// Vectors of a CTA: each stages its points' weights once for them, and the
// outputs that the running CTAs scatter to stay in L2 (4 x 2e6 points: 64 MB).
constexpr int kBlockVectors = 4;

// Strip sides (log2) along y and z: the rows a strip's windows reach fill the
// contracted index (8 rows in f32, multiples of 4 in f64); z strips of 4.
template <int W, bool F64>
struct Strip {
  static constexpr int kShiftY = F64 ? 2 : 1;
  static constexpr int kShiftZ = 2;
  static constexpr int kRows = F64 ? ((1 << kShiftY) + W - 1 + 3) / 4 * 4 : 8;
  static constexpr int kPitchY = kRows % 8 == 0 ? kRows + 4 : kRows;  // conflict-free fragment reads
  static constexpr int kPitchX = W | 1;
  // z weights at their place among the planes of the strip, zeros around them.
  static constexpr int kPlanes = (1 << kShiftZ) + W - 1;
  static constexpr int kPitchZ = kPlanes | 1;
};

template <int D, int W, typename Real>
struct WarpStage {
  using S = Strip<W, sizeof(Real) == 8>;
  Real wy[32 * S::kPitchY];
  Real wx[32 * S::kPitchX];
  Real wz[D == 3 ? 32 * S::kPitchZ : 1];
};

struct F32Strips {
  using Real = float;
  using Complex = float2;
  static constexpr int kWarps = 4;
};
struct F64Strips {
  using Real = double;
  using Complex = double2;
  static constexpr int kWarps = 2;
};

// Groups of a warp's 32 points, at most, that the 2D f64 products serve; beyond
// that each lane gathers its own w^2 cells, adding them in the products' order
// (the same bits). A group's products cost a half (w 5) to a fifth (w 13) of 32
// gathers. 1024^2 modes, uniform, us per transform with products alone and so: w 7,
// 1/16 point per cell 195 / 139, 1/4 244 / 224; w 13, 1/16 249 / 221.
template <int W>
constexpr int kMostGroups = W <= 6 ? 1 : (W <= 8 ? 2 : (W - 1) / 2);

// One point's w^2 cells, added in the products' order: down the rows, then
// along the columns of one residue modulo 4, as the four lanes of a product do.
// A call, so that the products keep their registers.
template <int W>
__device__ __noinline__ void gather_columns(const double* wx, const double* wy, int x0, int y0, int n0, int n1,
                                            const double2* grid, int64_t grid_stride, int vectors, double2* output,
                                            int64_t output_stride) {
  for (int b = 0; b < vectors; ++b, grid += grid_stride, output += output_stride) {
    double2 columns[W];
#pragma unroll
    for (int i = 0; i < W; ++i) columns[i] = make_double2(0.0, 0.0);
#pragma unroll 2
    for (int j = 0; j < W; ++j) {
      const int y = y0 + j >= n1 ? y0 + j - n1 : y0 + j;
      const double2* const row = grid + static_cast<int64_t>(y) * n0;
      const double weight = wy[j];
#pragma unroll
      for (int i = 0; i < W; ++i) {
        const int x = x0 + i >= n0 ? x0 + i - n0 : x0 + i;
        columns[i] = cfma(__ldg(row + x), weight, columns[i]);
      }
    }
    double2 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const int residue = (x0 + i) & 3;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (residue == t) v[t] = cfma(columns[i], wx[i], v[t]);
      }
    }
    *output = make_double2((v[0].x + v[2].x) + (v[1].x + v[3].x), (v[0].y + v[2].y) + (v[1].y + v[3].y));
  }
}

// CTAs of an SM that the registers of a kernel with gathers are held to: what the
// products alone take (0: free).
template <int W, bool Scattered>
constexpr int kMinBlocks = Scattered ? (W <= 9 ? 10 : 8) : 0;

// Scattered: with the gathers (2D f64).
template <int D, int W, int V, typename T, bool Scattered = false>
__global__ void __launch_bounds__(T::kWarps * 32, (kMinBlocks<W, Scattered>)) interp_strips_kernel(
    GridParams grid, const typename T::Real* __restrict__ points, const void* __restrict__ windows, int64_t count,
    const uint32_t* __restrict__ perm, const typename T::Complex* __restrict__ fine, int batch,
    typename T::Complex* __restrict__ output) {
  using Real = typename T::Real;
  using Complex = typename T::Complex;
  constexpr bool F64 = sizeof(Real) == 8;
  using S = Strip<W, F64>;
  constexpr int K = F64 ? S::kRows / 4 : 1;  // products along the rows
  __shared__ __align__(16) WarpStage<D, W, Real> stages[T::kWarps];
  // The f64 Horner table, bottom-aligned (EsHornerTable::fit drops leading rows that vanish).
  constexpr int kHorner = W + 3 < kMaxHornerCoefficients ? W + 3 : kMaxHornerCoefficients;
  __shared__ double table[F64 ? kHorner * W : 1];
  if constexpr (F64) {
    const int missing = (kHorner - grid.horner_rows) * W;
    for (int i = threadIdx.x; i < kHorner * W; i += T::kWarps * 32) {
      table[i] = i >= missing ? grid.horner[i - missing] : 0.0;
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t first = (static_cast<int64_t>(blockIdx.x) * T::kWarps + warp) * 32;
  if (first >= count) return;
  WarpStage<D, W, Real>& st = stages[warp];
  const int n0 = grid.axis[0].length, n1 = grid.axis[1].length, n2 = D == 3 ? grid.axis[2].length : 1;
  const int64_t plane_cells = D == 3 ? static_cast<int64_t>(n0) * n1 : 0;

  // Lane = point: its starts, and its windows staged.
  const int64_t slot = first + lane;
  const bool exists = slot < count;
  int start[3] = {0, 0, 0};
  bool reach = false;
  uint32_t point = 0;
  {
    Real w[W];
    auto place = [&](int a) {
      if (a == 1) {
        Real* row = st.wy + lane * S::kPitchY;
#pragma unroll
        for (int j = 0; j < S::kRows; ++j) row[j] = Real(0);
        row += start[1] & ((1 << S::kShiftY) - 1);
#pragma unroll
        for (int j = 0; j < W; ++j) row[j] = w[j];
      } else if (a == 0) {
        Real* row = st.wx + lane * S::kPitchX;
#pragma unroll
        for (int j = 0; j < W; ++j) row[j] = w[j];
      } else {
        Real* row = st.wz + lane * S::kPitchZ;
#pragma unroll
        for (int j = 0; j < S::kPlanes; ++j) row[j] = Real(0);
        row += start[2] & ((1 << S::kShiftZ) - 1);
#pragma unroll
        for (int j = 0; j < W; ++j) row[j] = w[j];
      }
    };
    if (exists) point = __ldg(perm + slot);
    if constexpr (!F64) {
      PreparedWindow<D> win{};
      win.start[0] = -1;
      if (exists) win = static_cast<const PreparedWindow<D>*>(windows)[slot];
      reach = win.start[0] >= 0;
#pragma unroll
      for (int a = 0; a < D; ++a) {
        start[a] = reach ? win.start[a] : 0;
        horner32_window<W>(win.offset[a], grid.horner32, w);
        place(a);
      }
    } else {
      double p[D];
#pragma unroll
      for (int a = 0; a < D; ++a) p[a] = exists ? points[slot * D + a] : 0.0;
      reach = exists;
#pragma unroll
      for (int a = 0; a < D; ++a) reach = reach && in_fold_reach64(p[a]);
#pragma unroll
      for (int a = 0; a < D; ++a) {
        int32_t s = 0;
        double offset = 0.0;
        if (reach) support_of64(p[a], grid.axis64[a], grid.half_width64, s, offset);
        start[a] = wrap_start(s, grid.axis[a].length);
        const double local = 2.0 * offset + static_cast<double>(W - 1);
        const bool inside = fabs(local) <= 1.0;
#pragma unroll
        for (int j = 0; j < W; ++j) w[j] = 0.0;
#pragma unroll 4
        for (int r = 0; r < kHorner; ++r) {
#pragma unroll
          for (int j = 0; j < W; ++j) w[j] = fma(w[j], local, table[r * W + j]);
        }
#pragma unroll
        for (int j = 0; j < W; ++j) w[j] = inside ? w[j] : 0.0;
        place(a);
      }
    }
  }
  const int first_vector = blockIdx.y * kBlockVectors, last_vector = min(first_vector + kBlockVectors, batch);
  if (exists && !reach) {
    Complex zero;
    zero.x = zero.y = Real(0);
    for (int b = first_vector; b < last_vector; ++b) output[static_cast<int64_t>(b) * count + point] = zero;
  }
  __syncwarp();

  const int strip_y = start[1] >> S::kShiftY, strip_z = D == 3 ? start[2] >> S::kShiftZ : 0;
  unsigned todo = __ballot_sync(0xFFFFFFFFu, reach);
  // The lanes of the next group: one strip, x starts within kSpan cells.
  struct Group {
    int x, y, z;
    bool mine;
    unsigned members;
  };
  auto next_group = [&](unsigned left) {
    const int leader = __ffs(left) - 1;
    Group q;
    q.x = __shfl_sync(0xFFFFFFFFu, start[0], leader);
    q.y = __shfl_sync(0xFFFFFFFFu, strip_y, leader);
    q.z = D == 3 ? __shfl_sync(0xFFFFFFFFu, strip_z, leader) : 0;
    q.mine = ((left >> lane) & 1u) && strip_y == q.y && strip_z == q.z && start[0] >= q.x && start[0] < q.x + kSpan;
    q.members = __ballot_sync(0xFFFFFFFFu, q.mine);
    return q;
  };
  if constexpr (Scattered) {
    // Points too far apart for products: every lane gathers its own.
    int groups = 0;
    for (unsigned left = todo; left != 0u && groups <= kMostGroups<W>; ++groups) left &= ~next_group(left).members;
    if (groups > kMostGroups<W>) {
      if (reach) {
        gather_columns<W>(st.wx + lane * S::kPitchX,
                          st.wy + lane * S::kPitchY + (start[1] & ((1 << S::kShiftY) - 1)), start[0], start[1], n0, n1,
                          fine + first_vector * grid.fine_count, grid.fine_count, last_vector - first_vector,
                          output + first_vector * count + point, count);
      }
      return;
    }
  }

  // Fragments: lane (g, t) holds rows (points) 8 m + g, and columns
  // x = 4 n + t (real and imaginary part) of the products.
  const int g = lane >> 2, t = lane & 3;
  int px[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    px[m] = __shfl_sync(0xFFFFFFFFu, start[0], 8 * m + g);
  }
  const uint32_t destination = __shfl_sync(0xFFFFFFFFu, point, 8 * t + g);
  // Left operands (row weights) of the 32 points.
  [[maybe_unused]] uint32_t ah[2][4], al[2][4];
  [[maybe_unused]] double a64[4][K];
  if constexpr (!F64) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const float* row = reinterpret_cast<const float*>(st.wy) + (16 * m + g) * S::kPitchY + t;
      split_tf32(row[0], ah[m][0], al[m][0]);
      split_tf32(row[8 * S::kPitchY], ah[m][1], al[m][1]);
      split_tf32(row[4], ah[m][2], al[m][2]);
      split_tf32(row[8 * S::kPitchY + 4], ah[m][3], al[m][3]);
    }
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
#pragma unroll
      for (int k = 0; k < K; ++k) a64[m][k] = st.wy[(8 * m + g) * S::kPitchY + 4 * k + t];
    }
  }
  while (todo != 0u) {
    const Group group = next_group(todo);
    const int lx = group.x, ly = group.y;
    [[maybe_unused]] const int lz = group.z;
    const bool mine = group.mine;
    const unsigned members = group.members;
    todo &= ~members;
    const int hx = __reduce_max_sync(0xFFFFFFFFu, mine ? start[0] : lx) + W - 1;
    // Blocks of columns that the windows of each 16 points reach (3D f32: one
    // product's rows); the others of the group's blocks weigh zero there. 96^3
    // modes, w 7, 1/4 point per cell: 451 -> 361 us, one point 866 -> 766; in 2D,
    // of one plane, the branch costs more than it saves (16 vectors 692 -> 817).
    [[maybe_unused]] int block_lo[2], block_hi[2];
    if constexpr (!F64 && D == 3) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const bool in = mine && (lane >> 4) == m;
        block_lo[m] = __reduce_min_sync(0xFFFFFFFFu, in ? start[0] : 0x7FFFFFFF) >> 2;
        block_hi[m] = (__reduce_max_sync(0xFFFFFFFFu, in ? start[0] : -W) + W - 1) >> 2;
      }
    }
    int z_lo = 0, z_hi = 0;
    if (D == 3) {
      z_lo = __reduce_min_sync(0xFFFFFFFFu, mine ? start[2] : 0x7FFFFFFF);
      z_hi = __reduce_max_sync(0xFFFFFFFFu, mine ? start[2] : 0) + W - 1;
    }
    // Grid rows of the lane's contracted indexes, as element offsets of a plane.
    int64_t row_at[F64 ? K : 2];
#pragma unroll
    for (int k = 0; k < (F64 ? K : 2); ++k) {
      int y = (ly << S::kShiftY) + 4 * k + t;
      while (y >= n1) y -= n1;
      row_at[k] = static_cast<int64_t>(y) * n0;
    }
    // V vectors at a time share the weights; the last pass of a batch that V
    // does not divide repeats its last vector.
    for (int b = first_vector; b < last_vector; b += V) {
      const Real* values[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const int vector = min(b + k, last_vector - 1);
        values[k] = reinterpret_cast<const Real*>(fine + static_cast<int64_t>(vector) * grid.fine_count) + (g & 1);
      }
      Complex v[V][4];
#pragma unroll
      for (int k = 0; k < V; ++k) {
#pragma unroll
        for (int m = 0; m < 4; ++m) v[k][m].x = v[k][m].y = Real(0);
      }
      for (int n = lx >> 2; n <= hx >> 2; ++n) {
        int column = 4 * n + (g >> 1);
        column = column >= n0 ? column - n0 : column;
        Real wx[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const int i = 4 * n + t - px[m];
          wx[m] = static_cast<unsigned>(i) < static_cast<unsigned>(W) ? st.wx[(8 * m + g) * S::kPitchX + i] : Real(0);
        }
        const Real* const weights_z = st.wz + g * S::kPitchZ - (lz << S::kShiftZ);
#pragma unroll 2
        for (int z = z_lo; z <= z_hi; ++z) {
          const int64_t plane = D == 3 ? static_cast<int64_t>(z >= n2 ? z - n2 : z) * plane_cells : 0;
          Real weight[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            weight[m] = wx[m];
            if (D == 3) weight[m] *= weights_z[8 * m * S::kPitchZ + z];
          }
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const Real* const at = values[k] + 2 * (plane + column);
            if constexpr (!F64) {
              uint32_t bh0, bl0, bh1, bl1;
              split_tf32(__ldg(at + 2 * row_at[0]), bh0, bl0);
              split_tf32(__ldg(at + 2 * row_at[1]), bh1, bl1);
#pragma unroll
              for (int m = 0; m < 2; ++m) {
                if (D == 3 && (n < block_lo[m] || n > block_hi[m])) continue;
                float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma_tf32(d, al[m], bh0, bh1);
                mma_tf32(d, ah[m], bl0, bl1);
                mma_tf32(d, ah[m], bh0, bh1);
                v[k][2 * m] = cfma(make_float2(d[0], d[1]), weight[2 * m], v[k][2 * m]);
                v[k][2 * m + 1] = cfma(make_float2(d[2], d[3]), weight[2 * m + 1], v[k][2 * m + 1]);
              }
            } else {
              double2 d[4];
#pragma unroll
              for (int m = 0; m < 4; ++m) d[m] = make_double2(0.0, 0.0);
#pragma unroll
              for (int i = 0; i < K; ++i) {
                const double value = __ldg(at + 2 * row_at[i]);
#pragma unroll
                for (int m = 0; m < 4; ++m) mma_f64(d[m], a64[m][i], value);
              }
#pragma unroll
              for (int m = 0; m < 4; ++m) v[k][m] = cfma(d[m], weight[m], v[k][m]);
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < V; ++k) {
        // The columns' sums, halved twice: lane t ends with point 8 t + g.
        const bool upper = (t & 2) != 0, odd = (t & 1) != 0;
        Complex half[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const Complex keep = upper ? v[k][2 + m] : v[k][m], give = upper ? v[k][m] : v[k][2 + m];
          half[m].x = keep.x + __shfl_xor_sync(0xFFFFFFFFu, give.x, 2);
          half[m].y = keep.y + __shfl_xor_sync(0xFFFFFFFFu, give.y, 2);
        }
        const Complex keep = odd ? half[1] : half[0], give = odd ? half[0] : half[1];
        Complex e;
        e.x = keep.x + __shfl_xor_sync(0xFFFFFFFFu, give.x, 1);
        e.y = keep.y + __shfl_xor_sync(0xFFFFFFFFu, give.y, 1);
        if (((members >> (8 * t + g)) & 1u) && b + k < last_vector) {
          output[static_cast<int64_t>(b + k) * count + destination] = e;
        }
      }
    }
  }
}

template <int D, int W, typename T>
void launch_width(const GridParams& g, const typename T::Real* points, const void* windows, int64_t count,
                  const uint32_t* perm, const typename T::Complex* fine, int batch, typename T::Complex* output,
                  cudaStream_t stream) {
  const dim3 blocks(static_cast<unsigned>((count + 32 * T::kWarps - 1) / (32 * T::kWarps)),
                    static_cast<unsigned>((batch + kBlockVectors - 1) / kBlockVectors));
  if constexpr (D == 2 && sizeof(typename T::Real) == 4) {
    if (batch > 1) {
      interp_strips_kernel<D, W, kBlockVectors, T><<<blocks, T::kWarps * 32, 0, stream>>>(g, points, windows, count,
                                                                                          perm, fine, batch, output);
      note_launch();
      return;
    }
  }
  if constexpr (D == 2 && sizeof(typename T::Real) == 8) {
    // From half a point per cell on (w 11 and wider: a twelfth) few warps are
    // scattered, and the kernel without gathers, whose bits are the same, is 1 to
    // 4 % faster.
    if ((W <= 10 ? 2 : 12) * count < g.fine_count) {
      interp_strips_kernel<D, W, 1, T, true><<<blocks, T::kWarps * 32, 0, stream>>>(g, points, windows, count, perm,
                                                                                    fine, batch, output);
      note_launch();
      return;
    }
  }
  interp_strips_kernel<D, W, 1, T><<<blocks, T::kWarps * 32, 0, stream>>>(g, points, windows, count, perm, fine, batch,
                                                                          output);
  note_launch();
}

}  // namespace

bool interp_strips_chosen(int dimensions, bool f64, int width, int64_t points, int64_t cells) {
  // 2D f64 warps choose for themselves (kMostGroups).
  if (f64 && (dimensions == 2 || width < 5)) return dimensions == 2 && width >= 5;
  if (dimensions != 3) return false;
  // Cells per point up to which a group's products cost less than its gathers;
  // and points from which the warps, whose groups follow one another, are enough
  // to hide it (20^3 to 40 x 36 x 30 modes, us per transform, gather against strips:
  // f32 w 6, 64 000 points 29 / 33, 172 800 51 / 56, 691 200 95 / 89 (clustered, 262 000
  // 44 / 35); w 7, 65 500 36 / 48, 87 400 47 / 43; f64 w 6, 57 600 58 / 70, 87 400 72 / 65).
  if (f64) return points * (width < 12 ? 6 : 12) >= cells && (width > 6 || points >= 80'000);
  return (width == 6 && points * 3 >= cells && points >= 250'000) ||
         (width == 7 && points * 4 >= cells && points >= 80'000);
}

void interp_strip_shifts(bool f64, int32_t shift[3]) {
  shift[0] = 0;
  shift[1] = f64 ? Strip<kMaxWidth, true>::kShiftY : Strip<7, false>::kShiftY;
  shift[2] = Strip<7, false>::kShiftZ;
}

void interp_strips_execute(const GridParams& g, const InterpLaunch& l, cudaStream_t stream) {
  if (l.point_count == 0) return;
  auto launch = [&](auto kernel) {
    kernel(g, l.points, l.windows, l.point_count, l.perm, l.fine, l.batch, l.output, stream);
  };
  if (g.dimensions == 2) {
    switch (g.width) {
      case 2: launch(launch_width<2, 2, F32Strips>); break;
      case 3: launch(launch_width<2, 3, F32Strips>); break;
      case 4: launch(launch_width<2, 4, F32Strips>); break;
      case 5: launch(launch_width<2, 5, F32Strips>); break;
      case 6: launch(launch_width<2, 6, F32Strips>); break;
      default: launch(launch_width<2, 7, F32Strips>); break;
    }
    return;
  }
  switch (g.width) {
    case 6: launch(launch_width<3, 6, F32Strips>); break;
    default: launch(launch_width<3, 7, F32Strips>); break;
  }
}

void interp_strips_execute64(const GridParams& g, const InterpLaunch64& l, cudaStream_t stream) {
  if (l.point_count == 0) return;
  auto launch = [&](auto kernel2, auto kernel3) {
    (g.dimensions == 2 ? kernel2 : kernel3)(g, l.points, nullptr, l.point_count, l.perm, l.fine, l.batch, l.output,
                                            stream);
  };
  switch (g.width) {
#define B200NUFFT_STRIPS_CASE(WIDTH) \
  case WIDTH: launch(launch_width<2, WIDTH, F64Strips>, launch_width<3, WIDTH, F64Strips>); break;
    B200NUFFT_STRIPS_CASE(5)
    B200NUFFT_STRIPS_CASE(6)
    B200NUFFT_STRIPS_CASE(7)
    B200NUFFT_STRIPS_CASE(8)
    B200NUFFT_STRIPS_CASE(9)
    B200NUFFT_STRIPS_CASE(10)
    B200NUFFT_STRIPS_CASE(11)
    B200NUFFT_STRIPS_CASE(12)
    B200NUFFT_STRIPS_CASE(13)
    B200NUFFT_STRIPS_CASE(14)
    B200NUFFT_STRIPS_CASE(15)
    default:
    B200NUFFT_STRIPS_CASE(16)
#undef B200NUFFT_STRIPS_CASE
  }
}

}  // namespace b200nufft
