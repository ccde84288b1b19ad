// Warp-level matrix products (mma.sync) of the spreading and interpolation
// strips, whose products are too small for tcgen05's 128-row tiles: measured
// on a B200, an m16n8k8 tf32 or m16n8k16 f16 product takes 2.0 cycles of an
// SM, an m8n8k4 f64 product 4.0 (64 fused multiply-adds per cycle, the rate
// of the scalar f64 units, from an eighth of the instructions).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace b200nufft {

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The tensor core cuts a sum of products off at 24 bits instead of rounding it:
// half a unit of the last place towards zero on average, over mantissas of
// uniform logarithm 2^-24 / (2 ln 2) of the sum. All sums of a cell lose this
// share of their magnitude alike, so f32 strips of one-signed strengths came
// out 4e-8 too small (radial 128^3, w 6: error against 64 bits 1.29e-7 with
// scalar multiply-adds, 1.40e-7 with the products).
constexpr float kProductLoss = 4.3e-8f;

// v to the nearest value of the 19 bits a tf32 operand keeps, and the exact
// remainder, whose sign is then independent of v's: what the products drop
// (the remainder's own last bits, low times low) does not add up.
__device__ __forceinline__ void split_tf32(float v, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(v) + 0x1000u) & 0xFFFFE000u;
  lo = __float_as_uint(v - __uint_as_float(hi));
}

__device__ __forceinline__ void mma_f64(double2& d, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d.x), "+d"(d.y)
      : "d"(a), "d"(b));
}

}  // namespace b200nufft
