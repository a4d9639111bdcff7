// Float64 tensor-core products of I x R by R x R matrices, rows in registers.
//
// A warp takes eight rows; lane l holds, of row l / 4, the columns
// 8 c + 2 (l % 4) and the one to its right of every 8-column tile c (the
// accumulator layout of mma.m8n8k4).  A product of these rows by a matrix M
// takes them as they lie: the k index of an m8n8k4 step is the lane's place in
// its quad, so step (c, e) multiplies columns 8 c + {0, 2, 4, 6} + e, and M's rows
// are put in that order when it is laid out in shared memory (fragment order:
// one conflict-free 8-byte read a lane and step).  The result has the layout of
// the input, so products chain without shuffles or shared memory, and every
// global load and store of a row is a pair.
#pragma once

#include <cstdint>

namespace alto {

// d += a b on the float64 tensor cores, one 8 x 8 x 4 step of a warp: lane l
// gives a = A[l / 4][l % 4] and b = B[l % 4][l / 4] and holds D[l / 4][2 (l % 4)]
// and the element to its right.  Float64 products and sums, as __fma_rn; the
// tensor cores' float64 rate is that of the FMA units (37 TFLOP/s measured for
// both), but an instruction is 256 multiply-adds for two operand registers a
// lane, where the FMA form reads shared memory for every few.
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// M (R x R, row-major) into fragment order over T column tiles (64 T^2
// doubles, zero past R); all threads of the block, no barrier.
__device__ __forceinline__ void load_fragments(double* __restrict__ frag, const double* __restrict__ M, int R, int T) {
  for (int p = threadIdx.x; p < 64 * T * T; p += blockDim.x) {
    const int l = p & 31, f = p >> 5, n = f % T, ce = f / T;
    const int k = (ce >> 1) * 8 + 2 * (l & 3) + (ce & 1), col = 8 * n + (l >> 2);
    frag[p] = k < R && col < R ? M[k * R + col] : 0.0;
  }
}

// x = a M, frag being M in fragment order.
template <int T>
__device__ __forceinline__ void rows_product(const double (&a)[T][2], const double* __restrict__ frag, int lane,
                                             double (&x)[T][2]) {
#pragma unroll
  for (int n = 0; n < T; ++n) x[n][0] = x[n][1] = 0.0;
#pragma unroll
  for (int c = 0; c < T; ++c)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int n = 0; n < T; ++n) dmma_8x8x4(x[n], a[c][e], frag[((c * 2 + e) * T + n) * 32 + lane]);
}

// This lane's pairs of row `row` of a float32 or float64 matrix of R = 8 T
// columns (zeros past I rows).
template <int T, typename TX>
__device__ __forceinline__ void load_pairs(const TX* __restrict__ X, uint64_t row, bool in, int quad,
                                           double (&x)[T][2]) {
#pragma unroll
  for (int c = 0; c < T; ++c) {
    if constexpr (sizeof(TX) == 4) {
      float2 v = make_float2(0.f, 0.f);
      if (in) v = *reinterpret_cast<const float2*>(X + row * (8 * T) + 8 * c + 2 * quad);
      x[c][0] = (double)v.x;
      x[c][1] = (double)v.y;
    } else {
      double2 v = make_double2(0.0, 0.0);
      if (in) v = *reinterpret_cast<const double2*>(X + row * (8 * T) + 8 * c + 2 * quad);
      x[c][0] = v.x;
      x[c][1] = v.y;
    }
  }
}

template <int T>
__device__ __forceinline__ void store_pairs(float* __restrict__ X, uint64_t row, int quad, const double (&x)[T][2]) {
#pragma unroll
  for (int c = 0; c < T; ++c)
    *reinterpret_cast<float2*>(X + row * (8 * T) + 8 * c + 2 * quad) = make_float2((float)x[c][0], (float)x[c][1]);
}
template <int T>
__device__ __forceinline__ void store_pairs(double* __restrict__ X, uint64_t row, int quad, const double (&x)[T][2]) {
#pragma unroll
  for (int c = 0; c < T; ++c)
    *reinterpret_cast<double2*>(X + row * (8 * T) + 8 * c + 2 * quad) = make_double2(x[c][0], x[c][1]);
}

}  // namespace alto
