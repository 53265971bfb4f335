// Sums over frequencies as products on the FP64 matrix instruction (m8n8k4),
// for the FP64 reverse passes (kernels.cu, xhm.cu). A block keeps the basis of
// the phases and amplitudes over kSpan frequencies as the rows of a matrix in
// shared memory; a warp writes eight values of each of its 32 frequencies (the
// cotangents of a phase, an amplitude, ...) as the columns of another, and the
// products of the rows with the columns are the sums of basis times cotangent
// that a reverse pass needs: 8 rows x 8 columns x 32 frequencies in eight
// instructions and four registers a lane, where a register per sum and lane
// costs two each, and a shuffle tree at the end.
#pragma once

#include <cuda_runtime.h>

namespace wfx {

constexpr int kSpan = 128;             // frequencies of the rows' matrix
constexpr int kRowStride = kSpan + 4;  // (doubles; = 4 mod 16: the fragments' loads are conflict-free)
constexpr int kStageStride = 36;       // (32 frequencies a column, = 4 mod 16)
constexpr int kStage = 8 * kStageStride;

// An entry of the rows: zero where it is not finite, so that it adds nothing to
// the sums of a column that is zero there (a power that overflows in a region
// that does not read it). Where the value itself is not finite its columns are.
__device__ __forceinline__ double row_entry(double x) { return isfinite(x) ? x : 0.0; }

// f^-7/6 as the amplitudes take it beside such rows: NaN where f or f^-5/3 is
// not finite (f <= 0, NaN, an infinity), since the powers read back from the
// rows no longer say so.
__device__ __forceinline__ double row_m76(double f, double y, double m76) {
  return isfinite(f) && isfinite(y) ? m76 : NAN;
}

// d += a b of one 8 x 4 by 4 x 8 product: lane l holds a[l / 4][l % 4],
// b[l % 4][l / 4] and d[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Puts eight values a lane into the warp's columns (frequency = lane).
__device__ __forceinline__ void put_columns(double* stage, const double (&v)[8], int lane) {
  __syncwarp();
#pragma unroll
  for (int n = 0; n < 8; ++n) stage[n * kStageStride + lane] = v[n];
  __syncwarp();
}

// d[t] += rows 8 t .. 8 t + 7 (of ROWS) times the columns, over 32
// frequencies; rows: the matrix from the first of them on.
template <int ROWS, int TILES>
__device__ __forceinline__ void mma_rows(double (&d)[TILES][2], const double* rows, const double* stage, int lane) {
  const int r = lane >> 2, k = lane & 3;
  const double* column = stage + r * kStageStride + k;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const double b = column[4 * s];
#pragma unroll
    for (int t = 0; t < TILES; ++t) {
      // (a last tile's rows past ROWS repeat the last row: not read back)
      const int row = 8 * t + 7 < ROWS ? 8 * t + r : min(8 * t + r, ROWS - 1);
      mma_f64(d[t], rows[row * kRowStride + k + 4 * s], b);
    }
  }
}

// d += the sums of the columns, in every row.
__device__ __forceinline__ void mma_ones(double (&d)[2], const double* stage, int lane) {
  const double* column = stage + (lane >> 2) * kStageStride + (lane & 3);
#pragma unroll
  for (int s = 0; s < 8; ++s) mma_f64(d, 1.0, column[4 * s]);
}

// Writes d (8 rows each) to the warp's stage as entries [8 row + column].
template <int TILES>
__device__ __forceinline__ void put_products(double* stage, const double (&d)[TILES][2], int lane) {
  __syncwarp();
#pragma unroll
  for (int t = 0; t < TILES; ++t) {
    double* at = stage + 8 * (8 * t + (lane >> 2)) + 2 * (lane & 3);
    at[0] = d[t][0];
    at[1] = d[t][1];
  }
  __syncwarp();
}

}  // namespace wfx
