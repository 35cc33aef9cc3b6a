// rows.cuh -- a patch's state between a packed array and its pitched fields.
#pragma once
#include <stdint.h>

namespace bsam {

// One problem's root state between the caller's Fortran-ordered q (both
// components, ghosts included: `rows` rows of e0 values per component) and
// the pitched master fields q0, q1 (row pitch sy; in 3D the plane pitch is
// sy * (n1 + 2), so the rows of every plane follow each other at pitch sy).
// The packed copy lives in the engine's device transfer buffer, which one
// contiguous DMA per problem fills from, or empties into, the caller's
// buffer: pitched host copies of rows this short run far below the link's
// speed.
struct RowsTask {
  double* packed;
  double* q[2];
  int64_t rows, sy;
  int32_t e0, pad_;
};

// Packed -> pitched (unpack) or pitched -> packed (pack), rows [r0, r1) of the
// 2 * rows of the task.  A warp per row, of rows above ROW_PART elements per equal
// part: a load over the bus takes a microsecond or two, so what counts is how many
// are in flight.  (A warp per row with one load a lane in flight: put of 2048^2, rows
// of 16 KB, 10.4 ms, of 1024 x 512 1.1 ms.)
constexpr int ROW_PART = 512, ROW_LOADS = 8;
template <bool UNPACK>
__device__ __forceinline__ void rows_copy(const RowsTask& t, int64_t r0, int64_t r1) {
  const int lane = threadIdx.x & 31;
  const int64_t wpb = blockDim.x >> 5;
  const int parts = (t.e0 + ROW_PART - 1) / ROW_PART;
  const int len = ((t.e0 + parts - 1) / parts + 31) / 32 * 32;
  for (int64_t w = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); w < (r1 - r0) * parts;
       w += (int64_t)gridDim.x * wpb) {
    const int64_t r = r0 + (parts == 1 ? w : w / parts);
    const int first = parts == 1 ? 0 : (int)(w % parts) * len;
    const int end = min(first + len, t.e0);
    const int c = r >= t.rows ? 1 : 0;
    double* pitched = t.q[c] + (r - c * t.rows) * t.sy;
    double* packed = t.packed + r * t.e0;
    const double* src = UNPACK ? packed : pitched;
    double* dst = UNPACK ? pitched : packed;
    for (int i = first + lane; i < end; i += 32 * ROW_LOADS) {
      double v[ROW_LOADS];
#pragma unroll
      for (int u = 0; u < ROW_LOADS; ++u)
        if (i + 32 * u < end) v[u] = src[i + 32 * u];
#pragma unroll
      for (int u = 0; u < ROW_LOADS; ++u)
        if (i + 32 * u < end) dst[i + 32 * u] = v[u];
    }
  }
}

template <bool UNPACK>
__global__ void __launch_bounds__(256) k_rows_list(const RowsTask* __restrict__ tasks) {
  const RowsTask t = tasks[blockIdx.y];
  rows_copy<UNPACK>(t, 0, 2 * t.rows);
}

// One task by value; packed is page-locked host memory, which the device reads
// and writes directly.
template <bool UNPACK>
__global__ void __launch_bounds__(256) k_rows(const RowsTask t, int64_t r0, int64_t r1) {
  rows_copy<UNPACK>(t, r0, r1);
}


}  // namespace bsam
