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

// A warp per row: packed -> pitched (unpack) or pitched -> packed (pack), rows
// [r0, r1) of the 2 * rows of the task.
template <bool UNPACK>
__device__ __forceinline__ void rows_copy(const RowsTask& t, int64_t r0, int64_t r1) {
  const int lane = threadIdx.x & 31;
  const int64_t wpb = blockDim.x >> 5;
  for (int64_t r = r0 + (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); r < r1;
       r += (int64_t)gridDim.x * wpb) {
    const int c = r >= t.rows ? 1 : 0;
    double* pitched = t.q[c] + (r - c * t.rows) * t.sy;
    double* packed = t.packed + r * t.e0;
    for (int i = lane; i < t.e0; i += 32) {
      if (UNPACK) pitched[i] = packed[i];
      else packed[i] = pitched[i];
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
