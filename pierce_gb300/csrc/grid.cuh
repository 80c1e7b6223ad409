// The xy column grid over a dataset's object boxes: cell of a coordinate.
#pragma once

#include <cuda_runtime.h>

namespace pgpu {

__device__ __forceinline__ void grid_cell_range(const float* b, int nx, int ny, float lo, float hi, int axis,
                                                int& c0, int& c1) {
    const float o = b[axis], e = b[2 + axis] - b[axis];
    const int n = axis ? ny : nx;
    const float inv = e > 0.0f ? (float)n / e : 0.0f;
    c0 = min(max((int)floorf((lo - o) * inv), 0), n - 1);
    c1 = min(max((int)floorf((hi - o) * inv), 0), n - 1);
}

}  // namespace pgpu
