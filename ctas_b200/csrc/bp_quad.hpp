// bp_quad.hpp -- launch interface of the four-slice backprojection kernel.
#pragma once
#include <cuda_runtime.h>

#include "fbp_kernels.hpp"

namespace ctas {
// Backprojects a.S slices of one geometry whose filtered rows are interleaved four
// slices to a sample (kQuadSlices, fbp_kernels.hpp): a.q points at row 0, column 0,
// with kQuadSlack samples allocated before it and behind the last row.  Reference
// truncation, float32, every sine >= 0 or the wide layout, 0 < geo_p <= 1; or linear
// interpolation of rows without guard columns, every sine >= 0.
// `check`: every shared-memory read is bounds-checked (violations set bit 8 of
// *a.err and read 0); for tests.
// Two tiles: 64 x 64, and 32 x 64 with half the pixels per thread (quad_small_tile).
cudaError_t launch_bp_quad(const BpLaunch &a, cudaStream_t st, bool check);
const char *bp_quad_error_detail();
}  // namespace ctas
