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
// Two tiles: 64 x 64 from one and a half tiles per SM on, else 32 x 64 with half the
// pixels per thread (4 slices of 1023 x 1023: 104 against 115 us per slice; 8 slices
// of 512 x 512: 26 for the small tile against 37 us one slice at a time).
cudaError_t launch_bp_quad(const BpLaunch &a, cudaStream_t st, bool check);
const char *bp_quad_error_detail();
// False where the groups are too few to fill the device and slices one at a time are
// faster: 4 slices of 300 x 300 (50 small tiles) take 26 us a slice in a group and 15
// alone, 4 of 512 x 512 (128 tiles) 40 and 41.
bool bp_quad_pays(int64_t rows, int64_t cols, int64_t slices, int sms);
}  // namespace ctas
